// Independent launches side by side: the first on a main stream, the others on
// side streams that are forked from it and joined to it by events.  Host code
// without CUDA headers, so that a test drives it with a recording stand-in.
#pragma once

namespace tfv {

// Work k of n: k = 0 on the main stream, k > 0 on side stream k between
// ops.enter(k) (the side stream waits for the fork) and ops.leave(k) (the main
// stream waits for the side stream).  Every side stream that was entered is
// left, also after an error: the caller may free what the launches use once the
// main stream has passed, so none of them may outlive it; where leaving itself
// fails, ops.drain(k) waits on the host.  Returns the first error.
template <typename Error, typename Ops, typename Work>
Error fork_join(Ops& ops, int n, Work work) {
  const Error ok{};  // success is zero
  Error first = n > 1 ? ops.fork() : ok;
  int entered = 0;
  for (int k = 0; k < n && first == ok; ++k) {
    if (k > 0) {
      first = ops.enter(k);
      if (first != ok) break;
      entered = k;
    }
    first = work(k);
  }
  for (int k = 1; k <= entered; ++k) {
    const Error e = ops.leave(k);
    if (e == ok) continue;
    ops.drain(k);
    if (first == ok) first = e;
  }
  return first;
}

}  // namespace tfv
