"""Fork and join of a step's limiter groups (fork_join in
torch_gb300/csrc/tfv_fork.h), compiled on the host with g++ and driven with a
stand-in for the streams whose n-th call fails: whatever fails, every side stream
that got work is joined to the main stream or waited for before the error is
returned, and the error is the first one."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "torch_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "tfv_fork.h"
struct Streams {
  int fail_at, calls = 0, first = 0;
  std::vector<int> busy, settled;  // side streams with work; joined or drained
  int call() {
    if (++calls < fail_at) return 0;
    if (!first) first = calls;
    return calls;  // this call and every later one fail
  }
  int fork() { return call(); }
  int enter(int) { return call(); }
  int leave(int k) {
    const int e = call();
    if (!e) settled[k] = 1;
    return e;
  }
  void drain(int k) { settled[k] = 1; }
};
int main() {
  int bad = 0;
  for (int n = 1; n <= 4; ++n)
    for (int once = 0; once < 2; ++once)  // all later calls fail too, or only one launch
      for (int fail_at = 1; fail_at <= 4 * n + 2; ++fail_at) {
        Streams s{once ? 1 << 20 : fail_at};
        s.busy.assign(n, 0);
        s.settled.assign(n, 0);
        int launches = 0, launch_error = 0;
        const int e = tfv::fork_join<int>(s, n, [&](int k) {
          int r = s.call();
          if (once && ++launches == fail_at) r = launch_error = -fail_at;
          if (!r) s.busy[k] = 1;
          return r;
        });
        bad += e != (launch_error ? launch_error : s.first);
        for (int k = 1; k < n; ++k) bad += s.busy[k] && !s.settled[k];
        if (e == 0)
          for (int k = 0; k < n; ++k) bad += !s.busy[k];
      }
  std::printf("bad %d\n", bad);
  return bad != 0;
}
"""


def test_started_work_is_joined_after_an_error(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    src = tmp_path / "fork.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "fork"
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", "-Werror", "-I" + str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
