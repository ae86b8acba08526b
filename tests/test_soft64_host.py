"""Integer-pipe double-precision operations (torch_gb300/csrc/tfv_soft64.cuh):
the header is compiled on the host with g++ and division, square root,
scaling by a power of two, comparisons and min / max are compared bit for bit
with the host's IEEE operations, on random bit patterns, on sparse and dense
mantissas, next to representable quotients and squares, on subnormal operands
and results, and on zeros, infinities and NaN.  The host's stand-ins for the
hardware's reciprocal estimates carry an error of either sign beyond the
hardware's (2^-22): the results must not depend on it."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "torch_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cmath>
#include <random>
#include "tfv_soft64.cuh"
using namespace tfv;
static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static double real(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
static std::mt19937_64 g(7);
static long bad = 0;
static void check(const char* what, double a, double b, double got, double want) {
  if ((got != got && want != want) || bits(got) == bits(want)) return;
  if (bad++ < 5) std::printf("%s %a %a: got %a want %a\n", what, a, b, got, want);
}
__attribute__((noinline)) static void truth(double a, double b, bool got, bool want) {
  if (got != want && bad++ < 5) std::printf("comparison %a %a: got %d\n", a, b, got);
}
// mantissa and sign of m, exponent near 1 (a span of 50) or as given
static double scaled(uint64_t m, uint64_t low = 1000, uint64_t span = 50) {
  return real((m & 0x800fffffffffffffull) | ((low + g() % span) << 52));
}
int main() {
  const double special[] = {0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 1e-14, 1e-12, INFINITY, -INFINITY,
                            NAN, -NAN, 5e-324, -5e-324, 2.2250738585072014e-308, 4.4e-308,
                            1.7976931348623157e308, 8.9e307};
  const int ns = sizeof(special) / sizeof(special[0]);
  for (long i = 0; i < 3000000; ++i) {
    const uint64_t m = g(), n = g();
    double a = scaled(m), b = scaled(n);
    switch (g() % 8) {
      case 0: a = real(m); b = real(n); break;
      case 1: a = scaled(m & g() & g()); b = scaled(n & g() & g()); break;
      case 2: a = scaled(m | g() | g()); b = scaled(n | g() | g()); break;
      case 3: {  // next to a representable quotient
        b = scaled(n, 1023, 1);
        a = real(bits(scaled(m, 1023, 1) * b) + g() % 3 - 1);
        break;
      }
      case 4: a = real(m & 0x801fffffffffffffull); b = scaled(n, 960, 120); break;
      case 5: a = scaled(m, 1, 60); b = scaled(n, 1000, 70);
        if (g() % 3 == 0) b = real(bits(b) & 0xfff0000000000000ull);  // ties in subnormals
        break;
      case 6: a = special[g() % ns]; if (g() % 2) b = special[g() % ns]; break;
      default: break;
    }
    check("div", a, b, soft_div(a, b), a / b);
    check("sqrt", a, 0, soft_sqrt(a), std::sqrt(a));
    const double sq = real(bits(b * b) + g() % 3 - 1);
    check("sqrt", sq, 0, soft_sqrt(sq), std::sqrt(sq));
    check("half", a, 0, soft_half(a), 0.5 * a);
    check("twice", a, 0, soft_twice(a), 2.0 * a);
    if (g() % 4 == 0) b = a;
    check("max", a, b, soft_max(a, b), (a >= b || a != a) ? a : b);
    check("min", a, b, soft_min(a, b), (a <= b || a != a) ? a : b);
    check("max_pos", a, 0, soft_max_pos(a, 1e-12), (a >= 1e-12 || a != a) ? a : 1e-12);
    const double run = b != b ? 0.0 : std::fabs(b);
    check("fmax", run, a, soft_fmax_run(run, a), a > run ? a : run);
    truth(a, b, soft_lt(a, b), a < b);
    truth(a, b, soft_le(a, b), a <= b);
    truth(a, 0, soft_le0(a), a <= 0);
    truth(a, 0, soft_gt0(a), a > 0);
    truth(a, 0, soft_lt0(a), a < 0);
    truth(a, 0, soft_ge0(a), a >= 0);
    truth(a, 1e-12, soft_gt_pos(a, 1e-12), a > 1e-12);
    truth(a, 1e-14, soft_abs_lt(a, 1e-14), std::fabs(a) < 1e-14);
    truth(a, 0, soft_isnan(a), a != a);
    truth(a, 0, soft_isfinite(a), std::isfinite(a));
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.parametrize("error", ["0.0f", "4.76837158e-7f", "-4.76837158e-7f"])
def test_results_equal_ieee(tmp_path, error):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    src = tmp_path / "soft.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "soft"
    subprocess.run([gxx, "-O2", "-std=c++17", "-DTFV_SOFT_TEST_ERROR=" + error,
                    "-I" + str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "bad 0" in out.stdout
