"""Limiter functions in double precision (limiter_phi in
torch_gb300/csrc/tfv_soft64.cuh), compiled on the host with g++ and compared bit
for bit with the maximum / minimum nests of the reference
(python/cfdSolver/torchSolver3D.py:86-111, python/cfdSolver/torchSolver2D.py:
147-165) written with plain IEEE operations: over random bit patterns, ratios
around the nests' corners, zeros of both signs, infinities, subnormals and NaN.
A 2D VanLeer or Albada ratio that is NaN gives 0, any other NaN gives NaN."""

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
static double mx(double a, double b) { return (a >= b || a != a) ? a : b; }  // numpy.maximum
static double mn(double a, double b) { return (a <= b || a != a) ? a : b; }  // numpy.minimum
static double nest(int dim, int lim, double r) {
  const double pos = mx(r, 0.0);
  switch (lim) {
    case 0: return dim == 2 && !(r > 0.0) ? 0.0 : 2.0 * pos / (1.0 + pos);
    case 1: return dim == 2 && !(r > 0.0) ? 0.0 : (pos * pos + pos) / (pos * pos + 1.0);
    case 2: return mx(0.0, mn(r, 1.0));
    case 3: return mx(0.0, mx(mn(2.0 * r, 1.0), mn(r, 2.0)));
    default: {
      double m = mn(mn(2.0, 2.0 * r), (2.0 + r) / 3.0);
      if (dim == 3) m = mn(m, (1.0 + 2.0 * r) / 3.0);
      return mx(0.0, m);
    }
  }
}
static long bad = 0;
static void check(int dim, int lim, double r, double got) {
  const double want = nest(dim, lim, r);
  if ((got != got && want != want) || bits(got) == bits(want)) return;
  if (bad++ < 8) std::printf("%dD limiter %d, r = %a: got %a want %a\n", dim, lim, r, got, want);
}
static void all(double r) {
  check(2, 0, r, limiter_phi<2, 0>(r));
  check(2, 1, r, limiter_phi<2, 1>(r));
  check(2, 2, r, limiter_phi<2, 2>(r));
  check(2, 3, r, limiter_phi<2, 3>(r));
  check(2, 4, r, limiter_phi<2, 4>(r));
  check(3, 0, r, limiter_phi<3, 0>(r));
  check(3, 1, r, limiter_phi<3, 1>(r));
  check(3, 2, r, limiter_phi<3, 2>(r));
  check(3, 3, r, limiter_phi<3, 3>(r));
  check(3, 4, r, limiter_phi<3, 4>(r));
}
int main() {
  const double corners[] = {0.0, 0.25, 0.5, 1.0, 2.0, 4.0, 5e-324, 2.2250738585072014e-308,
                            1e154, 1e155, 8.98846567431158e307, 1.7976931348623157e308, INFINITY,
                            NAN};
  for (double c : corners)
    for (int k = -3; k <= 3; ++k)
      for (int s = 0; s < 2; ++s) all(real((bits(c) + (uint64_t)(int64_t)k) ^ ((uint64_t)s << 63)));
  std::mt19937_64 g(11);
  for (long i = 0; i < 400000; ++i) {
    const uint64_t m = g();
    all(real(m));
    all(real((m & 0x800fffffffffffffull) | ((1013 + g() % 20) << 52)));
  }
  std::printf("bad %ld\n", bad);
  return bad != 0;
}
"""


def test_phi_equals_the_nests(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    src = tmp_path / "phi.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "phi"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + str(CSRC), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
