"""Staged range of a step tile (halo_before, halo_after in
torch_gb300/csrc/tfv_types.h), compiled on the host with g++: over every tiling of
short axes, one-cell tiles among them, the cells that the tile copies lie inside
the axis, and with the ghost cells before and after them they make up the tile and
its two-cell halo."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "torch_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "tfv_types.h"
int main() {
  int bad = 0, tiles = 0;
  for (int n = 2; n <= 40; ++n)
    for (int t = 1; t <= n + 3; ++t)
      for (int at = 0; at < n; at += t, ++tiles) {
        const int len = std::min(t, n - at);
        const int before = tfv::halo_before(at), after = tfv::halo_after(at, len, n);
        int outside_lo = 0, outside_hi = 0;
        for (int k = at - 2; k < at + len + 2; ++k) {
          outside_lo += k < 0;
          outside_hi += k >= n;
        }
        bad += before != outside_lo || after != outside_hi || len + 4 - before - after < 1;
      }
  std::printf("%d tiles, %d bad\n", tiles, bad);
  return bad != 0;
}
"""


def test_staged_cells_lie_inside_the_axis(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("needs g++")
    src = tmp_path / "halo.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "halo"
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + str(CSRC), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_kernel_forms_its_ranges_with_them():
    text = (CSRC / "tfv_kernels.cuh").read_text()
    tile = text[text.index("struct HydroTile"):text.index("Cell stage of the cell")]
    assert "y0 == 0" not in tile and "x0 == 0" not in tile
    assert tile.count("halo_before(y0)") == 2 and tile.count("halo_after(y0, by, g.nb)") == 2
