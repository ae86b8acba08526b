"""Default tilings against explicit ones, and per-cell gamma staged by tensor
copies.  Per-cell arithmetic does not depend on the tile shape, so states of
the default tiling (double precision: chosen by a cost model; 1D: 122 cells in
128 threads) equal those of another tiling bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402
from torch_gb300 import stepfn  # noqa: E402


def rough(counts, seed=3):
    rng = np.random.default_rng(seed)
    shape = tuple(counts[::-1])
    dim = len(counts)
    p = np.empty((dim + 2,) + shape)
    p[0] = 0.5 + rng.random(shape)
    p[1:-1] = 0.4 * (rng.random((dim,) + shape) - 0.5)
    p[-1] = 0.5 + rng.random(shape)
    return p


def test_2d_fp32_step_with_gamma_per_cell():
    """Two 124-cell tiles by tensor copy, gamma as an array: the single
    precision step stays within the L1 criterion of the double one (1e-5)."""
    p = rough((132, 37))
    u = p.copy()
    u[1:3] *= p[0]
    gamma = 1.3 + 0.2 * np.random.default_rng(1).random((37, 132))
    u[3] = p[3] / (gamma - 1) + 0.5 * p[0] * (p[1] ** 2 + p[2] ** 2)
    args = (1 / 132, 1 / 37, 1e-3, gamma, "VanLeer", "Reflective", "Periodic")
    want = stepfn.muscl_hancock_step_2d(u, *args)
    got = stepfn.muscl_hancock_step_2d(u, *args, precision="fp32")
    for c in range(4):
        assert np.abs(got[c] - want[c]).mean() <= 1e-5 * np.abs(want[c]).mean()


@pytest.mark.parametrize("counts,tile", [
    ((31, 7), (128, 1, 32)), ((62, 5), (32, 1, 4)), ((126, 33), (128, 1, 32)),
    ((250, 18), (64, 1, 16)), ((2, 2), (128, 1, 32)),
    ((15, 9, 5), (32, 4, 32)), ((28, 16, 33), (16, 8, 16)), ((14, 14, 2), (32, 4, 32)),
    ((29, 43, 17), (32, 4, 32)),
])
@pytest.mark.parametrize("boundary", ["Open", "Reflective", "Periodic"])
def test_fp64_default_tiling_equals_explicit_tiles(counts, tile, boundary):
    dim = len(counts)
    states = []
    for t in (None, tile):
        sim = torch_gb300.Simulation(rough(counts), [1.0] * dim, t_end=1.0, limiter="Superbee",
                                     boundaries=[boundary] * dim, tile=t)
        for _ in range(3):
            sim.step()
        states.append((sim.state, sim.time))
    np.testing.assert_array_equal(states[0][0], states[1][0])
    assert states[0][1] == states[1][1]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [5, 121, 122, 123, 245, 1000])
def test_1d_default_tiling_equals_whole_warp_tiles(n, precision):
    for boundary in ("Open", "Reflective", "Periodic"):
        states = []
        for t in (None, (256, 1, 1)):
            sim = torch_gb300.Simulation(rough((n,)), [1.0], t_end=1.0, limiter="VanLeer",
                                         boundaries=[boundary], precision=precision, tile=t)
            for _ in range(5):
                sim.step()
            states.append((sim.state, sim.time))
        np.testing.assert_array_equal(states[0][0], states[1][0])
        assert states[0][1] == states[1][1]


@pytest.mark.parametrize("counts,tile,precision", [
    ((132, 9), (124, 1, 32), "fp32"), ((4, 3), (128, 1, 4), "fp32"),
    ((20, 17, 9), (16, 16, 40), "fp32"), ((16, 16, 16), (16, 16, 5), "fp32"),
    ((4, 2, 3), (32, 8, 16), "fp32"), ((34, 11), (32, 1, 4), "fp64"),
    ((18, 5, 6), (32, 4, 32), "fp64"),
])
@pytest.mark.parametrize("boundary", ["Open", "Reflective", "Periodic"])
def test_element_copies_stage_what_tensor_copies_stage(counts, tile, precision, boundary):
    """Grids whose rows allow tensor copies, staged by tensor copies and by one
    asynchronous copy per cell (what rows of other lengths take)."""
    states = []
    for tma in (1, 0):
        sim = torch_gb300.Simulation(rough(counts), [1.0] * len(counts), t_end=1.0,
                                     limiter="MINBEE", boundaries=[boundary] * len(counts),
                                     precision=precision, tile=tile + (0, tma))
        for _ in range(3):
            sim.step()
        states.append(sim.state)
    np.testing.assert_array_equal(states[0], states[1])
