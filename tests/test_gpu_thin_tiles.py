"""3D tiles one cell high: the second row of tiles has one ghost row in its halo.
States equal those of other tile shapes of the same kernel, bit for bit, on rows
that a tensor copy can stage and on rows that it cannot."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402


def rough(counts, seed=11):
    rng = np.random.default_rng(seed)
    shape = tuple(counts[::-1])
    p = np.empty((5,) + shape)
    p[0] = 0.5 + rng.random(shape)
    p[1:-1] = 0.4 * (rng.random((3,) + shape) - 0.5)
    p[-1] = 0.5 + rng.random(shape)
    return p


@pytest.mark.parametrize("counts", [(33, 5, 4), (32, 4, 3), (36, 2, 5), (65, 3, 2)])
@pytest.mark.parametrize("precision,thin,other", [
    ("fp64", (32, 1, 2), (32, 4, 32)), ("fp32", (32, 1, 2), (32, 2, 8)),
])
@pytest.mark.parametrize("boundary", ["Open", "Reflective", "Periodic"])
def test_one_cell_high_tiles(counts, precision, thin, other, boundary):
    states = []
    for tile in (thin, other):
        sim = torch_gb300.Simulation(rough(counts), [1.0] * 3, t_end=1.0, limiter="Superbee",
                                     boundaries=[boundary] * 3, precision=precision, tile=tile)
        for _ in range(3):
            sim.step()
        states.append((sim.state, sim.time, sim.fallback_steps))
    np.testing.assert_array_equal(states[0][0], states[1][0])
    assert states[0][1:] == states[1][1:]
