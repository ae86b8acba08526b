"""Single-precision default chunks: grids that take short chunks (one cell thick
to three tiles) give the same state, bit for bit, as the longest chunk does, and
conserved sums agree to the rounding of their double-precision order."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402


def smooth(counts):
    axes = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in counts], indexing="ij")
    phase = sum((k + 1) * a for k, a in enumerate(axes)).transpose()
    p = np.zeros((len(counts) + 2,) + phase.shape)
    p[0] = 1 + 0.3 * np.sin(2 * np.pi * phase)
    p[1] = 0.2 * np.cos(2 * np.pi * phase)
    p[-1] = 1 + 0.4 * np.cos(2 * np.pi * phase)
    return p


@pytest.mark.parametrize("counts,tile", [
    ((24, 24, 24), (16, 16, 40)), ((33, 17, 19), (16, 16, 40)), ((64, 64, 64), (16, 16, 40)),
    ((100, 90, 5), (16, 16, 40)), ((16, 16, 256), (16, 16, 40)),
    ((48, 48), (124, 1, 32)), ((125, 3), (124, 1, 32)), ((123, 257), (124, 1, 32)),
    ((512, 300), (124, 1, 32)),
])
def test_default_chunks_match_longest(counts, tile):
    lengths = [1.0] * len(counts)
    for bc in ("Open", "Periodic"):
        kw = dict(t_end=10.0, precision="fp32", limiter="Superbee",
                  boundaries=[bc] * len(counts))
        a = torch_gb300.Simulation(smooth(counts), lengths, **kw)
        b = torch_gb300.Simulation(smooth(counts), lengths, tile=tile, **kw)
        for _ in range(4):
            a.step()
            b.step()
        np.testing.assert_array_equal(a.state, b.state)
        assert a.time == b.time and a.fallback_steps == b.fallback_steps
