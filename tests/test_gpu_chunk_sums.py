"""Balances under the default (short) single-precision chunks: boundary sums,
integrals and the balance residual equal those of the longest chunk up to the
order of their double-precision sums.  The fluxes and states that are summed are the
same bit for bit; 1e5 double-precision additions in another order move a sum by at
most 1e5 * 1.1e-16 of the sum of magnitudes, 1e-11 (boundaries: 1e4 faces, 1e-12)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402


def flow(counts):
    axes = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in counts], indexing="ij")
    phase = sum((k + 1) * a for k, a in enumerate(axes)).transpose()
    p = np.zeros((len(counts) + 2,) + phase.shape)
    p[0] = 1 + 0.3 * np.sin(5 * phase)
    p[1:-1] = 0.4  # through every boundary
    p[-1] = 1 + 0.4 * np.cos(5 * phase)
    return p


@pytest.mark.parametrize("counts,tile", [
    ((24, 24, 24), (16, 16, 40)), ((33, 17, 19), (16, 16, 40)), ((100, 90, 5), (16, 16, 40)),
    ((48, 48), (124, 1, 32)), ((125, 3), (124, 1, 32)), ((123, 257), (124, 1, 32)),
])
@pytest.mark.parametrize("bc", ["Open", "Reflective", "Periodic"])
def test_balances_match_longest_chunk(counts, tile, bc):
    kw = dict(t_end=10.0, precision="fp32", limiter="VanLeer", boundaries=[bc] * len(counts))
    a = torch_gb300.Simulation(flow(counts), [1.0] * len(counts), **kw)
    b = torch_gb300.Simulation(flow(counts), [1.0] * len(counts), tile=tile, **kw)
    for _ in range(4):
        a.step()
        b.step()
    np.testing.assert_array_equal(a.state, b.state)
    total = np.abs(b.initial_integral).max()
    scale = max(np.abs(b.boundary_integral).max(), 1e-3 * total)
    np.testing.assert_allclose(a.boundary_integral, b.boundary_integral, rtol=0,
                               atol=1e-12 * scale)
    np.testing.assert_allclose(a.integral, b.integral, rtol=0, atol=1e-11 * total)
    np.testing.assert_allclose(a.balance_residual, b.balance_residual, rtol=0, atol=2e-11 * total)
