"""Reaction half steps and the fused transport + reaction pass at tile edges:
sessions on grids one short of, at and one past the tile widths against the
oracle (rtol 1e-10, as every reactive comparison: exp's last bit differs)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402
from oracle.session import OracleSimulation  # noqa: E402


def hot_spot(counts):
    mesh = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in counts[::-1]], indexing="ij")
    r2 = sum((m - 0.4) ** 2 for m in mesh)
    p = np.zeros((len(counts) + 2,) + tuple(counts[::-1]))
    p[0] = 1.0
    p[1] = 30.0
    p[-1] = np.where(r2 < 0.1, 3e6, 101325.0)
    return p


@pytest.mark.parametrize("counts", [(29, 3), (30, 5), (31, 4), (9, 7, 5), (10, 8, 2), (15, 17, 3)])
@pytest.mark.parametrize("model,boundary", [("znd", "Reflective"), ("arrhenius", "Periodic"),
                                            ("arrhenius", "Open")])
def test_reactive_sessions_at_tile_edges(counts, model, boundary):
    dim = len(counts)
    kw = dict(t_end=1.0, limiter="MINBEE", reactive=True, kinetic_model=model,
              boundaries=[boundary] * dim)
    ref = OracleSimulation(hot_spot(counts), [1.0] * dim, **kw)
    gpu = torch_gb300.Simulation(hot_spot(counts), [1.0] * dim, **kw)
    for _ in range(4):
        ref.step()
        gpu.step()
    scale = np.abs(ref.state).max(axis=tuple(range(1, dim + 1)), keepdims=True)
    assert np.all(np.abs(gpu.state - ref.state) <= 1e-10 * scale)
    np.testing.assert_allclose(gpu.lam, ref.lam, rtol=1e-10, atol=1e-14)
    if model == "znd":
        np.testing.assert_allclose(gpu.beta, ref.beta, rtol=1e-10, atol=1e-14)
    np.testing.assert_allclose(gpu.source_integral[-1], ref.source_integral[-1], rtol=1e-8)


@pytest.mark.parametrize("counts", [(15, 17, 41), (16, 16, 40), (17, 15, 5)])
def test_fp32_ignition_at_tile_edges_tracks_fp64(counts):
    """Single precision within the L1 criterion (1e-5) of double precision."""
    p = hot_spot(counts)
    p[1] = 0.0
    p[-1] = np.where(p[-1] > 1e6, 3.0, 1.0)
    kw = dict(t_end=1.0, gamma=1.2, reactive=True, limiter="Albada",
              chemistry=dict(closure="nondimensional", q_heat=20.0, activation_energy=25.0,
                             pre_exponential=1e3))
    s64 = torch_gb300.Simulation(p, [1, 1, 1], **kw)
    s32 = torch_gb300.Simulation(p, [1, 1, 1], precision="fp32", **kw)
    for _ in range(5):
        s64.step()
        s32.step()
    assert np.abs(s32.state[0] - s64.state[0]).mean() <= 1e-5 * np.abs(s64.state[0]).mean()
    assert np.abs(s32.lam - s64.lam).mean() <= 1e-5
