"""Tiled metric kernels at block edges: sessions on grids one short of, at and
one past the block widths (30 / 126 cells in 2D, 15 x 15 in 3D) against the
oracle, bit for bit in double precision (no boundary state here needs pow), and
single precision against double within the repository's L1 criterion."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402
from oracle import metric as M  # noqa: E402

FACES = {
    "walls": {},
    "periodic": dict(y_min="periodic", y_max="periodic"),
    "mixed": dict(x_min="outflow", x_max="wall"),
}


def waves(counts, seed=5):
    rng = np.random.default_rng(seed)
    shape = tuple(counts[::-1])
    p = np.empty((len(counts) + 2,) + shape)
    p[0] = 0.6 + rng.random(shape)
    p[1:-1] = 0.3 * (rng.random((len(counts),) + shape) - 0.5)
    p[-1] = 0.6 + rng.random(shape)
    return p


def session(counts, faces, precision, limiter):
    dim = len(counts)
    spec = {a + e: "wall" for a in "xyz"[:dim] for e in ("_min", "_max")}
    spec.update(FACES[faces])
    kw = dict(t_end=1.0, limiter=limiter, face_boundaries=spec)
    if dim == 2:  # annulus: y is the azimuth, closed where it is periodic
        kw.update(geometry="annular", origins=[0.5, 0.0])
        lengths = [1.0, 2 * np.pi if faces == "periodic" else 2.0]
    else:  # Cartesian box with face boundaries, or a spherical wedge
        lengths = [1.0, 0.9, 0.8]
        if faces == "mixed":
            kw.update(geometry="spherical", origins=[0.5, 0.6, 0.0])
    return torch_gb300.Simulation(waves(counts), lengths, precision=precision, **kw), lengths


@pytest.mark.parametrize("counts", [(2, 3), (29, 5), (30, 3), (31, 7), (61, 4),
                                    (2, 3, 2), (14, 15, 5), (15, 16, 9), (16, 14, 3), (31, 30, 4)])
@pytest.mark.parametrize("faces", sorted(FACES))
def test_fp64_matches_oracle_bitwise(counts, faces):
    for limiter in ("VanLeer", "Superbee"):
        sim, lengths = session(counts, faces, "fp64", limiter)
        c = sim.config
        ref = M.OracleMetricSimulation(sim.primitive, lengths, t_end=c["t_end"], cfl=c["cfl"],
                                       gamma=c["gamma"], limiter=limiter, geometry=c["geometry"],
                                       origins=c["origins_xyz"], faces=c["face_boundaries"])
        ref.state = sim.state.copy()
        for _ in range(3):
            ref.step()
            sim.step()
        np.testing.assert_array_equal(sim.state, ref.state)
        assert sim.time == ref.time and sim.fallback_steps == ref.fallback_steps
        scale = max(1.0, np.abs(sim.initial_integral).max())
        np.testing.assert_allclose(sim.balance_residual, 0, atol=1e-12 * scale)


@pytest.mark.parametrize("counts", [(125, 6), (126, 9), (127, 5), (15, 16, 9), (31, 14, 33)])
@pytest.mark.parametrize("faces", sorted(FACES))
def test_fp32_tracks_fp64(counts, faces):
    for limiter in ("VanLeer", "Albada", "MINBEE", "Superbee", "Unos"):
        s64, _ = session(counts, faces, "fp64", limiter)
        s32, _ = session(counts, faces, "fp32", limiter)
        for _ in range(3):
            s64.step()
            s32.step()
        for row in (0, -1):
            want = s64.state[row]
            assert np.abs(s32.state[row] - want).mean() <= 1e-5 * np.abs(want).mean()
