"""March of the tiled metric kernels through chunks of several planes: grids whose
step is tiled in chunks of 2 to 12 planes (asserted), with several blocks, a
remainder plane and chunks that start anywhere.  Double precision (2D) equals the
oracle bit for bit.  Single precision (2D and 3D) is compared with the
double-precision session cell by cell on every row: three steps are six stages of
some fifty roundings on the way of a value, 300 units of 6e-8, so 2e-5 of the row's
largest value; sums over faces and cells within 1e-5 of the largest of them, and the
balance within six roundings of every cell, 1e-6 of the total."""

import ctypes as C

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
        if faces != "periodic":
            kw.update(geometry="spherical", origins=[0.5, 0.6, 0.0])
    return torch_gb300.Simulation(waves(counts), lengths, precision=precision, **kw), lengths


def tiling(sim):
    lib = torch_gb300._lib.load()
    t = (C.c_int32 * 4)()
    torch_gb300._lib.check(lib.tfv_metric_tile(sim._engine.handle, t))
    return tuple(t)


@pytest.mark.parametrize("counts,width,chunk", [
    ((256, 193), 32, 2), ((400, 301), 32, 2), ((512, 257), 32, 3), ((1000, 301), 128, 4)])
@pytest.mark.parametrize("faces", sorted(FACES))
@pytest.mark.parametrize("limiter", ["VanLeer", "Superbee"])
def test_fp64_matches_oracle_bitwise(counts, width, chunk, faces, limiter):
    sim, lengths = session(counts, faces, "fp64", limiter)
    if torch.cuda.get_device_properties(0).multi_processor_count == 152:
        assert tiling(sim)[:3] == (width, 1, chunk)
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


@pytest.mark.parametrize("counts,width,chunk", [
    ((400, 301), 128, 2), ((512, 257), 128, 3), ((1000, 301), 128, 4),
    ((46, 45, 64), 16, 3), ((64, 48, 49), 16, 4), ((61, 46, 100), 16, 8), ((128, 96, 97), 16, 12)])
@pytest.mark.parametrize("faces", sorted(FACES))
@pytest.mark.parametrize("limiter", ["VanLeer", "Superbee"])
def test_fp32_tracks_fp64_per_cell(counts, width, chunk, faces, limiter):
    s64, _ = session(counts, faces, "fp64", limiter)
    s32, _ = session(counts, faces, "fp32", limiter)
    if torch.cuda.get_device_properties(0).multi_processor_count == 152:
        assert tiling(s32)[0] == width and tiling(s32)[2] == chunk
    if len(counts) == 3:
        assert tiling(s64) == (0, 0, 0, 0)  # separate kernels: another code path
    for _ in range(3):
        s64.step()
        s32.step()
    want = s64.state
    axes = tuple(range(1, want.ndim))
    scale = np.abs(want).max(axis=axes, keepdims=True)
    assert (np.abs(s32.state - want) / scale).max() <= 2e-5
    for a, b in ((s32.boundary_integral, s64.boundary_integral),
                 (s32.source_integral, s64.source_integral)):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-5 * max(np.abs(b).max(), 1e-30))
    total = np.abs(s32.initial_integral).max()
    np.testing.assert_allclose(s32.balance_residual, 0, atol=1e-6 * total)
