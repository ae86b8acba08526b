"""Single-precision curvilinear and face-boundary sessions on states where the
single-precision forms of the tiled kernels could part from the double-precision
solution: gamma so close to one that gamma - 1 loses digits, and pressures whose
differences have no square in single precision.  The measure is the repository's
L1 criterion (mean error below 1e-5 of the row's mean)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402


def sessions(p, limiter="VanLeer", **kw):
    dim = p.ndim - 1
    faces = {a + e: "periodic" for a in "xyz"[:dim] for e in ("_min", "_max")}
    return [torch_gb300.Simulation(p, [1.0] * dim, t_end=1.0, limiter=limiter, precision=prec,
                                   face_boundaries=faces, **kw) for prec in ("fp64", "fp32")]


def stream(counts, pressure, speed):
    """A pressure and density wave carried along x, y and z."""
    axes = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in counts], indexing="ij")
    phase = 2 * np.pi * sum(axes).transpose()
    p = np.empty((len(counts) + 2,) + phase.shape)
    p[0] = 1 + 0.2 * np.sin(phase)
    p[1:-1] = speed
    p[-1] = pressure * (1 + 0.4 * np.cos(phase))
    return p


def errors(s64, s32):
    want = s64.state
    return [np.abs(s32.state[r] - want[r]).mean() / np.abs(want[r]).mean() for r in (0, -1)]


@pytest.mark.parametrize("counts", [(32, 24), (32, 24, 16)])
def test_gamma_close_to_one(counts):
    """An energy formed with another gamma - 1 than the pressure carries an error
    of 1.7e-4 of the energy carried over: 3e-5 in ten steps, which carry a fifth."""
    s64, s32 = sessions(stream(counts, 1.0, 10.0), gamma=1.0001)
    for _ in range(10):
        s64.step()
        s32.step()
    assert max(errors(s64, s32)) <= 1e-5


@pytest.mark.parametrize("limiter", ["VanLeer", "Albada", "MINBEE", "Superbee", "Unos"])
@pytest.mark.parametrize("counts", [(32, 24), (32, 24, 16)])
def test_pressures_of_1e20(counts, limiter):
    """Differences of neighbouring pressures around 1e19 to 1e20, whose product is
    beyond single precision: slopes stay finite and the step second order."""
    s64, s32 = sessions(stream(counts, 3e20, 1e9), limiter=limiter)
    for _ in range(4):
        s64.step()
        s32.step()
    assert s64.fallback_steps == 0 and s32.fallback_steps == 0
    assert max(errors(s64, s32)) <= 1e-5
