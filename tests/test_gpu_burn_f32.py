"""Single-precision reactive steps (the fused transport and reaction pass) against
double precision, in 2D and 3D, for both kinetic models and closures' gamma forms:
density and energy within the repository's L1 criterion (1e-5), fractions within
1e-5 on average, and the energy source, summed in single precision with
compensation per column, within what those fractions allow: 1e-5 of the heat of all
the fuel, and four roundings of every cell's energy a step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402

STEPS = 5
Q = 20.0


@pytest.mark.parametrize("counts", [(31, 30), (125, 9), (124, 40), (15, 17, 41), (16, 16, 40),
                                    (33, 18, 5)])
@pytest.mark.parametrize("model", ["arrhenius", "znd"])
@pytest.mark.parametrize("boundary", ["Open", "Reflective", "Periodic"])
def test_tracks_double_precision(counts, model, boundary):
    dim = len(counts)
    mesh = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in counts[::-1]], indexing="ij")
    r2 = sum((m - 0.4) ** 2 for m in mesh)
    p = np.zeros((dim + 2,) + tuple(counts[::-1]))
    p[0] = 1.0
    p[-1] = 1.0 + 2.0 * np.exp(-r2 / 0.3)
    kw = dict(t_end=1.0, gamma=1.2, reactive=True, limiter="Albada", kinetic_model=model,
              boundaries=[boundary] * dim,
              chemistry=dict(closure="nondimensional", q_heat=Q, activation_energy=25.0,
                             pre_exponential=5e4))
    if model == "znd":
        # the fastest cells burn from the first half step on: where nothing burnt in it, the
        # CFL check of the heated state would be a tie that rounding decides, and the
        # two precisions would take different steps
        kw["beta_init"] = np.where(r2 < 0.05, 0.0, 0.01)
    s64, s32 = (torch_gb300.Simulation(p, [1.0] * dim, precision=prec, **kw)
                for prec in ("fp64", "fp32"))
    for _ in range(STEPS):
        s64.step()
        s32.step()
    assert abs(s32.time - s64.time) <= 1e-5 * s64.time
    for r in (0, -1):
        want = s64.state[r]
        assert np.abs(s32.state[r] - want).mean() <= 1e-5 * np.abs(want).mean()
    assert np.abs(s32.lam - s64.lam).mean() <= 1e-5
    if model == "znd":
        assert np.abs(s32.beta - s64.beta).mean() <= 1e-5
    mass, energy = s64.initial_integral[0], s64.initial_integral[-1]
    released = s64.source_integral[-1]
    allowed = 1e-5 * Q * mass + 4 * STEPS * 2.0 ** -24 * (energy + released)
    assert released > 20 * allowed  # enough burnt to tell
    assert abs(s32.source_integral[-1] - released) <= allowed
    np.testing.assert_array_equal(s32.source_integral[:-1], 0)
