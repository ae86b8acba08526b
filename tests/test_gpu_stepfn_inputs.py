"""Step function on host arrays of every memory form (plain, read-only, reversed,
Fortran order, sliced, single precision): the same values and an input that is
left as it was."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from torch_gb300.stepfn import muscl_hancock_step_2d  # noqa: E402


def state(ny=37, nx=41):
    rng = np.random.default_rng(3)
    u = np.empty((4, ny, nx))
    u[0] = 1 + 0.3 * rng.random((ny, nx))
    u[1:3] = 0.1 * (rng.random((2, ny, nx)) - 0.5)
    u[3] = 2.5 + 0.5 * rng.random((ny, nx))
    return u


def read_only(u):
    v = u.copy()
    v.flags.writeable = False
    return v


FORMS = {
    "plain": lambda u: u.copy(),
    "read_only": read_only,
    "reversed": lambda u: np.ascontiguousarray(u[:, ::-1, ::-1])[:, ::-1, ::-1],
    "fortran": lambda u: np.asfortranarray(u),
    "sliced": lambda u: np.repeat(u, 2, axis=2)[:, :, ::2],
}


@pytest.mark.parametrize("form", sorted(FORMS))
def test_forms_agree(form):
    u = state()
    want = muscl_hancock_step_2d(torch.as_tensor(u.copy(), device="cuda"), 0.1, 0.1, 1e-3,
                                 return_fluxes=True)
    x = FORMS[form](u)
    got = muscl_hancock_step_2d(x, 0.1, 0.1, 1e-3, return_fluxes=True)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w.cpu().numpy())
    np.testing.assert_array_equal(x, u)


def test_single_precision_array():
    u = state().astype(np.float32)
    want = muscl_hancock_step_2d(u.astype(float), 0.1, 0.1, 1e-3)
    np.testing.assert_array_equal(muscl_hancock_step_2d(u, 0.1, 0.1, 1e-3), want)
