"""Host arrays on their way to the step functions' device (stepfn._as_device),
here with the CPU as the device: every memory form that NumPy calls contiguous is
taken, reversed axes of one cell among them, and the array is left as it was."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from torch_gb300 import stepfn  # noqa: E402

BASE = np.arange(20.0)
FORMS = {
    "plain": BASE.reshape(4, 5),
    "one_row_reversed": BASE[:5].reshape(1, 5)[::-1],
    "one_column_reversed": BASE[:5].reshape(5, 1)[:, ::-1],
    "middle_reversed": BASE.reshape(4, 1, 5)[:, ::-1],
    "reversed": BASE.reshape(4, 5)[::-1, ::-1],
    "fortran": np.asfortranarray(BASE.reshape(4, 5)),
    "strided": np.arange(40.0).reshape(4, 10)[:, ::2],
    "broadcast": np.broadcast_to(np.float64(1.4), (3, 4)),
    "empty": BASE[:0].reshape(0, 5)[::-1],
    "number": np.array(1.4),
    "single": BASE.reshape(4, 5).astype(np.float32),
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_forms_are_taken(form, dtype):
    x = FORMS[form]
    want = np.array(x, dtype=np.float64 if dtype == torch.float64 else np.float32)
    got = stepfn._as_device(x, dtype, torch.device("cpu"))
    assert got.dtype == dtype and got.is_contiguous() and tuple(got.shape) == x.shape
    np.testing.assert_array_equal(got.numpy(), want)
