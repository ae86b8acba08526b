"""Per-cell gamma staged by tensor copies."""


import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import torch_gb300  # noqa: E402
from torch_gb300 import stepfn  # noqa: E402


def rough(counts, seed=3):
    rng = np.random.default_rng(seed)
    shape = tuple(counts[::-1])
    dim = len(counts)
    p = np.empty((dim + 2,) + shape)
    p[0] = 0.5 + rng.random(shape)
    p[1:-1] = 0.4 * (rng.random((dim,) + shape) - 0.5)
    p[-1] = 0.5 + rng.random(shape)
    return p


def test_2d_fp32_step_with_gamma_per_cell():
    """Two 124-cell tiles by tensor copy, gamma as an array: the single
    precision step stays within the L1 criterion of the double one (1e-5)."""
    p = rough((132, 37))
    u = p.copy()
    u[1:3] *= p[0]
    gamma = 1.3 + 0.2 * np.random.default_rng(1).random((37, 132))
    u[3] = p[3] / (gamma - 1) + 0.5 * p[0] * (p[1] ** 2 + p[2] ** 2)
    args = (1 / 132, 1 / 37, 1e-3, gamma, "VanLeer", "Reflective", "Periodic")
    want = stepfn.muscl_hancock_step_2d(u, *args)
    got = stepfn.muscl_hancock_step_2d(u, *args, precision="fp32")
    for c in range(4):
        assert np.abs(got[c] - want[c]).mean() <= 1e-5 * np.abs(want[c]).mean()
