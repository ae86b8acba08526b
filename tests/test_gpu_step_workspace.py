"""Workspace of the step function: the size query is not smaller than the plan
that a step makes, and it costs less than making one."""

import ctypes as C
import statistics
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from torch_gb300 import _lib  # noqa: E402
from torch_gb300.session import make_config  # noqa: E402


def config(counts):
    dim = len(counts)
    return make_config(dim, list(counts), [1.0] * dim, ["Open"] * dim, t_end=1.0, cfl=0.4,
                       gamma=1.4, limiter="VanLeer", max_steps=1)


def query(cfg, prec):
    ws = C.c_size_t()
    _lib.check(_lib.load().tfv_step_workspace_size(C.byref(cfg), prec, C.byref(ws)))
    return ws.value


def create(cfg, prec):
    h = C.c_void_p()
    _lib.check(_lib.load().tfv_batch_create(cfg.dim, prec, 1, C.byref(cfg), None, C.byref(h)))
    return h


@pytest.mark.parametrize("prec", [_lib.TFV_FP64, _lib.TFV_FP32])
@pytest.mark.parametrize("counts", [
    (5,), (1000,), (7, 5), (192, 192), (300, 260), (1000, 700), (2048, 2048), (4096, 4096),
    (9, 7, 5), (64, 64, 64), (100, 90, 110), (160, 150, 170), (256, 256, 256), (300, 280, 260)])
def test_bounds_the_plan(counts, prec):
    lib = _lib.load()
    cfg = config(counts)
    h = create(cfg, prec)
    plan = C.c_size_t()
    _lib.check(lib.tfv_batch_workspace_size(h, C.byref(plan)))
    lib.tfv_batch_destroy(h)
    assert plan.value <= query(cfg, prec)


def test_costs_less_than_a_plan():
    cfg = config((8192, 4096))
    plans, queries = [], []
    for _ in range(9):
        t = time.perf_counter()
        h = create(cfg, _lib.TFV_FP32)
        plans.append(time.perf_counter() - t)
        _lib.load().tfv_batch_destroy(h)
        t = time.perf_counter()
        query(cfg, _lib.TFV_FP32)
        queries.append(time.perf_counter() - t)
    assert statistics.median(queries) < statistics.median(plans)
