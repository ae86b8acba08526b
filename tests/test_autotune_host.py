"""The autotuner's choice and its cache, without a GPU (times are made up): the
library's own tile is a candidate of every batch, comes back as a tile that a batch
can be given, and wins where it is the fastest; plans of other limiters, chemistry
or library sources are not taken from the cache."""

import ctypes as C
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")
from torch_gb300 import _lib, autotune  # noqa: E402
from torch_gb300.session import make_config  # noqa: E402


def grid(counts, precision, limiter="VanLeer", reactive=False, model="arrhenius"):
    dim = len(counts)
    cfg = make_config(dim, list(counts), [1.0] * dim, ["Open"] * dim, t_end=1.0, cfl=0.4,
                      gamma=1.4, limiter=limiter, max_steps=10)
    cfg.reactive, cfg.kinetic_model = int(reactive), _lib.MODELS[model]
    return SimpleNamespace(dim=dim, counts=list(counts), precision=precision, cfg=cfg,
                           reactive=reactive, device="cuda:0")


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d=None: "chip")
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d=None: SimpleNamespace(multi_processor_count=152))
    monkeypatch.setattr(autotune, "CACHE", tmp_path / "plans.json")
    calls = []

    def fastest(best):
        def time_config(grids, tile, steps=4, warmup=2):
            calls.append(tile)
            return 1.0 if best(tile) else 2.0
        monkeypatch.setattr(autotune, "time_config", time_config)
        return calls
    return fastest


CASES = [((1000,), "fp32"), ((1000,), "fp64"), ((64, 64), "fp64"), ((256, 256), "fp64"),
         ((1024, 1024), "fp64"), ((48, 40, 32), "fp64"), ((160, 160, 160), "fp64"),
         ((64, 64), "fp32"), ((512, 512), "fp32"), ((32, 32, 32), "fp32"),
         ((128, 128, 128), "fp32")]


def create(g, tile):
    lib = _lib.load()
    h, ws, t = C.c_void_p(), C.c_size_t(), _lib.Tile()
    code = lib.tfv_batch_create(g.dim, _lib.TFV_FP64 if g.precision == "fp64" else _lib.TFV_FP32,
                                1, C.byref(g.cfg), C.byref(_lib.Tile(*tile)) if tile else None,
                                C.byref(h))
    if code:
        return code, None, None
    lib.tfv_batch_workspace_size(h, C.byref(ws))
    lib.tfv_batch_tile(h, C.byref(t))
    lib.tfv_batch_destroy(h)
    return code, ws.value, (t.tx, t.ty, t.chunk, t.persistent_ctas, t.tma)


@pytest.mark.parametrize("counts,precision", CASES)
def test_own_tile_is_reached(tuner, counts, precision):
    g = grid(counts, precision)
    code, want_bytes, own = create(g, None)
    assert code == _lib.TFV_OK
    calls = tuner(lambda t: t == own)
    assert autotune.tune([g]) == own
    assert calls.count(own) == 1
    assert create(g, own) == (_lib.TFV_OK, want_bytes, own)  # the same batch when named
    # another candidate wins where it is faster
    other = next(t for t in calls if t != own)
    tuner(lambda t: t == other)
    assert autotune.tune([g], use_cache=False) == other


def test_cache_is_per_limiter_chemistry_and_sources(tuner, monkeypatch):
    calls = tuner(lambda t: True)
    base = grid((64, 64), "fp32")
    first = autotune.tune([base])
    n = len(calls)
    assert autotune.tune([base]) == first and len(calls) == n  # cached
    for g in (grid((64, 64), "fp32", limiter="Superbee"),
              grid((64, 64), "fp32", reactive=True),
              grid((64, 64), "fp32", reactive=True, model="znd")):
        n = len(calls)
        autotune.tune([g])
        assert len(calls) > n
    monkeypatch.setattr(autotune, "_sources", lambda: "other kernels")
    n = len(calls)
    autotune.tune([base])
    assert len(calls) > n


@pytest.mark.parametrize("dim,precision,tile", [
    (2, "fp64", (31, 1, 2)), (2, "fp64", (124, 1, 32)), (3, "fp64", (10, 9, 4)),
    (3, "fp64", (12, 12, 8)), (1, "fp64", (100, 1, 1)), (1, "fp32", (123, 1, 1)),
])
def test_other_shapes_stay_refused(dim, precision, tile):
    g = grid((64,) * dim, precision)
    assert create(g, tile + (0, 1))[0] == _lib.TFV_EINVAL
