"""The library's own tile named explicitly (as the autotuner returns it): the batch
it gives equals the default batch bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from torch_gb300 import autotune  # noqa: E402
from torch_gb300.batch import Batch, Grid, default_tile  # noqa: E402


def grids(counts, precision):
    rng = np.random.default_rng(2)
    out = []
    for k in range(2):
        shape = tuple(c + 3 * k for c in counts[::-1])
        p = np.zeros((len(counts) + 2,) + shape)
        p[0] = 0.5 + rng.random(shape)
        p[1] = 0.2 * rng.random(shape)
        p[-1] = 0.5 + rng.random(shape)
        out.append(Grid(p, [1.0] * len(counts), precision=precision, t_end=1.0))
    return out


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("counts", [(300,), (70, 41), (1030, 600), (21, 18, 9), (60, 50, 40)])
def test_named_tile_equals_default(counts, precision):
    a, b = grids(counts, precision), grids(counts, precision)
    tile = default_tile(a)
    for gs, t in ((a, None), (b, tile)):
        batch = Batch(gs, tile=t)
        batch.advance(4)
        batch.refresh()
        batch.close()
    for g, h in zip(a, b):
        assert g.time == h.time and g.steps == 4
        np.testing.assert_array_equal(g.state_host(), h.state_host())


def test_tuner_offers_it_first(monkeypatch):
    seen = []
    time_config = autotune.time_config
    monkeypatch.setattr(autotune, "time_config",
                        lambda gs, t, *a: seen.append(t) or time_config(gs, t, *a))
    gs = grids((70, 41), "fp64")
    tile = autotune.tune(gs, steps=1, warmup=1, use_cache=False)
    assert seen[0] == default_tile(gs) and tile in seen
