"""Loads of the kernels that are launched over the end of their predecessor
(programmatic dependent launch): non-coherent loads (__ldg, ro) promise data that
nothing writes during the kernel's lifetime, which there begins before the
predecessor has ended.  The sources of those kernels may use them for the
geometry factors alone, which are written once at bind."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "torch_gb300" / "csrc"
CONSTANT = ("&A.ff[", "&A.vf[")


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_tiled_metric_kernels_read_the_state_with_ordinary_loads():
    text = code("tfv_metric_tile.cuh")
    args = re.findall(r"\bro\(([^;]{0,24})", text)
    assert args
    for a in args:
        assert a.startswith(CONSTANT), a
    assert "__ldg" not in text and "ld.global.nc" not in text


def test_step_kernels_use_no_read_only_loads():
    for name in ("tfv_kernels.cuh", "tfv_1d.cuh", "tfv_inst.inc", "tfv_f64.cu",
                 "tfv_metric_tile_f64.cu"):
        text = code(name)
        assert "__ldg" not in text and "ld.global.nc" not in text
        assert "__restrict__" not in text and not re.search(r"\bro\(", text)
