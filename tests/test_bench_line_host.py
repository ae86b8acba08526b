"""The benchmark's result line does not grow with the number of comparisons."""

import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def rows(count):
    return [dict(l1_rho=2.9353285191118725e-07 * (1 + k % 7), linf_rho=1.8238264368086732e-05,
                 l1_p=7.391792257451918e-08, linf_p=7.538307843502068e-06, rid=k, dim=3, n=223,
                 steps=509) for k in range(count)]


def test_comparisons_are_summarised(capsys):
    few, many = bench.compared("x", rows(8)), bench.compared("x", rows(128))
    assert len(json.dumps(many)) <= len(json.dumps(few)) + 8
    assert many["compared"] == 128 and many["worst"]["rid"] == 6
    assert many["l1_rho_max"] == many["worst"]["l1_rho"]
    out = capsys.readouterr()
    assert out.out == ""
    assert len(json.loads(out.err.splitlines()[1])["x"]) == 128


def test_legs_put_no_list_of_comparisons_into_the_line():
    text = open(os.path.join(ROOT, "bench.py")).read()
    for leg in ("batched_leg", "served_leg"):
        body = text[text.index("def " + leg):]
        body = body[:body.index("\ndef ", 1)]
        assert "=errors" not in body and "for e in errors]" not in body
        assert body.count("compared(") == 1
