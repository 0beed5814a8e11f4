"""bench.py's lines are strict JSON whatever the samples hold: an empty sample's chi^2 is not a number,
and JSON has no form for that but null."""
import json

import numpy as np

import bench
from pacuda_b200 import unweight


def strict(text):
    def refuse(name):
        raise ValueError(name)

    return json.loads(text, parse_constant=refuse)


def test_an_empty_sample_s_chi2():
    w = np.array([1.0, 2.0, 3.0])
    c2, bins = unweight.chi2_against(w, w, np.zeros(0), np.zeros(0), np.linspace(0.0, 4.0, 5))
    assert bins == 0
    line = bench.json_line({"value": 2.5, "chi2": {"family": {"pt": round(c2 / max(1, bins), 3)}}})
    assert "\n" not in line
    assert strict(line) == {"value": 2.5, "chi2": {"family": {"pt": None}}}


def test_every_kind_of_value():
    value = {"a": [1, 2.5, (float("inf"), -0.0)], "b": None, "c": True, "d": "NaN", "e": np.float64("nan"), "f": 1e308}
    assert strict(bench.json_line(value)) == {"a": [1, 2.5, [None, 0.0]], "b": None, "c": True, "d": "NaN", "e": None,
                                              "f": 1e308}
