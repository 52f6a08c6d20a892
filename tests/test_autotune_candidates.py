"""The autotuner's candidates stand around the library's defaults."""
import os
import re

from loom_b200 import autotune as AT

HOST = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "loom_b200", "csrc", "host.cuh")


def defaults():
    with open(HOST) as f:
        text = f.read()
    body = text[text.index("struct Tuning {"):]
    return {k: int(v) for k, v in re.findall(r"uint32_t (\w+) = (\d+);", body[:body.index("} tune;")])}


def test_candidates_hold_the_default_and_values_on_both_sides_of_a_line():
    d = defaults()
    for name, values in AT.CANDIDATES.items():
        assert d[name] in values, name
        if name.endswith("_per_sm"):
            assert sum(v < d[name] for v in values) >= 2 and sum(v > d[name] for v in values) >= 2, name
