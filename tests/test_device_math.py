"""Divisions, square roots and the like are the language's operations and
CUDA's functions, so their rounding is the documented one: no kernel builds
one from the hardware's approximate instructions."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "diff_fem_b200" / "csrc"
APPROXIMATE = re.compile(r"\b(rcp|rsqrt|sqrt|div|ex2|lg2|sin|cos|tanh)\.(approx|full)\b|__(frcp|fdividef|nv_)\w*")


def test_no_arithmetic_from_approximate_instructions():
    found = [(p.name, n) for p in sorted(CSRC.iterdir()) for n, line in enumerate(p.read_text().splitlines(), 1)
             if APPROXIMATE.search(line)]
    assert not found, found
