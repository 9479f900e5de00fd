"""The bytes a benchmark line holds against a kernel's time are those of the
work its launches did."""

import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("launches,passes,share", [(1000, 500, 0.5), (460, 460, 1.0), (20, 0, 1.0)])
def test_a_schur_pass_is_counted_once(bench, launches, passes, share):
    stats = {"schur_blocks": (launches, 100.0), "chi2": (40, 1.0)}
    if passes:
        stats["schur_landmark"] = (passes, 5.0)
    assert bench.passes_per_launch("schur_blocks", stats) == share
    assert bench.passes_per_launch("chi2", stats) == 1.0
