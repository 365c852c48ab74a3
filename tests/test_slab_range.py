"""The interval that a slab's range is taken from (thea_gb300/csrc/slab_range.cuh), compiled on the host and checked against
exact values rounded outwards (tests/cpp/slab_range_check.cpp)."""

import os
import subprocess

from tests.conftest import ROOT


def test_slab_ranges_hold_and_are_tight():
    src = os.path.join(ROOT, "tests", "cpp", "slab_range_check.cpp")
    out = os.path.join(ROOT, "tests", "cpp", "_build", "slab_range_check")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", src, "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "ranges hold and are tight" in r.stdout
