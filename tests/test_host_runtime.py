"""What the library's host code asks of the CUDA runtime, checked without a GPU: its object files linked with a runtime of
the tests' own (tests/cpp/fake_cuda.hpp) that counts kernels instead of running them, copies as late as a runtime may, and
keeps the sum of what is allocated."""

import glob
import os
import subprocess

import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def run():
    from thea_gb300 import build as B
    B.build()
    objects = sorted(glob.glob(os.path.join(B.BUILD, "*.o")))
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc())))

    def go(name, *args):
        src = os.path.join(ROOT, "tests", "cpp", name + ".cpp")
        out = os.path.join(ROOT, "tests", "cpp", "_build", name)
        os.makedirs(os.path.dirname(out), exist_ok=True)
        r = subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(cuda, "include"), src] + objects +
                           ["-o", out, "-lpthread", "-ldl", "-Wl,--unresolved-symbols=ignore-all"],
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-4000:]
        r = subprocess.run([out] + list(args), capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout

    return go


def test_segment_cuts_outlive_their_copy(run):
    assert "segment cuts whole" in run("segment_cuts_check")


def test_batches_fetch_work_as_asked(run):
    assert "fetches as asked" in run("batch_fetch_check")


def test_mixed_precision_scratch_is_bounded(run):
    assert "batches bounded" in run("scratch_check")


def test_build_scratch_is_bounded(run):
    assert "builds bounded" in run("scratch_check", "build")


def test_small_calls_ask_little_of_the_runtime(run):
    assert "small calls are small" in run("small_call_check")


def test_closest_point_routes(run):
    assert "routes as measured" in run("closest_routes_check")
