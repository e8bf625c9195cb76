"""Threads per tree by tree count and depth, on 148 SMs of three CTAs."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CTAS = 444


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("pprf") / "libpprf_rule.so")
    subprocess.check_call([nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                           "-gencode", "arch=compute_100a,code=sm_100a",
                           os.path.join(ROOT, "tests", "cpp", "pprf_rule.cu"), "-o", so])
    lib = ctypes.CDLL(so)
    lib.pprf_rule.argtypes = [ctypes.c_uint64, ctypes.c_int, ctypes.c_uint64]
    return lambda t, h: lib.pprf_rule(t, h, CTAS)


@pytest.mark.parametrize("h", [1, 9, 12, 13, 20])
def test_no_more_than_a_tree_per_cta(rule, h):
    assert rule(1, h) == rule(CTAS, h) == 256


@pytest.mark.parametrize("h", [12, 13, 14, 20])
def test_deep_trees_of_a_few_waves(rule, h):
    """One by one where two groups per CTA would share them out badly."""
    for t in (533, 592, 740, 963, 1036, 1184):
        assert rule(t, h) == 256, t
    for t in (445, 532, 741, 888, 962, 1185, 1332):
        assert rule(t, h) == 128, t


def test_shallow_and_many(rule):
    for h in (1, 8, 11):
        assert rule(445, h) == rule(1332, h) == 128
        assert rule(1333, h) == rule(60000, h) == 64
    assert rule(1333, 12) == 64 and rule(1333, 13) == rule(60000, 13) == 128
