"""The cable solve's quotients by FMA are IEEE quotients wherever its range checks accept them.

tests/quotients.cu compares them bit for bit with division: random significands, divisors next to
the all-ones significand (the method's exception) and to one, quotients next to short numbers, and
exponents at the edges of the accepted ranges.  On the CPU the reciprocal's seed is the documented
20 bits; on the GPU it is the instruction's.
"""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mind.jl_b200", "csrc")
FAMILIES = range(5)


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    out = str(tmp_path_factory.mktemp("quotients") / "quotients.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-fPIC", "-Xcompiler", "-ffp-contract=off", "-shared", "-cudart", "shared", "-I", CSRC,
                    "-o", out, os.path.join(HERE, "quotients.cu")], check=True)
    return ctypes.CDLL(out)


def _check(call, count, family):
    counts = (ctypes.c_ulonglong * 3)()
    assert not call(ctypes.c_uint64(12345 + family), ctypes.c_uint64(count), family, counts)
    accepted, wrong, refused_ordinary = counts
    assert wrong == 0 and refused_ordinary == 0, list(counts)
    assert accepted > count // 4, list(counts)


@pytest.mark.parametrize("family", FAMILIES)
def test_quotients_on_the_cpu(checks, family):
    checks.check_on_host.restype = None
    _check(checks.check_on_host, 400_000, family)


@pytest.mark.gpu
@pytest.mark.parametrize("family", FAMILIES)
def test_quotients_on_the_gpu(checks, family):
    _check(checks.check_on_device, 200_000_000, family)
