"""Large copies from pageable memory (csrc/upload.hpp): when the pinned buffers are made, and every byte.

Built with g++ against tests/uploads.cpp, which stands in for the CUDA runtime (bound to it before any
runtime that the process has loaded).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mind.jl_b200", "csrc")
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("uploads") / "uploads.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I", CSRC, "-I",
                    "/usr/local/cuda/include",
                    "-o", out, os.path.join(HERE, "uploads.cpp")], check=True)
    lib = ctypes.CDLL(out)
    lib.uploader_new.restype = ctypes.c_void_p
    lib.uploader_copy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t]
    lib.set_registered.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    for name in ("uploader_release", "uploader_delete"):
        getattr(lib, name).argtypes = [ctypes.c_void_p]
    return lib


@pytest.fixture
def up(lib):
    handle = lib.uploader_new()
    lib.set_registered(None, 0)
    lib.set_failures(0, 0)
    _counts(lib)
    yield handle
    lib.uploader_release(handle)
    lib.uploader_delete(handle)


def _counts(lib):
    c = (ctypes.c_longlong * 4)()
    lib.counts(c)
    return list(c)


def _copy(lib, up, n, seed=0):
    src = np.random.default_rng(seed).integers(0, 256, n, dtype=np.uint8)
    dst = np.zeros(n, np.uint8)
    status = lib.uploader_copy(up, dst.ctypes.data, src.ctypes.data, n)
    return status, np.array_equal(src, dst)


def test_a_network_used_once_makes_no_buffers(lib, up):
    """One prediction of 20,000 rows, or a few training sets: plain copies, nothing pinned."""
    for n in (20000 * 645 * 4, 8192 * 645 * 4, 8192 * 645 * 4, 100):
        assert _copy(lib, up, n) == (0, True)
    assert _counts(lib) == [0, 0, 4, 0]


def test_buffers_are_made_when_256_mb_have_come_and_given_back(lib, up):
    for k in range(3):
        assert _copy(lib, up, 64 * MB, k) == (0, True)
    for _ in range(100):
        assert _copy(lib, up, MB) == (0, True)          # small copies do not count
    assert _counts(lib) == [0, 0, 103, 0]
    assert _copy(lib, up, 64 * MB, 4) == (0, True)
    assert _counts(lib) == [1, 0, 0, 128]
    for n in (4 * MB, 4 * MB + 1, 5 * MB - 3, 21 * MB + 777):
        assert _copy(lib, up, n, n) == (0, True)
    assert _copy(lib, up, 4 * MB - 1) == (0, True)      # below the line: as it is
    made, freed, plain, staged = _counts(lib)
    assert (made, freed, plain) == (0, 0, 1) and staged == 8 + 9 + 10 + 43
    lib.uploader_release(up)
    assert _counts(lib) == [0, 1, 0, 0]
    assert _copy(lib, up, 64 * MB) == (0, True)
    assert _counts(lib) == [0, 0, 1, 0]


def test_one_large_copy_is_staged_at_once(lib, up):
    assert _copy(lib, up, 256 * MB + 5) == (0, True)
    assert _counts(lib) == [1, 0, 0, 513]


def test_pinned_sources_go_as_they_are(lib, up):
    n = 300 * MB
    src, dst = np.ones(n, np.uint8), np.zeros(n, np.uint8)
    lib.set_registered(src.ctypes.data, n)
    assert lib.uploader_copy(up, dst.ctypes.data, src.ctypes.data, n) == 0 and dst.all()
    assert _counts(lib) == [0, 0, 1, 0]


def test_without_buffers_copies_go_as_they_are_and_errors_are_returned(lib, up):
    lib.set_failures(1, 0)
    assert _copy(lib, up, 260 * MB) == (0, True)
    assert _counts(lib) == [0, 0, 1, 0]
    lib.set_failures(0, 1)
    assert _copy(lib, up, 8 * MB) == (0, True)          # not asked for again at once
    assert _copy(lib, up, 260 * MB)[0] != 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1626, 1627, 20011])
def test_staged_predictions_equal_plain_ones(rows):
    """A network that has taken more than 256 MB stages its inputs: the bits of small calls of
    another network, which never does."""
    from mind_b200 import surrogate

    rng = np.random.default_rng(rows)
    net, small = surrogate.Mlp(seed=9), surrogate.Mlp(seed=9)
    warm = np.zeros((20000, surrogate.N_FEATURES), np.float32)
    for _ in range(6):
        net.predict(warm)
    flat = rng.normal(0.0, 1.0, rows * surrogate.N_FEATURES + 1).astype(np.float32)
    for x in (flat[1:].reshape(rows, -1), flat[:-1].reshape(rows, -1)):
        parts = np.concatenate([small.predict(x[k:k + 128]) for k in range(0, rows, 128)])
        for _ in range(3):
            assert np.array_equal(net.predict(x), parts)
    small.close()
    net.close()
