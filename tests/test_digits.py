"""The digit counters of the exact sums (``abd_warp_b200/csrc/abd_digits.cuh``) on the host: folding any
number of times keeps the sum, of either sign and up to the largest that can occur, and its limbs
hold it.  CPU only."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
DW, SLOTS = 14, 32


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("digits") / "libdigits.so")
    src = os.path.join(HERE, "native", "digits_host.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", out, src], check=True)
    lib = ctypes.CDLL(out)
    lib.digits_fold.argtypes = [ctypes.c_void_p]
    lib.digits_limbs.argtypes = [ctypes.c_void_p, ctypes.c_void_p]
    return lib


def _digits(m):
    """The signed 14-bit digits of an integer, its sign on each."""
    s, m = (-1, -m) if m < 0 else (1, m)
    out = np.zeros(SLOTS, dtype=np.int64)
    k = 0
    while m:
        out[k], m, k = s * (m & ((1 << DW) - 1)), m >> DW, k + 1
    return out


def _check(L, s, total):
    assert s.min() > -2**31 and s.max() < 2**31
    c = s.astype(np.int32)
    d = np.zeros(10, dtype=np.int64)
    assert L.digits_limbs(c.ctypes.data, d.ctypes.data) == 0
    assert sum(int(d[j]) << (32 * j) for j in range(10)) == total


# a value's exponent over the sum's grid 2^-192: 1e-4, 1, 1e4, 1e8, 2^127
@pytest.mark.parametrize("power", [-14, 0, 13, 26, 127])
@pytest.mark.parametrize("signs", [(-1,), (1,), (-1, 1, -1)])
@pytest.mark.parametrize("folds", [0, 1, 9, 17, 40, 200])
def test_folds_keep_the_sum(L, power, signs, folds):
    rng = np.random.default_rng(1000 * (power + 20) + folds)
    s, total = np.zeros(SLOTS, dtype=np.int64), 0
    for r in range(folds + 1):
        block = 0
        for k in range(8):
            m = int(rng.integers(1 << 52, 1 << 53)) << (power - 52 + 192)
            m *= signs[(r + k) % len(signs)]
            s += 4096 * _digits(m)  # (that many terms)
            block += 4096 * m
        total += block
        if r < folds:
            assert np.abs(s).max() < 2**31
            c = s.astype(np.int32)
            L.digits_fold(c.ctypes.data)
            assert np.abs(c).max() <= 2**17 + 2**14
            s = c.astype(np.int64)
    _check(L, s, total)


def test_many_folds_of_a_small_negative_sum(L):
    s = _digits(-(10_000 << 192))
    for _ in range(64):
        c = s.astype(np.int32)
        L.digits_fold(c.ctypes.data)
        s = c.astype(np.int64)
    _check(L, s, -(10_000 << 192))
