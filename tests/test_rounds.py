"""The bound of a step's round loop (``abd_warp_b200/csrc/abd_rounds.cuh``): no step that can occur
meets it, and a step whose rounds make no progress ends.  CPU only."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rounds") / "librounds.so")
    src = os.path.join(HERE, "native", "rounds_host.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", out, src], check=True)
    lib = ctypes.CDLL(out)
    lib.rounds_host.argtypes = [ctypes.c_int, ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("max_iter", [0, 1, 2, 10, 60])
def test_bound(L, max_iter):
    n = max(1, max_iter)
    rng = np.random.default_rng(max_iter)
    for trial in range(50):
        leave = (rng.random(n) < trial / 49).astype(np.int32)
        assert L.rounds_host(max_iter, leave.ctypes.data) == 1 + leave.sum()
    for stuck in range(n):
        leave = np.zeros(n, dtype=np.int32)
        leave[stuck] = 10**6
        assert L.rounds_host(max_iter, leave.ctypes.data) == -(n + 1)
