"""The clustering's merging rounds (``abd_warp_b200/csrc/abd_merge.cuh``) by host threads that reach each
step at different times: every thread takes the same number of rounds, and the clusters are those
of a sequential restatement.  CPU only."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("merge") / "libmerge.so")
    src = os.path.join(HERE, "native", "merge_host.cpp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-o", out, src], check=True)
    lib = ctypes.CDLL(out)
    lib.merge_host.argtypes = [ctypes.c_int, ctypes.c_uint] + [ctypes.c_int] * 3 + [ctypes.c_void_p, ctypes.c_int] + [ctypes.c_void_p] * 2
    lib.merge_host.restype = None
    return lib


def _sequential(n, cap, rounds, act):
    label, size = list(range(n)), [1] * n
    for _ in range(rounds if cap > 1 else 0):
        best = [None] * n
        for p, i, j, w in act:
            a, b = label[i], label[j]
            if a == b or size[a] + size[b] > cap:
                continue
            for c in (a, b):
                best[c] = max(best[c] or (w, -p, 0), (w, -p, 1))
        to, new, merged = list(range(n)), list(size), False
        for p, i, j, w in act:
            a, b = label[i], label[j]
            if a != b and best[a] == best[b] == (w, -p, 1):
                to[max(a, b)] = min(a, b)
                new[min(a, b)] += size[max(a, b)]
                merged = True
        if not merged:
            break
        label, size = [to[c] for c in label], new
    return label, size


@pytest.mark.parametrize("n,pairs,cap", [(1, 0, 12), (2, 1, 12), (5, 4, 1), (9, 20, 2), (33, 60, 12), (64, 200, 12)])
def test_late_threads(L, n, pairs, cap):
    for seed in range(6):
        rng = np.random.default_rng(100 * n + seed)
        ij = sorted({tuple(sorted(rng.choice(n, 2, replace=False))) for _ in range(pairs)}) if n > 1 else []
        act = np.array([[p, i, j, rng.integers(1, 8)] for p, (i, j) in enumerate(ij)], dtype=np.int32).reshape(-1, 4)
        label, size = np.arange(n, dtype=np.int32), np.ones(n, dtype=np.int32)
        shuffled = np.ascontiguousarray(act[rng.permutation(len(act))])
        L.merge_host(7, seed, n, cap, 48, shuffled.ctypes.data, len(act), label.ctypes.data, size.ctypes.data)
        want, sizes = _sequential(n, cap, 48, act.tolist())
        assert label.tolist() == want
        assert [size[c] for c in sorted(set(want))] == [sizes[c] for c in sorted(set(want))]
