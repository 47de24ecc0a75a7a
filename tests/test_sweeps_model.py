"""The bound on a colour block's sweeps, in a CPU model of its racing stores: random
and stalled interleavings over cliques, chains and random acyclic lists, with colours
so far of any size, always settle within it at the right colours."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("model") / "libsweeps_model.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-o", out,
                    os.path.join(HERE, "model", "sweeps_model.cpp")], check=True)
    lib = C.CDLL(out)
    lib.model_sweeps.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_uint64]
    return lib


def _edges(kind, n, rng):
    pairs = [(i, j) for j in range(n) for i in range(j)]
    if kind == "chain":
        pairs = [(i, i + 1) for i in range(n - 1)]
    elif kind == "random":
        pairs = [p for p in pairs if rng.random() < 0.4]
    elif kind == "none":
        pairs = []
    return np.array(pairs, np.int32).reshape(-1, 2)


@pytest.mark.parametrize("stall", [0, 1])
@pytest.mark.parametrize("kind", ["clique", "chain", "random", "none"])
def test_sweeps_settle_within_the_bound(model, kind, stall):
    for seed in range(40):
        rng = np.random.default_rng(seed)
        n = int(rng.integers(2, 14))
        e = _edges(kind, n, rng)
        src, dst = e[:, 0].copy(), e[:, 1].copy()
        col = rng.integers(1, [2, 8, 100][seed % 3], n).astype(np.int32)
        want = col.copy()
        for v in range(n):  # sources come before their targets
            for u in src[dst == v]:
                want[v] = max(want[v], want[u] + 1)
        got = model.model_sweeps(len(src), src.ctypes.data, dst.ctypes.data, col.ctypes.data,
                                 stall, seed)
        assert got > 0 and np.array_equal(col, want), (kind, seed, got)
