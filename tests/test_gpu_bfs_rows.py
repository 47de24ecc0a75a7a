"""One-CTA BFS with its columns kept as 4 or 8 per vertex: largest degrees around
4 and 8 (9 walks the CSR), the loader's last-edge quirk, out-of-range columns and
frontiers past the shared buffers; levels against the oracle and the grid form, level
count included."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _regular(n, deg, seed):
    """Every vertex has out-degree deg or less, at random; some have none."""
    rng = np.random.default_rng(seed)
    d = rng.integers(0, deg + 1, n)
    d[rng.integers(0, n)] = deg
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(d)
    return graphs.Graph(rp, rng.integers(0, n, int(rp[-1])).astype(np.int32))


@pytest.mark.parametrize("deg", [1, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("n", [33, 5000, 60001])
def test_bfs_rows(deg, n):
    g = _regular(n, deg, 7 * deg + n)
    bad = graphs.Graph(g.row_ptr, g.col.copy())
    bad.col[::5] = np.array([n, -1, np.iinfo(np.int32).min, 2**31 - 1], np.int64)[
        np.arange(len(bad.col[::5])) % 4].astype(np.int32)
    with Runtime() as r:
        for x in (g, graphs.lonestar_view(g), bad):
            src = int(np.argmax(np.diff(x.row_ptr)))
            out = {}
            for mode in (0, 1):
                with PersistentApp(r, "lonestar_bfs", x, source=src, bfs_mode=mode) as a:
                    st = a.run()
                    out[mode] = (a.result(), st.rounds)
            assert np.array_equal(out[1][0], out[0][0])
            assert out[1][1] == out[0][1]
            if x is not bad:
                assert np.array_equal(out[1][0], oracle.lonestar_bfs(x, src))


def test_bfs_wide_frontier(rt):
    """A tree of eight children a vertex: its last level has more vertices than
    both shared frontier buffers."""
    n = 65536
    kids = [np.arange(8 * v + 1, min(8 * v + 9, n), dtype=np.int32) for v in range(n)]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum([len(k) for k in kids])
    g = graphs.Graph(rp, np.concatenate(kids).astype(np.int32))
    with PersistentApp(rt, "lonestar_bfs", g) as a:
        st = a.run()
        assert st.groups == 1
        assert np.array_equal(a.result(), oracle.lonestar_bfs(g, 0))
