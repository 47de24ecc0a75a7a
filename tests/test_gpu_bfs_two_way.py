"""BFS that turns to the unreached side on wide levels (graphs of two million edges
or more), bit exact against the oracle, level count included: directed graphs, the
loader's last-edge quirk, out-of-range columns, vertices of more in-edges than one
warp looks at, and two dense parts joined by a path (from the worklist to the other
side, back, and there again)."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _from_pairs(n, s, d):
    o = np.lexsort((d, s))
    s, d = s[o], d[o]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(s, minlength=n))
    return graphs.Graph(rp, d.astype(np.int32))


def _pairs(g):
    return np.repeat(np.arange(g.num_nodes), g.degrees()), g.col.astype(np.int64)


def _dumbbell(path):
    a, b = graphs.rmat(15, 48, seed=3), graphs.rmat(15, 48, seed=4)
    (sa, da), (sb, db) = _pairs(a), _pairs(b)
    na = a.num_nodes
    p0 = 2 * na
    chain = np.concatenate([[int(da[0])], np.arange(p0, p0 + path), [na + int(db[0])]])
    s = np.concatenate([sa, sb + na, chain[:-1], chain[1:]])
    d = np.concatenate([da, db + na, chain[1:], chain[:-1]])
    return _from_pairs(p0 + path, s, d)


def _funnel():
    """Every vertex points at two sinks (more in-edges than a warp looks at);
    one sink's only reached in-neighbour comes last in its row."""
    g = graphs.rmat(16, 24, seed=6)
    s, d = _pairs(g)
    n = g.num_nodes
    lone = np.flatnonzero(g.degrees() == 0)
    s = np.concatenate([s, np.arange(n), lone, [int(s[0])]])
    d = np.concatenate([d, np.full(n, n), np.full(len(lone), n + 1), [n + 1]])
    return _from_pairs(n + 2, s, d)


def _directed():
    s, d = _pairs(graphs.rmat(17, 24, seed=7))
    keep = np.random.default_rng(1).random(len(s)) < 0.6
    return _from_pairs(1 << 17, s[keep], d[keep])


GRAPHS = {"rmat": lambda: graphs.rmat(17, 16, seed=2), "directed": _directed,
          "dumbbell": lambda: _dumbbell(300), "dumbbell0": lambda: _dumbbell(1),
          "funnel": _funnel}


@pytest.mark.parametrize("which", list(GRAPHS))
def test_bfs_two_way(which):
    g = GRAPHS[which]()
    assert g.num_edges >= 2 << 20
    with Runtime() as r:
        for x in (g, graphs.lonestar_view(g)):
            for src in (graphs.max_degree_vertex(g), int(g.col[12345])):
                want = oracle.lonestar_bfs(x, src)
                # the count is the first level L that nothing with out-edges at L - 1 feeds
                levels = int(want[(want < 1000000000) & (x.degrees() > 0)].max()) + 2
                with PersistentApp(r, "lonestar_bfs", x, source=src) as a:
                    for groups in (0, 3):
                        st = a.run(groups)
                        assert np.array_equal(a.result(), want), (which, src, groups)
                        assert st.rounds == levels


def test_bfs_two_way_out_of_range_columns(rt):
    g = graphs.rmat(17, 16, seed=9)
    bad = graphs.Graph(g.row_ptr, g.col.copy())
    bad.col[::7] = np.where(np.arange(len(bad.col[::7])) % 2, -1, g.num_nodes).astype(np.int32)
    s, d = _pairs(bad)
    keep = (d >= 0) & (d < g.num_nodes)
    clean = _from_pairs(g.num_nodes, s[keep], d[keep])
    src = graphs.max_degree_vertex(clean)
    with PersistentApp(rt, "lonestar_bfs", bad, source=src) as a:
        a.run()
        assert np.array_equal(a.result(), oracle.lonestar_bfs(clean, src))
