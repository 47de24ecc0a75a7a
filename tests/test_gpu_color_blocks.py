"""Colour in priority blocks (the default of standalone runs where the layout picks
it): colours and round count against the oracle, bit exact, at the edges of its
blocks - one block and many, vertex counts that are no multiple of four, hubs
across block borders and a low hub threshold, directed graphs, degree-1 leaves - on
one group, three and the default; new priorities and a new graph on the same app;
and priorities that follow the edges, which stay with the rounds."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _csr(rows):
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return graphs.Graph(rp, np.array([c for r in rows for c in r], np.int32))


def _clique(n):
    return _csr([[j for j in range(n) if j != i] for i in range(n)])


def _cut(g, n):
    """The first n vertices of g."""
    src = np.repeat(np.arange(g.num_nodes), g.degrees())
    keep = (src < n) & (g.col < n)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(src[keep], minlength=n))
    return graphs.Graph(rp, g.col[keep].astype(np.int32))


def _directed(seed):
    g = graphs.rmat(12, 12, seed=seed)
    keep = np.random.default_rng(seed).random(g.num_edges) < 0.6
    src = np.repeat(np.arange(g.num_nodes), g.degrees())
    rp = np.zeros(g.num_nodes + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(src[keep], minlength=g.num_nodes))
    return graphs.Graph(rp, g.col[keep].astype(np.int32))


GRAPHS = {
    "three": lambda: _clique(3), "clique61": lambda: _clique(61),
    "clique150": lambda: _clique(150), "path": lambda: graphs.grid(1, 999),
    "grid": lambda: graphs.grid(65, 63), "rmat10": lambda: graphs.rmat(10, 8, seed=2),
    "odd": lambda: _cut(graphs.rmat(12, 16, seed=3), 2999),
    "odd2": lambda: _cut(graphs.rmat(15, 16, seed=4), 30001),
    "directed": lambda: _directed(5),
    "leaves": lambda: _csr([list(range(1, 700))] + [[0]] * 699),
}


@pytest.mark.parametrize("cfg", [dict(), dict(hub_threshold=32), dict(threads_per_wg=64),
                                 dict(threads_per_wg=1024)])
@pytest.mark.parametrize("which", list(GRAPHS))
def test_color_blocks(which, cfg):
    g = GRAPHS[which]()
    with Runtime(**cfg) as r, PersistentApp(r, "color", g) as a:
        for nv in (graphs.seeded_node_values(g.num_nodes, 4),
                   graphs.reference_node_values(g.num_nodes),
                   graphs.seeded_node_values(g.num_nodes, 5)):
            a.set_node_values(nv)
            want = oracle.color(g, nv)
            for groups in (0, 1, 3):
                st = a.run(groups)
                assert np.array_equal(a.result(), want), (which, cfg, groups)
                assert st.rounds == want.max()


def test_color_blocks_reupload(rt):
    """A new graph of the same size keeps the priorities and gets their blocks."""
    g = graphs.rmat(11, 10, seed=1)
    perm = np.random.default_rng(2).permutation(g.num_nodes)
    inv = np.argsort(perm)
    rows = [np.sort(inv[g.col[g.row_ptr[v]:g.row_ptr[v + 1]]]) for v in perm]
    h = _csr([r.tolist() for r in rows])
    nv = graphs.seeded_node_values(g.num_nodes, 8)
    with PersistentApp(rt, "color", g, node_values=nv) as a:
        for x in (g, h, g):
            a.upload(x)
            a.run()
            assert np.array_equal(a.result(), oracle.color(x, nv))
