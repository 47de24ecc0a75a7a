"""SSSP on sparse graphs with hubs, around the degree from which their narrow levels
go another way (128 edges): stars, hubs joined in a chain, leaves between several
hubs, several edges between a hub and a leaf, weights of zero, from a hub and from a
leaf; on one group, three and the default; distances against the oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _graph(n, u, v, seed, wlo=1, whi=1000):
    """Both directions of every pair, each with a weight of its own."""
    s, d = np.concatenate([u, v]), np.concatenate([v, u])
    o = np.lexsort((d, s))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(s, minlength=n))
    w = np.random.default_rng(seed).integers(wlo, whi + 1, len(s)).astype(np.uint32)
    return graphs.Graph(rp, d[o].astype(np.int32), w)


def _stars(hubs, leaves, **kw):
    n = hubs * (leaves + 1)
    h = np.arange(hubs) * (leaves + 1)
    u = np.concatenate([np.repeat(h, leaves), h[:-1]])
    v = np.concatenate([np.setdiff1d(np.arange(n), h), h[1:]])
    return _graph(n, u, v, hubs, **kw)


def _between(hubs, leaves, times=1):
    u = np.tile(np.repeat(np.arange(hubs), leaves), times)
    v = np.tile(np.tile(np.arange(hubs, hubs + leaves), hubs), times)
    return _graph(hubs + leaves, u, v, leaves)


GRAPHS = {
    "star": lambda: _stars(1, 30000), "star33": lambda: _stars(1, 33),
    "128": lambda: _stars(1, 128), "129": lambda: _stars(1, 129),
    "126 joined": lambda: _stars(50, 126), "127 joined": lambda: _stars(50, 127),
    "chain": lambda: _stars(40, 700), "zero": lambda: _stars(12, 300, wlo=0, whi=1),
    "two hubs": lambda: _between(2, 9000), "three": lambda: _between(3, 500),
    "twice": lambda: _between(1, 2500, 3), "late hub": lambda: _graph(
        20101, np.concatenate([np.arange(100), np.full(20000, 100)]),
        np.concatenate([np.arange(1, 101), np.arange(101, 20101)]), 3),
}


@pytest.mark.parametrize("which", list(GRAPHS))
def test_sssp_hubs(which):
    g = GRAPHS[which]()
    assert g.num_edges <= 8 * g.num_nodes
    with Runtime() as r, PersistentApp(r, "lonestar_sssp", g) as a:
        for src in (0, g.num_nodes - 1, graphs.max_degree_vertex(g)):
            a.set_source(src)
            want = oracle.lonestar_sssp(g, src)
            for groups in (0, 1, 3, 0):
                a.run(groups)
                assert np.array_equal(a.result(), want), (which, src, groups)
