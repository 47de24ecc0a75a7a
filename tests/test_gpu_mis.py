"""Independent set at the edges of its kernel: vertex counts around the 32
vertices of a mask word, rows around the four edges a lane looks at, the 128 of a
warp's step and the `scan` limit past which the whole grid takes over
(2 x hub_threshold), on one group and on many; s_array against the oracle (bit
exact) and a directed graph."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _csr(rows):
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return graphs.Graph(rp, np.array([c for r in rows for c in r], np.int32))


def _star(leaves):
    return _csr([list(range(1, leaves + 1))] + [[0]] * leaves)


def _clique(n):
    return _csr([[j for j in range(n) if j != i] for i in range(n)])


def _directed(seed):
    g = graphs.rmat(11, 12, seed=seed)
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(g.num_nodes), g.degrees())
    keep = rng.random(g.num_edges) < 0.5
    rp = np.zeros(g.num_nodes + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(src[keep], minlength=g.num_nodes))
    return graphs.Graph(rp, g.col[keep].astype(np.int32))


GRAPHS = {
    "one": lambda: _csr([[]]), "pair": lambda: _csr([[1], [0]]),
    "v31": lambda: graphs.grid(1, 31), "v32": lambda: graphs.grid(4, 8),
    "v33": lambda: graphs.grid(3, 11), "v1025": lambda: graphs.grid(25, 41),
    "clique5": lambda: _clique(5), "clique130": lambda: _clique(130),
    "star64": lambda: _star(64), "star65": lambda: _star(65), "star513": lambda: _star(513),
    "star20000": lambda: _star(20000), "rmat": lambda: graphs.rmat(13, 16, seed=5),
    "odd": lambda: graphs.rmat(9, 24, seed=6), "directed": lambda: _directed(3),
}


@pytest.mark.parametrize("hub_threshold", [32, 256])
@pytest.mark.parametrize("which", list(GRAPHS))
def test_mis_edges_of_the_kernel(which, hub_threshold):
    g = GRAPHS[which]()
    # three priority orders: random, the hub (vertex 0) first, the hub last
    orders = [graphs.seeded_node_values(g.num_nodes, 9), graphs.reference_node_values(g.num_nodes),
              graphs.reference_node_values(g.num_nodes)[::-1].copy()]
    with Runtime(hub_threshold=hub_threshold) as r:
        for nv in orders:
            want = oracle.mis(g, nv)
            with PersistentApp(r, "mis", g, node_values=nv) as a:
                rounds = set()
                for groups in (0, 1, 3):
                    st = a.run(groups)
                    rounds.add(st.rounds)
                    assert np.array_equal(a.result(), want), (which, groups)
                assert len(rounds) == 1
