"""Which form a colour run takes: blocks of priorities where they are independent of
the graph and its chains are long, rounds where the priorities follow the edges or a
dozen rounds do; each against the oracle, also when one app goes from one to the other."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _band(n, half):
    """Vertex i next to i - half .. i + half."""
    rows = [np.setdiff1d(np.arange(max(0, i - half), min(n, i + half + 1)), [i])
            for i in range(n)]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return graphs.Graph(rp, np.concatenate(rows).astype(np.int32))


GRAPHS = {"clique": lambda: _band(150, 150), "rmat10": lambda: graphs.rmat(10, 8, seed=2),
          "rmat15": lambda: graphs.rmat(15, 16, seed=4), "band": lambda: _band(16000, 16),
          "grid": lambda: graphs.grid(300, 300)}
# (seeded priorities, priorities by vertex number)
BLOCKS = {"clique": (True, True), "rmat10": (True, True), "rmat15": (True, True),
          "band": (True, False), "grid": (False, False)}


@pytest.mark.parametrize("which", list(GRAPHS))
def test_color_forms(which):
    g = GRAPHS[which]()
    seeded = graphs.seeded_node_values(g.num_nodes, 4)
    numbered = graphs.reference_node_values(g.num_nodes)
    with Runtime() as r, PersistentApp(r, "color", g) as a:
        for nv, blocks in zip((seeded, numbered, seeded), BLOCKS[which] + BLOCKS[which][:1]):
            a.set_node_values(nv)
            assert (a.color_blocks() > 0) == blocks
            want = oracle.color(g, nv)
            st = a.run()
            assert np.array_equal(a.result(), want) and st.rounds == want.max()


def test_forms_of_the_block_tests_graphs():
    """The graphs that the block tests mean for blocks take them at every block size."""
    from test_gpu_color_blocks import GRAPHS as block_graphs
    for cfg in (dict(), dict(hub_threshold=32), dict(threads_per_wg=64),
                dict(threads_per_wg=1024)):
        with Runtime(**cfg) as r:
            for which in ("three", "clique61", "clique150", "rmat10", "odd", "odd2", "directed"):
                g = block_graphs[which]()
                nv = graphs.seeded_node_values(g.num_nodes, 4)
                with PersistentApp(r, "color", g, node_values=nv) as a:
                    assert a.color_blocks() > 0, (cfg, which)
