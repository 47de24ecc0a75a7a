"""The Lonestar loader's quirk on a graph whose last vertices have no edges, with as
many columns as the last row pointer says: the row before them ends one past the
columns.  BFS (one CTA, worklist, from both sides) and SSSP walk the columns that
there are."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _quirk(g, lonely):
    """(g without its last edge and with `lonely` vertices after it, the same as the
    loader leaves it)"""
    rp = np.concatenate([g.row_ptr, np.full(lonely, g.num_edges, np.int32)])
    col, wt = g.col[:-1].copy(), g.weights[:-1].copy()
    clean = np.minimum(rp, len(col)).astype(np.int32)
    quirk = rp.copy()
    quirk[-1] = len(col)
    return graphs.Graph(clean, col, wt), graphs.Graph(quirk, col, wt)


GRAPHS = {"grid": lambda: graphs.grid(37, 41), "rmat": lambda: graphs.rmat(10, 8, seed=3),
          "large": lambda: graphs.rmat(17, 16, seed=4)}


@pytest.mark.parametrize("lonely", [1, 3])
@pytest.mark.parametrize("which", list(GRAPHS))
def test_row_past_columns(which, lonely):
    g = GRAPHS[which]()
    if g.weights is None:
        g.weights = graphs.uniform_weights(g, 1)
    # the row that ends past the columns is the last one with edges
    last = int(np.flatnonzero(g.degrees())[-1])
    g = graphs.Graph(g.row_ptr[:last + 2], np.minimum(g.col, last).astype(np.int32), g.weights)
    clean, quirk = _quirk(g, lonely)
    assert quirk.row_ptr[-2] == quirk.num_edges + 1 and quirk.row_ptr[-1] == quirk.num_edges
    with Runtime() as r:
        for app, ref in (("lonestar_bfs", oracle.lonestar_bfs),
                         ("lonestar_sssp", oracle.lonestar_sssp)):
            for src in (0, last, graphs.max_degree_vertex(clean)):
                with PersistentApp(r, app, quirk, source=src) as a:
                    want = ref(clean, src)
                    for _ in range(2):
                        a.run()
                        assert np.array_equal(a.result(), want), (app, src)
                        a.upload(quirk)
