"""An upload leaves the last run's result alone, for every app: read back after the
upload it is the old graph's, and the next run gives the new one's.  BFS in its three
forms (one CTA, worklist, from both sides)."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs

pytestmark = pytest.mark.gpu

SMALL, LARGE = (9, 8), (17, 16)
CASES = {"bfs_cta": ("lonestar_bfs", None), "bfs_list": ("lonestar_bfs", SMALL),
         "bfs_both": ("lonestar_bfs", LARGE), "sssp": ("lonestar_sssp", SMALL),
         "psssp": ("sssp", SMALL), "color": ("color", (11, 10)), "mis": ("mis", SMALL),
         "pagerank": ("pagerank", SMALL), "pagerank_large": ("pagerank", LARGE),
         "bc": ("bc", SMALL)}


def _two_graphs(size):
    """A graph and the same one with its vertices renumbered: equal counts."""
    g = graphs.rmat(*size, seed=5) if size else graphs.grid(40, 25)
    if g.weights is None:
        g.weights = graphs.uniform_weights(g, 5)
    n = g.num_nodes
    p = np.random.default_rng(3).permutation(n)
    s = p[np.repeat(np.arange(n), g.degrees())]
    d = p[g.col]
    o = np.lexsort((d, s))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(s, minlength=n))
    return g, graphs.Graph(rp, d[o].astype(np.int32), g.weights[o]), p


@pytest.mark.parametrize("case", list(CASES))
def test_upload_keeps_the_last_result(case):
    app, size = CASES[case]
    g, h, p = _two_graphs(size)
    src = graphs.max_degree_vertex(g)
    with Runtime() as r, PersistentApp(r, app, g) as a:
        if app in ("color", "mis"):
            nv = graphs.seeded_node_values(g.num_nodes, 2)
            a.set_node_values(nv)
        elif app != "bc" and app != "pagerank":
            a.set_source(src)
        a.launch()
        a.upload(h)  # on the runtime's stream, after the run
        old = a.result()
        with PersistentApp(r, app, g) as b:
            if app in ("color", "mis"):
                b.set_node_values(nv)
            elif app != "bc" and app != "pagerank":
                b.set_source(src)
            b.run()
            ref = b.result()
        if ref.dtype == np.float32:
            assert np.allclose(old, ref, rtol=2e-6, atol=0)
        else:
            assert np.array_equal(old, ref)
        if app in ("lonestar_bfs", "lonestar_sssp", "sssp"):
            a.set_source(int(p[src]))
            a.run()
            assert np.array_equal(a.result()[p], ref)
        elif app in ("pagerank", "bc"):
            a.run()
            assert np.allclose(a.result()[p], ref, rtol=1e-4, atol=1e-9)
