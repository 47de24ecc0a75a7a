"""BFS and SSSP on small dense graphs, whose list pieces are as long as the average
row, around the lengths where a short level changes its walker (64 edges): on one
group, three and the default; bit exact against the oracle."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree", [(700, 33), (700, 63), (700, 64), (700, 65), (300, 129),
                                      (1000, 999), (40, 2500)])
def test_dense_rows(n, degree):
    rng = np.random.default_rng(degree)
    d = rng.multinomial(n * degree, rng.dirichlet(np.full(n, 5.0)))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(d)
    g = graphs.Graph(rp, rng.integers(0, n, n * degree).astype(np.int32),
                     rng.integers(0, 500, n * degree).astype(np.uint32))
    with Runtime() as r:
        for app, ref in (("lonestar_bfs", oracle.lonestar_bfs),
                         ("lonestar_sssp", oracle.lonestar_sssp)):
            with PersistentApp(r, app, g) as a:
                for src in (0, graphs.max_degree_vertex(g)):
                    a.set_source(src)
                    want = ref(g, src)
                    for groups in (0, 1, 3):
                        a.run(groups)
                        assert np.array_equal(a.result(), want), (app, src, groups)
