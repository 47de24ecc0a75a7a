"""Pannotia SSSP where the parts of very long rows lower their row's cost in every
pass while other warps decide whether to leave that row out; costs against the
oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hubs,edges,path", [(1, 70000, 40), (24, 60000, 64), (3, 2049, 9)])
def test_wide_rows_lowered_in_every_pass(hubs, edges, path):
    """Vertex i of a path costs i; a hub's edge to it costs less by 3 than the one
    before, so every pass that reaches a vertex lowers every hub again."""
    rng = np.random.default_rng(hubs)
    rows = [np.array([], np.int64)] + [np.array([i - 1]) for i in range(1, path)]
    wts = [np.array([], np.int64)] + [np.array([1])] * (path - 1)
    for _ in range(hubs):
        c = rng.integers(0, path, edges)
        rows.append(c)
        wts.append(3 * path - 3 * c)
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    g = graphs.Graph(rp, np.concatenate(rows).astype(np.int32),
                     np.concatenate(wts).astype(np.uint32))
    want = oracle.pannotia_sssp(g, 0)
    with Runtime() as r, PersistentApp(r, "sssp", g) as a:
        for groups in (0, 1, 7, 0, 0):
            a.run(groups)
            assert np.array_equal(a.result(), want)
