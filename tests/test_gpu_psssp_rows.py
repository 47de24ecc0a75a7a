"""Pannotia SSSP over rows by degree: degrees around the borders of the bins and of
the parts of wide rows, vertices without edges, unreachable ones, zero and large
weights, negative weights (no cycle), sources at both ends of the degree order; on
the default groups, one and five, with the same app re-run for another source; costs
against the oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu

EDGE = [0, 1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 255, 256, 257, 513, 2048, 2049, 5000]


def _graph(d, seed, wlo, whi, dag=False):
    rng = np.random.default_rng(seed)
    d = np.asarray(d).copy()
    if dag:
        d[0] = 0
    rp = np.zeros(len(d) + 1, np.int32)
    rp[1:] = np.cumsum(d)
    row = np.repeat(np.arange(len(d)), d)
    hi = row if dag else np.full(len(row), len(d))  # a DAG's edges go to smaller vertices
    col = (rng.random(len(row)) * hi).astype(np.int32)
    w = rng.integers(wlo, whi + 1, len(row)).astype(np.int32).view(np.uint32)
    return graphs.Graph(rp, col, w)


GRAPHS = {
    "borders": lambda: _graph(EDGE * 3, 1, 1, 1000),
    "zero": lambda: _graph(np.random.default_rng(3).permutation(EDGE * 10), 2, 0, 3),
    "large": lambda: _graph(EDGE * 5, 3, 20_000_000, 60_000_000),
    "negative": lambda: _graph(np.random.default_rng(4).permutation(EDGE * 10), 4, -50, 100, True),
    "wide": lambda: _graph([70000, 30000, 1, 0, 0, 3], 5, 1, 9),
    "none": lambda: _graph([0] * 9, 6, 1, 1),
    "sparse": lambda: _graph(np.random.default_rng(5).integers(0, 3, 3001), 7, 1, 1000),
}


@pytest.mark.parametrize("which", list(GRAPHS))
def test_psssp_rows(which):
    g = GRAPHS[which]()
    deg = np.diff(g.row_ptr)
    with Runtime() as r, PersistentApp(r, "sssp", g) as a:
        for src in (0, int(np.argmax(deg)), int(np.argmin(deg)), g.num_nodes - 1):
            a.set_source(src)
            want = oracle.pannotia_sssp(g, src)
            for groups in (0, 1, 5):
                a.run(groups)
                assert np.array_equal(a.result(), want), (which, src, groups)
