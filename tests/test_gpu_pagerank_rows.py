"""PageRank's rows by degree: degrees around the borders of its bins (8, 16, ...,
128 edges for 1, 2, ..., 16 lanes) and of the parts of wide rows (256 edges, several
parts), vertices without edges, no edges at all, a directed graph, 0 and 1 iterations;
on the default groups, one group and an odd count of small ones; within 1e-5
relative L-inf of the FP64 oracle, and the same bits from run to run."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _degrees(d, seed):
    rng = np.random.default_rng(seed)
    d = np.asarray(d)
    rp = np.zeros(len(d) + 1, np.int32)
    rp[1:] = np.cumsum(d)
    return graphs.Graph(rp, rng.integers(0, len(d), int(rp[-1])).astype(np.int32))


EDGE = [0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512,
        513, 2047, 2048, 2049, 5000]
GRAPHS = {
    "borders": lambda: _degrees(EDGE * 3, 1), "shuffled": lambda: _degrees(
        np.random.default_rng(2).permutation(EDGE * 20), 2),
    "wide": lambda: _degrees([70000, 30000, 1, 0, 0, 3], 3), "none": lambda: _degrees([0] * 37, 4),
    "one_edge": lambda: _degrees([0, 1, 0], 5), "regular": lambda: _degrees([8] * 1000, 6),
    "rmat": lambda: graphs.rmat(13, 16, seed=7),
}


def _f64(g, iterations):
    deg = np.diff(g.row_ptr).astype(np.int64)
    row = np.repeat(np.arange(g.num_nodes), deg)
    pr = np.full(g.num_nodes, 1.0 / g.num_nodes)
    for _ in range(iterations):
        c = np.divide(pr, deg, out=np.zeros_like(pr), where=deg > 0)
        s = np.bincount(row, weights=c[g.col], minlength=g.num_nodes)
        pr = 0.15 / g.num_nodes + 0.85 * (s + pr[deg == 0].sum() / g.num_nodes)
    return pr


@pytest.mark.parametrize("threads", [64, 256])
@pytest.mark.parametrize("which", list(GRAPHS))
def test_pagerank_rows(which, threads):
    g = GRAPHS[which]()
    with Runtime(threads_per_wg=threads) as r:
        for it in (0, 1, 20):
            with PersistentApp(r, "pagerank", g, iterations=it) as a:
                want = oracle.pagerank_f64(g) if it == 20 else _f64(g, it)
                for groups in (0, 1, 5, 0):
                    a.run(groups)
                    got = a.result()
                    err = np.max(np.abs(got.astype(np.float64) - want)) / np.max(want)
                    assert err <= 1e-5, (which, it, groups, err)
                a.run()
                assert np.array_equal(a.result(), got)
