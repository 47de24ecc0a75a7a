"""PageRank on its default groups: 1024 threads per SM in groups of the size that the
runtime was given, one group of 1024 where it was left at 256, fewer for small
graphs but a warp for every unit of work, with a unit more and a unit less; against
the oracle."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,size,per_sm", [(256, 1024, 1), (1024, 1024, 1), (512, 512, 2),
                                                 (128, 128, 8), (64, 64, 16)])
@pytest.mark.parametrize("scale", [7, 16])
def test_default_groups(threads, size, per_sm, scale):
    g = graphs.rmat(scale, 16, seed=2)
    with Runtime(threads_per_wg=threads) as r, PersistentApp(r, "pagerank", g) as a:
        groups = a.run().groups
        assert groups <= r.sm_count() * per_sm
        assert groups >= min(r.sm_count() * per_sm, max(1, g.num_edges // (4 * size)))
        want = oracle.pagerank_f64(g)
        # the bound of the row tests: 20 iterations of a few float roundings each
        assert np.max(np.abs(a.result().astype(np.float64) - want)) <= 1e-5 * np.max(want)


@pytest.mark.parametrize("threads,size", [(256, 1024), (64, 64)])
@pytest.mark.parametrize("groups", [1, 5, 40])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_a_warp_for_every_unit(threads, size, groups, more):
    n = groups * (size // 32) * 32 + more  # a unit holds 32 rows of 3 edges
    rng = np.random.default_rng(n)
    g = graphs.Graph(np.arange(0, 3 * n + 1, 3, dtype=np.int32),
                     rng.integers(0, n, 3 * n).astype(np.int32))
    with Runtime(threads_per_wg=threads) as r, PersistentApp(r, "pagerank", g) as a:
        assert a.run().groups == groups + (more > 0)
        want = oracle.pagerank_f64(g)
        assert np.max(np.abs(a.result().astype(np.float64) - want)) <= 1e-5 * np.max(want)
