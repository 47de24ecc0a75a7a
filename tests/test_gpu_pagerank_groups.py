"""PageRank on its default groups: 1024 threads per SM in groups of the size that the
runtime was given, one group of 1024 where it was left at 256, fewer for small
graphs; against the oracle."""
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
        assert groups == max(1, min(r.sm_count() * per_sm, g.num_edges // (4 * size)))
        want = oracle.pagerank_f64(g)
        # the bound of the row tests: 20 iterations of a few float roundings each
        assert np.max(np.abs(a.result().astype(np.float64) - want)) <= 1e-5 * np.max(want)
