"""Pannotia SSSP on its default groups - a warp for every unit of a pass, whole groups
per SM - at the sizes where the rule steps, with a unit more and a unit less; costs
against the oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 256, 1024])
@pytest.mark.parametrize("turns", [1, 2])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_default_groups(threads, turns, more):
    with Runtime(threads_per_wg=threads) as r:
        sms, per_sm = r.sm_count(), 1024 // threads
        n = turns * sms * (threads // 32) * 32 + more  # a unit holds 32 rows of 3 edges
        rng = np.random.default_rng(n)
        g = graphs.Graph(np.arange(0, 3 * n + 1, 3, dtype=np.int32),
                         rng.integers(0, n, 3 * n).astype(np.int32),
                         rng.integers(1, 100, 3 * n).astype(np.uint32))
        with PersistentApp(r, "sssp", g, source=5) as a:
            st = a.run()
            assert st.groups == sms * min(per_sm, turns + (more > 0))
            assert np.array_equal(a.result(), oracle.pannotia_sssp(g, 5))
