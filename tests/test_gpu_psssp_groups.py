"""Pannotia SSSP on its default groups - 256, 512 or 1024 threads per SM by the work of
a pass - at the sizes where the rule steps, with a row more and a row less; costs
against the oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [64, 256, 512, 1024])
@pytest.mark.parametrize("units_per_sm,degree,per_sm", [
    (2, 3, (256, 256, 256)), (8, 3, (256, 256, 512)), (13, 5, (512, 512, 1024)),
    (32, 8, (1024, 1024, 1024)), (32, 40, (512, 512, 1024))])
def test_default_groups(threads, units_per_sm, degree, per_sm):
    with Runtime(threads_per_wg=threads) as r:
        sms = r.sm_count()
        rows = 32 if degree <= 8 else 4  # of a unit
        for more, want_threads in zip((-1, 0, 1), per_sm):
            n = units_per_sm * sms * rows + more
            rng = np.random.default_rng(n)
            g = graphs.Graph(np.arange(0, degree * n + 1, degree, dtype=np.int32),
                             rng.integers(0, n, degree * n).astype(np.int32),
                             rng.integers(1, 100, degree * n).astype(np.uint32))
            with PersistentApp(r, "sssp", g, source=5) as a:
                st = a.run()
                assert st.groups == sms * max(1, want_threads // threads), (more, n)
                assert np.array_equal(a.result(), oracle.pannotia_sssp(g, 5))
