"""Betweenness centrality with the sources spread over CTAs: the rows in turn
(average degree up to 4) and the rows handed out, levels of one to thousands
of vertices, each number of threads a source takes, graphs smaller than a
warp, one source and more sources than CTAs, against the float64 oracle."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-4


@pytest.mark.parametrize("name,sources", [
    ("grid1x2", None), ("grid15x8", None), ("grid24x24", None), ("grid3x400", 64),
    ("rmat1024", None), ("rmat1025", 200), ("rmat3584", 40), ("rmat3585", 40), ("rmat3585", 1)])
def test_bc_levels_and_threads(name, sources):
    if name.startswith("grid"):
        g = graphs.grid(*map(int, name[4:].split("x")))
    else:
        full, n = graphs.rmat(12, 8, seed=5), int(name[4:])
        src = np.repeat(np.arange(full.num_nodes), np.diff(full.row_ptr))
        keep = (src < n) & (full.col < n)
        rp = np.zeros(n + 1, np.int32)
        rp[1:] = np.cumsum(np.bincount(src[keep], minlength=n))
        g = graphs.Graph(rp, full.col[keep].astype(np.int32))
    with Runtime(run_timeout_ns=20_000_000_000) as rt, \
            PersistentApp(rt, "bc", g, bc_sources=sources, bc_mode=1) as a:
        want = oracle.pannotia_bc_f64(g, sources)
        for _ in range(2):
            assert a.run().rounds == (sources or g.num_nodes)
            err = np.abs(a.result().astype(np.float64) - want).max() / max(np.abs(want).max(), 1e-30)
            assert err <= TOL, err
