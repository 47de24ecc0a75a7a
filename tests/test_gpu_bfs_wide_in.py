"""BFS from the unreached side with many vertices of far more in-edges than one warp
looks at, found by several warps at once: sinks whose reached in-neighbours lie
anywhere in their rows, and sinks without any, bit exact against the oracle."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sinks", [1, 40])
def test_sinks_of_very_many_in_edges(sinks):
    g = graphs.rmat(16, 24, seed=11)
    rng = np.random.default_rng(sinks)
    n = g.num_nodes
    s0 = np.repeat(np.arange(n), g.degrees())
    lone = np.flatnonzero(g.degrees() == 0)
    src = [s0]
    dst = [g.col.astype(np.int64)]
    for k in range(sinks):
        # every unreachable vertex of the graph names the sink, and a few others do
        few = rng.choice(s0, [0, 1, 3, 300][k % 4])
        src += [lone, few]
        dst += [np.full(len(lone), n + k), np.full(len(few), n + k)]
    s, d = np.concatenate(src), np.concatenate(dst)
    o = np.lexsort((d, s))
    rp = np.zeros(n + sinks + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(s, minlength=n + sinks))
    x = graphs.Graph(rp, d[o].astype(np.int32))
    assert x.num_edges >= 2 << 20 and len(lone) > 4096
    with Runtime() as r, PersistentApp(r, "lonestar_bfs", x) as a:
        for start in (graphs.max_degree_vertex(g), int(g.col[999])):
            a.set_source(start)
            want = oracle.lonestar_bfs(x, start)
            for groups in (0, 0, 5):
                a.run(groups)
                assert np.array_equal(a.result(), want), (start, groups)
