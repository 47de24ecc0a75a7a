"""SSSP on graphs of average degree 8 or less, whose narrow levels relax what they
improve at once: a long path, grids with the loader's last-edge quirk, rows of up to
40 edges among short ones (more than a warp's 32), zero weights and weights at the
skip limit, several edges between two vertices, average degrees on both sides of 8; on
one group, three and the default; distances against the oracle, bit exact."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _random(n, degrees, seed, wlo=1, whi=1000):
    rng = np.random.default_rng(seed)
    d = rng.choice(degrees, n)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(d)
    e = int(rp[-1])
    return graphs.Graph(rp, rng.integers(0, n, e).astype(np.int32),
                        rng.integers(wlo, whi + 1, e).astype(np.uint32))


def _weighted(g, seed, **kw):
    g.weights = graphs.uniform_weights(g, seed, **kw)
    return g


GRAPHS = {
    "path": lambda: _weighted(graphs.grid(1, 3000), 1),
    "grid": lambda: _weighted(graphs.grid(61, 67), 2),
    "quirk": lambda: graphs.lonestar_view(_weighted(graphs.grid(130, 33), 3)),
    "rows": lambda: _random(4000, [0, 1, 2, 3, 40], 4),
    "zero": lambda: _random(3000, [1, 2, 3, 4], 5, 0, 2),
    "limit": lambda: _random(900, [2, 3], 6, 999_999_998, 1_000_000_001),
    "many": lambda: _random(7, [9], 7, 1, 50), "eight": lambda: _random(5000, [8], 8),
    "nine": lambda: _random(5000, [9], 9), "one": lambda: _random(1, [1], 10),
}


@pytest.mark.parametrize("which", list(GRAPHS))
def test_sssp_narrow(which):
    g = GRAPHS[which]()
    with Runtime() as r:
        for src in (0, g.num_nodes // 2):
            want = oracle.lonestar_sssp(g, src)
            with PersistentApp(r, "lonestar_sssp", g, source=src) as a:
                for groups in (0, 1, 3, 0):
                    a.run(groups)
                    assert np.array_equal(a.result(), want), (which, src, groups)
