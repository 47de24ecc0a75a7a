"""Colour's layout over one app's life: new priorities and new graphs of the same
size with no, few and as many hubs as the edges allow, in any order, fill the same
buffers; colours and round count against the oracle."""
import numpy as np
import pytest

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from oracle import oracle

pytestmark = pytest.mark.gpu

V, E = 3001, 33 * 900


def _graph(kind, seed):
    """E directed edges, none to its own vertex, rows by kind."""
    rng = np.random.default_rng(seed)
    d = np.zeros(V, np.int64)
    if kind == "none":
        d[:] = E // V
        d[rng.choice(V, E - d.sum(), replace=False)] += 1
    elif kind == "all":  # every edge on a vertex just past the threshold
        d[rng.choice(V, E // 33, replace=False)] = 33
    else:
        d[rng.choice(V, 7, replace=False)] = E // 7
        d[0] += E - d.sum()
    rp = np.zeros(V + 1, np.int32)
    rp[1:] = np.cumsum(d)
    row = np.repeat(np.arange(V), d)
    return graphs.Graph(rp, ((row + rng.integers(1, V, E)) % V).astype(np.int32))


@pytest.mark.parametrize("order", [("none", "all", "few"), ("few", "none", "all"),
                                   ("all", "few", "none", "all")])
def test_color_relayout(order):
    with Runtime(hub_threshold=32) as r:
        g = _graph(order[0], 1)
        with PersistentApp(r, "color", g) as a:
            for i, kind in enumerate(order):
                g = _graph(kind, i + 2)
                a.upload(g)
                for seed in (3, 4):
                    nv = graphs.seeded_node_values(V, seed)
                    a.set_node_values(nv)
                    want = oracle.color(g, nv)
                    for mode_groups in (0, 2):
                        st = a.run(mode_groups)
                        assert np.array_equal(a.result(), want), (kind, seed)
                        assert st.rounds == want.max()
