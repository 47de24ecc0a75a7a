"""The framework's work as a user's program has it done, for timing: graph apps run
through `PersistentApp.run` + `result` on a graph that stays on the device, and
batches of jobs through `Batch.run` + `results`.  Results land in a pinned buffer
that the program keeps.

Graphs are the two families of this repository's benchmark: RMAT (0.57, 0.19,
0.19), symmetric, weights U[1,1000] per undirected edge, and 4-neighbour grids;
vertex counts need not be powers of two.  A seed picks the edges, the weights,
the priorities and the source.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gpu_workgroup_managment_gb300 import PersistentApp, Runtime, graphs
from gpu_workgroup_managment_gb300.batch import Batch

_RMAT_APPS = ("lonestar_bfs", "lonestar_sssp", "color", "mis", "sssp", "pagerank")


def listed() -> list[dict]:
    return [
        # one hop-count query on a small graph: a call is mostly launch and latency
        {"name": "bfs-rmat10", "app": "lonestar_bfs", "graph": "rmat", "n": 1024, "ef": 8},
        # the plain persistent BFS of the benchmark: hundreds of levels of little work
        # (the CSR as the Lonestar loader leaves it)
        {"name": "bfs-grid256", "app": "lonestar_bfs", "graph": "grid", "n": 256, "cols": 256,
         "view": True},
        # hop counts over a large, low-diameter graph
        {"name": "bfs-rmat20", "app": "lonestar_bfs", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # shortest paths on a road-like map: about a thousand dependent levels, ragged sides
        {"name": "sssp-grid", "app": "lonestar_sssp", "graph": "grid", "n": 509, "cols": 517},
        # shortest paths on the benchmark's large graph
        {"name": "sssp-rmat20", "app": "lonestar_sssp", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # scheduling by colours on the same graph: long chains of short rounds
        {"name": "color-rmat20", "app": "color", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # an independent set of the same graph: few rounds of much work
        {"name": "mis-rmat20", "app": "mis", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # the Pannotia form of shortest paths, a mid-sized graph of odd size
        {"name": "psssp-rmat18", "app": "sssp", "graph": "rmat", "n": 200_003, "ef": 12},
        # ranking a large graph, the benchmark's bandwidth case
        {"name": "pagerank-rmat22", "app": "pagerank", "graph": "rmat", "n": 1 << 22, "ef": 16,
         "iterations": 20},
        # ranking a small graph: launches and barriers
        {"name": "pagerank-rmat14", "app": "pagerank", "graph": "rmat", "n": 15_013, "ef": 10,
         "iterations": 20},
        # centrality of every vertex of a small graph
        {"name": "bc-rmat12", "app": "bc", "graph": "rmat", "n": 4096, "ef": 16},
        # many graphs of mixed size at once, one BFS and one SSSP job each
        {"name": "batch-128", "app": "batch", "graph": "mixed", "n": 128, "lo": 8.0, "hi": 16.5},
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    app = rng.choice(_RMAT_APPS + ("bc", "batch"))
    if app == "batch":
        lo = rng.uniform(6.0, 9.0)
        return {"app": app, "graph": "mixed", "n": rng.randint(16, 128), "lo": round(lo, 2),
                "hi": round(lo + rng.uniform(1.0, 7.5), 2)}
    if app == "bc":
        if rng.random() < 0.25:
            r = rng.randint(8, 24)
            return {"app": app, "graph": "grid", "n": r, "cols": rng.randint(8, 24)}
        return {"app": app, "graph": "rmat", "n": _log_uniform(rng, 200, 4096),
                "ef": rng.randint(4, 16)}
    if rng.random() < 0.3:
        c = {"app": app, "graph": "grid", "n": _log_uniform(rng, 16, 512),
             "cols": _log_uniform(rng, 16, 512)}
    else:
        c = {"app": app, "graph": "rmat", "ef": rng.randint(4, 16),
             "n": _log_uniform(rng, 500, (1 << 21) if app == "pagerank" else (1 << 20))}
    if app in ("lonestar_bfs", "lonestar_sssp"):
        c["view"] = rng.random() < 0.5
    if app == "pagerank":
        c["iterations"] = rng.randint(5, 20)
    return c


# ---- inputs -----------------------------------------------------------------

def _rmat(n: int, ef: int, seed: int, weights: bool) -> graphs.Graph:
    """Symmetric RMAT graph on n vertices, about n*ef undirected edges before
    duplicates go, rows sorted, no self loops."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    s = max(1, (n - 1).bit_length())
    m = int(ef * n * ((1 << s) / n) ** 2)  # edges outside the n vertices are dropped
    u = torch.zeros(m, dtype=torch.int32, device=dev)
    v = torch.zeros(m, dtype=torch.int32, device=dev)
    for _ in range(s):
        r = torch.rand(m, device=dev, generator=gen)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(1 << s, device=dev, generator=gen).to(torch.int32)
    u, v = perm[u.long()].long(), perm[v.long()].long()
    keep = (u < n) & (v < n) & (u != v)
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat([u * n + v, v * n + u]))
    del u, v, r, keep, perm
    row = torch.div(key, n, rounding_mode="floor")
    col = key - row * n
    rp = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    rp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    wt = None
    if weights:
        x = torch.minimum(row, col) * n + torch.maximum(row, col)
        x = (x + seed) * 0x1E3779B97F4A7C15
        x = (x ^ (x >> 29)) * 0x3F58476D1CE4E5B9
        wt = (((x >> 33) & 0x7FFFFFFF) % 1000 + 1).to(torch.int32).cpu().numpy().astype(np.uint32)
    return graphs.Graph(rp.to(torch.int32).cpu().numpy(), col.to(torch.int32).cpu().numpy(), wt,
                        f"rmat{n}")


def _graph(case: dict, seed: int, weights: bool) -> graphs.Graph:
    if case["graph"] == "rmat":
        g = _rmat(case["n"], case["ef"], seed, weights)
    else:
        g = graphs.grid(case["n"], case["cols"])
        if weights:
            g.weights = graphs.uniform_weights(g, seed)
    return graphs.lonestar_view(g) if case.get("view") else g


def _source(g: graphs.Graph, seed: int) -> int:
    """A random vertex that has an edge (the end of a random one)."""
    rng = np.random.default_rng(seed)
    return int(g.col[rng.integers(0, g.num_edges)]) if g.num_edges else 0


def _batch_sizes(case: dict) -> list[float]:
    """log2 of the vertex counts, spread evenly over [lo, hi] in a mixed order."""
    return [case["lo"] + (case["hi"] - case["lo"]) * ((i * 0.6180339887) % 1.0)
            for i in range(case["n"])]


def _pinned(n: int, dtype) -> np.ndarray:
    return torch.empty(max(n, 1), dtype=dtype, pin_memory=True).numpy()[:n]


_OUT = {"mis": torch.int32, "color": torch.int32, "sssp": torch.int32,
        "pagerank": torch.float32, "bc": torch.float32}


def prepare(case: dict, seed: int) -> dict:
    rt = Runtime()
    if case["app"] == "batch":
        gs, jobs = [], []
        rng = np.random.default_rng(seed)
        for i, x in enumerate(_batch_sizes(case)):
            n = int(round(2 ** x))
            if i % 2 == 0:
                g = _rmat(n, 4 + (5 * i) % 13, seed * 131 + i, True)
            else:
                r = max(2, int(round(n ** 0.5)))
                g = graphs.grid(r, max(2, n // r))
                g.weights = graphs.uniform_weights(g, seed * 131 + i)
            gs.append(g)
            jobs += [(i, "bfs", int(rng.integers(0, g.num_nodes))),
                     (i, "sssp", int(rng.integers(0, g.num_nodes)))]
        b = Batch(rt, gs, jobs)
        return {"batch": b, "out": _pinned(int(b.offsets[-1]), torch.int32).view(np.uint32)}
    g = _graph(case, seed, case["app"] in ("lonestar_sssp", "sssp"))
    kw = {}
    if case["app"] in ("color", "mis"):
        kw["node_values"] = graphs.seeded_node_values(g.num_nodes, seed)
    elif case["app"] == "pagerank":
        kw["iterations"] = case["iterations"]
    elif case["app"] != "bc":
        kw["source"] = _source(g, seed)
    a = PersistentApp(rt, case["app"], g, **kw)
    out = _pinned(g.num_nodes, _OUT.get(case["app"], torch.int32))
    if case["app"] in ("lonestar_bfs", "lonestar_sssp"):
        out = out.view(np.uint32)
    return {"app": a, "out": out}


def run(state: dict):
    if "batch" in state:
        state["batch"].run()
        return state["batch"].results(state["out"])
    state["app"].run()
    return state["app"].result(state["out"])


# ---- what the path cannot do without -------------------------------------------

def _sizes(case: dict) -> tuple[float, float]:
    """(vertices, directed edges): RMAT counts before duplicates go."""
    if case["graph"] == "rmat":
        return case["n"], 2.0 * case["n"] * case["ef"]
    v = case["n"] * case["cols"]
    return v, 4.0 * v - 2.0 * (case["n"] + case["cols"])


def work(case: dict) -> dict:
    """Each array of the graph read once, the results written once, and one
    operation for each edge that the result depends on: an iteration of PageRank
    has a multiply-add for every edge, a source of the centrality one forward
    and two backward."""
    if case["app"] == "batch":
        by = fl = 0.0
        for i, x in enumerate(_batch_sizes(case)):
            v = 2.0 ** x
            e = v * 2.0 * (4 + (5 * i) % 13) if i % 2 == 0 else 4.0 * v
            by += 8.0 * e + 4.0 * v + 8.0 * v  # columns, weights, rows, two results
            fl += 3.0 * e
        return {"bytes": by, "flops": fl}
    v, e = _sizes(case)
    w = {"bytes": 4.0 * e + 8.0 * v, "flops": e}
    if case["app"] in ("lonestar_sssp", "sssp"):
        w = {"bytes": 8.0 * e + 8.0 * v, "flops": 2.0 * e}
    elif case["app"] in ("color", "mis"):
        w["bytes"] += 4.0 * v  # priorities
    elif case["app"] == "pagerank":
        w["flops"] = 2.0 * e * case["iterations"]
    elif case["app"] == "bc":
        w["flops"] = 4.0 * v * e
    return w


# ---- the floating-point results in 64 bits ---------------------------------------

def _exact_pagerank(g: graphs.Graph, iterations: int) -> np.ndarray:
    dev, v = torch.device("cuda"), g.num_nodes
    deg = torch.from_numpy(np.diff(g.row_ptr).astype(np.int64)).to(dev)
    col = torch.from_numpy(g.col).to(dev).long()
    row = torch.repeat_interleave(torch.arange(v, device=dev), deg)
    pr = torch.full((v,), 1.0 / v, dtype=torch.float64, device=dev)
    for _ in range(iterations):
        c = torch.where(deg > 0, pr / deg.clamp(min=1), torch.zeros_like(pr))
        s = torch.zeros_like(pr).index_add_(0, row, c[col])
        pr = 0.15 / v + 0.85 * (s + pr[deg == 0].sum() / v)
    return pr.cpu().numpy()


def _exact_bc(g: graphs.Graph) -> np.ndarray:
    """Brandes' dependencies of every source, a block of sources at a time."""
    dev, v = torch.device("cuda"), g.num_nodes
    a = torch.sparse_csr_tensor(torch.from_numpy(g.row_ptr).long(),
                                torch.from_numpy(g.col).long(),
                                torch.ones(g.num_edges, dtype=torch.float64), (v, v)).to(dev)
    bc = torch.zeros(v, dtype=torch.float64, device=dev)
    for s0 in range(0, v, 1024):
        src = torch.arange(s0, min(s0 + 1024, v), device=dev)
        k = torch.arange(src.numel(), device=dev)
        dist = torch.full((v, src.numel()), -1, dtype=torch.int32, device=dev)
        rho = torch.zeros((v, src.numel()), dtype=torch.float64, device=dev)
        dist[src, k], rho[src, k] = 0, 1.0
        level = 0
        while True:
            n = a @ torch.where(dist == level, rho, 0.0)
            new = (n > 0) & (dist < 0)
            if not bool(new.any()):
                break
            level += 1
            dist[new] = level
            rho = torch.where(new, n, rho)
        sigma = torch.zeros_like(rho)
        for lv in range(level, 0, -1):
            t = a @ torch.where(dist == lv, (1.0 + sigma) / rho.clamp(min=1e-300), 0.0)
            sigma = torch.where(dist == lv - 1, rho * t, sigma)
        sigma[src, k] = 0.0
        bc += sigma.sum(1)
    return bc.cpu().numpy()


def exact(case: dict, seed: int):
    """PageRank and centrality; every other result is whole numbers."""
    if case["app"] == "pagerank":
        return _exact_pagerank(_graph(case, seed, False), case["iterations"])
    if case["app"] == "bc":
        return _exact_bc(_graph(case, seed, False))
    return None
