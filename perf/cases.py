"""The work users have this library do, as cases that can be timed.

Every case goes through the package's public entry points (``Graph.bfs``,
``Graph.bfs_many``, ``Graph.bfs_batch``, ``MultiGraph.bfs``, ``Server.run``) on
seeded synthetic graphs of the families the tests and the benchmark use: Graph500
R-MAT, Erdos-Renyi (mean degree 8), 2D grids and directed CSRs uploaded from the
host. A state holds what a program has in hand before the call: the graph handle on
the device, the sources and the output buffer.

Outputs are whole numbers (int32 level arrays and the counts of the call), which are
the same for every schedule of a traversal. Parent arrays are not among them: any
neighbour one level up is a right answer and two runs may differ.
"""
from __future__ import annotations

import numpy as np
import torch

from xbfs_b200 import BfsOptions, Graph, MultiGraph, learned, pick_sources
from xbfs_b200.api import Server

DEVICE = 0


def listed() -> list[dict]:
    return [
        # one query on a graph that fits in a cache: launch and call overhead
        {"name": "one_rmat_s10", "call": "bfs", "graph": "rmat", "scale": 10, "ef": 16, "order": "id",
         "policy": "heuristic", "out": "device"},
        # an interactive query whose answer the caller reads on the host
        {"name": "one_rmat_s16_host", "call": "bfs", "graph": "rmat", "scale": 16, "ef": 16, "order": "id",
         "policy": "heuristic", "out": "host"},
        # a stream of queries on a mid-size social graph, neighbours as loaded
        {"name": "many_rmat_s20", "call": "many", "graph": "rmat", "scale": 20, "ef": 16, "order": "id",
         "policy": "heuristic", "out": "device", "n": 16},
        # the benchmark's graph: scale 23, edge factor 32, hubs first in every list
        {"name": "many_rmat_s23", "call": "many", "graph": "rmat", "scale": 23, "ef": 32, "order": "degree",
         "policy": "heuristic", "out": "device", "n": 16},
        # the learned direction switch, rows copied to pinned host memory
        {"name": "many_rmat_s21_learned", "call": "many", "graph": "rmat", "scale": 21, "ef": 16, "order": "degree",
         "policy": "mlp", "out": "host", "n": 8},
        # no hubs: uniform random graph of an odd size
        {"name": "one_er_1m", "call": "bfs", "graph": "er", "n_vertices": 1000003, "order": "id",
         "policy": "heuristic", "out": "device"},
        # road-like: thousands of small levels
        {"name": "one_grid_4096", "call": "bfs", "graph": "grid", "width": 4096, "height": 4096, "order": "id",
         "policy": "heuristic", "out": "device"},
        # a directed link graph loaded from the caller's arrays: top-down only
        {"name": "one_directed", "call": "bfs", "graph": "directed", "n_vertices": 400009, "mean_degree": 12,
         "order": "id", "policy": "heuristic", "out": "device"},
        # one word of sources: centrality estimates from a sample of vertices
        {"name": "batch64_rmat_s18", "call": "batch", "graph": "rmat", "scale": 18, "ef": 16, "order": "id", "n": 64},
        # the benchmark's batched form: 512 sources, all distances to landmarks
        {"name": "batch512_rmat_s22", "call": "batch", "graph": "rmat", "scale": 22, "ef": 16, "order": "id",
         "n": 512},
        # many graphs of uneven size, one query each
        {"name": "multi_96", "call": "multi", "graphs": 96, "max_scale": 18, "max_vertices": 200000},
        # a burst of requests to a server that holds several graphs, answers on the host
        {"name": "serve_40", "call": "serve", "requests": 40, "scale": 20, "width": 1024, "height": 512,
         "n_vertices": 300007, "rate": 100000.0},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _draw_graph(rng, top_scale: int, top_vertices: int, top_side: int) -> dict:
    kind = rng.choice(["rmat", "rmat", "rmat", "er", "grid"])
    if kind == "rmat":
        return {"graph": "rmat", "scale": rng.randint(10, top_scale), "ef": rng.randint(4, 32)}
    if kind == "er":
        return {"graph": "er", "n_vertices": _log_int(rng, 1000, top_vertices)}
    return {"graph": "grid", "width": _log_int(rng, 3, top_side), "height": _log_int(rng, 3, top_side)}


def draw(rng) -> dict:
    call = rng.choice(["bfs", "bfs", "many", "many", "batch", "batch", "multi", "serve", "directed"])
    if call == "directed":
        return {"call": "bfs", "graph": "directed", "n_vertices": _log_int(rng, 1000, 500000),
                "mean_degree": rng.randint(2, 16), "order": rng.choice(["id", "degree"]), "policy": "heuristic",
                "out": rng.choice(["device", "host"])}
    if call in ("bfs", "many"):
        case = {"call": call, **_draw_graph(rng, 22, 4000000, 3000 if call == "bfs" else 200),
                "order": rng.choice(["id", "degree"]), "policy": rng.choice(["heuristic", "heuristic", "mlp", "beamer"]),
                "out": rng.choice(["device", "device", "host"])}
        if call == "many":
            case["n"] = rng.randint(2, 16)
        return case
    if call == "batch":
        return {"call": "batch", **_draw_graph(rng, 21, 2000000, 400), "order": rng.choice(["id", "degree"]),
                "n": _log_int(rng, 1, 512)}
    if call == "multi":
        return {"call": "multi", "graphs": _log_int(rng, 4, 128), "max_scale": rng.randint(11, 18),
                "max_vertices": _log_int(rng, 2000, 200000)}
    return {"call": "serve", "requests": rng.randint(4, 48), "scale": rng.randint(12, 20),
            "width": rng.randint(20, 1000), "height": rng.randint(20, 500),
            "n_vertices": _log_int(rng, 2000, 300000), "rate": float(rng.choice([10000, 100000]))}


def _directed(n: int, mean_degree: int, seed: int):
    """Out-lists of uneven length whose targets favour low ids; a few vertices link nowhere."""
    rng = np.random.default_rng(seed)
    deg = np.minimum(rng.geometric(1.0 / (mean_degree + 1), size=n) - 1, n - 1)
    beg = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(deg, out=beg[1:])
    csr = (n * rng.random(int(beg[-1])) ** 2).astype(np.int32)
    return beg, np.minimum(csr, n - 1)


def _graph(case: dict, seed: int) -> Graph:
    kind = case["graph"]
    if kind == "rmat":
        g = Graph.rmat(case["scale"], case["ef"], seed, device=DEVICE)
    elif kind == "er":
        g = Graph.er(case["n_vertices"], 8.0, seed, device=DEVICE)
    elif kind == "grid":
        g = Graph.grid(case["width"], case["height"], device=DEVICE)
    else:
        g = Graph.from_csr(*_directed(case["n_vertices"], case["mean_degree"], seed), device=DEVICE)
    if case["order"] == "degree":
        g.sort_adjacency("degree")
    return g


def prepare(case: dict, seed: int) -> dict:
    call = case["call"]
    if call == "multi":
        rng = np.random.default_rng(case["graphs"])  # the sizes belong to the case, the edges and sources to the seed
        half = case["graphs"] // 2
        graphs = [Graph.rmat(int(rng.integers(10, case["max_scale"] + 1)), int(rng.integers(8, 33)), seed + i,
                             device=DEVICE) for i in range(half)]
        graphs += [Graph.er(int(rng.integers(1000, case["max_vertices"] + 1)), 8.0, seed + i, device=DEVICE)
                   for i in range(half, case["graphs"])]
        srcs = np.array([pick_sources(g.offsets(), 1, seed + i)[0] for i, g in enumerate(graphs)], dtype=np.int32)
        mg = MultiGraph(graphs, device=DEVICE)
        return {"call": call, "multi": mg, "srcs": srcs,
                "levels": torch.empty(mg.total_V, dtype=torch.int32, device="cuda")}
    if call == "serve":
        rng = np.random.default_rng(seed)
        graphs = [Graph.rmat(case["scale"], 16, seed, device=DEVICE),
                  Graph.rmat(max(10, case["scale"] - 3), 16, seed + 1, device=DEVICE),
                  Graph.er(case["n_vertices"], 8.0, seed, device=DEVICE),
                  Graph.grid(case["width"], case["height"], device=DEVICE)]
        n = case["requests"]
        gid = (np.arange(n) % len(graphs)).astype(np.int32)
        begs = [g.offsets() for g in graphs]
        srcs = np.array([pick_sources(begs[k], 1, seed + i)[0] for i, k in enumerate(gid)], dtype=np.int32)
        arrival = np.cumsum(rng.exponential(1e6 / case["rate"], size=n))
        return {"call": call, "server": Server(graphs, device=DEVICE), "gid": gid, "srcs": srcs, "arrival": arrival}
    g = _graph(case, seed)
    n = case.get("n", 1)
    state = {"call": call, "g": g, "srcs": pick_sources(g.offsets(), n, seed)}
    if call == "batch":
        state["levels"] = torch.empty((n, g.V), dtype=torch.int32, device="cuda")
        return state
    if case["policy"] == "mlp":
        learned.install(learned.load(learned.DEFAULT_WEIGHTS)[0], device=DEVICE)
    state["opts"] = BfsOptions(policy=case["policy"])
    if call == "many":
        state["levels"] = (torch.empty((n, g.V), dtype=torch.int32, device="cuda") if case["out"] == "device"
                           else torch.empty((n, g.V), dtype=torch.int32, pin_memory=True).numpy())
    else:
        state["levels"] = torch.empty(g.V, dtype=torch.int32, device="cuda") if case["out"] == "device" else None
    return state


def run(state: dict):
    call = state["call"]
    if call == "bfs":
        r = state["g"].bfs(int(state["srcs"][0]), levels=state["levels"], opts=state["opts"])
    elif call == "many":
        r = state["g"].bfs_many(state["srcs"], levels=state["levels"], opts=state["opts"])
    elif call == "batch":
        r = state["g"].bfs_batch(state["srcs"], levels=state["levels"])
    elif call == "multi":
        r = state["multi"].bfs(state["srcs"], levels=state["levels"])
        return {"levels": r.levels, "edges_mc": int(r.edges_mc)}
    else:
        r = state["server"].run(state["gid"], state["srcs"], state["arrival"], to_host=True)
        return {"levels": r["levels"], "edges_mc": r["edges_mc"]}
    out = {"levels": r.levels, "depth": int(r.depth), "edges_mc": int(r.edges_mc)}
    if call != "batch":
        out["reached"] = int(r.reached)
    return out


def _size(case: dict) -> tuple[float, float]:
    """Vertices and (about) CSR entries of a case's graph."""
    kind = case["graph"]
    if kind == "rmat":
        v = 2.0 ** case["scale"]
        return v, 2.0 * case["ef"] * v * min(0.95, 0.5 + 0.02 * case["scale"])
    if kind == "er":
        return float(case["n_vertices"]), 8.0 * case["n_vertices"]
    if kind == "grid":
        w, h = case["width"], case["height"]
        return float(w * h), 2.0 * (2 * w * h - w - h)
    return float(case["n_vertices"]), float(case["mean_degree"]) * case["n_vertices"]


def work(case: dict) -> dict:
    """The CSR pair once (int64 offsets, int32 neighbours) and every level row once."""
    if case["call"] == "multi":
        half = case["graphs"] // 2
        scales = np.arange(10, case["max_scale"] + 1)
        v = half * float(np.mean(2.0 ** scales)), (case["graphs"] - half) * (500.0 + case["max_vertices"] / 2.0)
        e = v[0] * 2 * 20 * 0.8 + v[1] * 8
        return {"bytes": 12.0 * sum(v) + 4.0 * e, "flops": 0.0}
    if case["call"] == "serve":
        sizes = [(2.0 ** s, 2.0 ** s * 28) for s in (case["scale"], max(10, case["scale"] - 3))]
        sizes += [(case["n_vertices"], 8.0 * case["n_vertices"]),
                  (case["width"] * case["height"], 4.0 * case["width"] * case["height"])]
        total = sum(8 * v + 4 * e for v, e in sizes)
        return {"bytes": total + case["requests"] * 4.0 * sum(v for v, _ in sizes) / 4, "flops": 0.0}
    v, e = _size(case)
    return {"bytes": 8.0 * (v + 1) + 4.0 * e + 4.0 * v * case.get("n", 1), "flops": 0.0}
