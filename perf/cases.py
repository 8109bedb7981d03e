"""The work a user of gpu_graphs_gb300 has it do, as measurable cases.

A case is a dict of plain values.  "path" names the entry point:

  bfs     Graph.bfs on a resident graph, levels into a device buffer
  parents Graph.bfs_parents on a resident graph, both arrays on the device
  multi   Graph.bfs_multi: k searches of one graph
  batch   gbfs_bfs_batch: one search in each member of a graph set, one launch
  build   Graph.from_edges from device arrays, the CSR exported to the device
  graph   the whole host path: host edge list -> Graph -> bfs -> host levels
  scan    exclusive_scan of an int32 device array
  serve   Server: a burst of queries over resident graphs, host results

Graphs ("kind"): "er" (uniform pairs), "rmat" (Graph500 quadrant weights
0.57/0.19/0.19, ids permuted) and "grid" (4-connected, 10 % of the edges
dropped, 0.1 % added within Manhattan radius 8).  "directed" keeps the edges
as stored, as the csr class does; otherwise the graph is symmetrised,
deduplicated and free of self-loops.  "hub" asks for hub-first rows, "wide"
for 64-bit row offsets.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gpu_graphs_gb300 as gb
from gpu_graphs_gb300 import _lib

GRAPH = {"kind": "rmat", "n": 0, "pairs": 0, "directed": False, "hub": False, "wide": False}


def _graph(kind: str, n: int, pairs: int, **opts) -> dict:
    return {**GRAPH, "kind": kind, "n": n, "pairs": pairs, **opts}


def _grid(side: int, **opts) -> dict:
    return {**GRAPH, "kind": "grid", "n": side * side, "pairs": 2 * side * (side - 1), "side": side, **opts}


def listed() -> list[dict]:
    return [
        # the smallest call: one query on a graph of a thousand vertices,
        # where launches, barriers and host work are all there is
        {"name": "bfs_er1000", "path": "bfs", "direction": gb.DIR_OPTIMIZING, **_graph("er", 1000, 4000)},
        # the reference's CPU-sized case: plain top-down search of a uniform random graph
        {"name": "bfs_er65536_topdown", "path": "bfs", "direction": gb.DIR_TOPDOWN, **_graph("er", 65536, 262144)},
        # the headline: direction-optimising search of a scale-22 power-law graph
        {"name": "bfs_rmat22", "path": "bfs", "direction": gb.DIR_OPTIMIZING,
         **_graph("rmat", 1 << 22, 1 << 26, hub=True)},
        # a road-like graph: thousands of levels of small frontiers
        {"name": "bfs_grid7000", "path": "bfs", "direction": gb.DIR_OPTIMIZING, **_grid(7000)},
        # a directed graph as its file stores it (odd vertex count), searched over its transpose
        {"name": "bfs_directed_rmat", "path": "bfs", "direction": gb.DIR_OPTIMIZING,
         **_graph("rmat", 300007, 4800111, directed=True)},
        # levels and BFS tree of a million-vertex power-law graph
        {"name": "parents_rmat20", "path": "parents", "direction": gb.DIR_OPTIMIZING, **_graph("rmat", 1 << 20, 1 << 24)},
        # 64 sources in one launch
        {"name": "multi64_rmat20", "path": "multi", "direction": gb.DIR_OPTIMIZING, "k": 64,
         **_graph("rmat", 1 << 20, 1 << 24)},
        # 512 uneven small graphs in one launch
        {"name": "batch512_er", "path": "batch", "count": 512, "n_min": 256, "n_max": 65536, "degree": 8},
        # CSR build of a power-law graph from device arrays (hub rows, all sort classes)
        {"name": "build_rmat22", "path": "build", **_graph("rmat", 1 << 22, 1 << 26, hub=True)},
        # the reference's own program: edge list in, CSR, one search, levels out, all on the host side
        {"name": "graph_grid1000", "path": "graph", "direction": gb.DIR_OPTIMIZING, **_grid(1000)},
        # the prefix-sum primitive
        {"name": "scan_2e28", "path": "scan", "n": 1 << 28},
        # a burst of queries at a server of 4 power-law graphs and 4 grids
        {"name": "serve_mix", "path": "serve", "graphs": 8, "scale_max": 18, "side_max": 1024, "queries": 60,
         "slots": 6},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, n_max: int, m_max: int, side_max: int, kinds=("er", "rmat", "grid"), **opts) -> dict:
    kind = rng.choice(kinds)
    if kind == "grid":
        return _grid(_log(rng, 48, side_max), **opts)
    n = _log(rng, 300, n_max)
    degree = rng.uniform(2, 16)
    return _graph(kind, n, max(1, min(int(n * degree), m_max)), **opts)


def draw(rng) -> dict:
    path = rng.choice(("bfs", "bfs", "bfs", "parents", "multi", "batch", "build", "build", "graph", "scan", "serve"))
    if path == "bfs":
        directed = rng.random() < 0.25
        wide = not directed and rng.random() < 0.15
        return {"path": path, "direction": rng.choice((gb.DIR_OPTIMIZING, gb.DIR_OPTIMIZING, gb.DIR_TOPDOWN)),
                **_draw_graph(rng, 1 << 22, 1 << 26, 3000, directed=directed, hub=rng.random() < 0.4, wide=wide)}
    if path == "parents":
        return {"path": path, "direction": gb.DIR_OPTIMIZING,
                **_draw_graph(rng, 1 << 21, 1 << 25, 1500, directed=rng.random() < 0.3)}
    if path == "multi":
        return {"path": path, "direction": gb.DIR_OPTIMIZING, "k": rng.randint(1, 64),
                **_draw_graph(rng, 1 << 20, 1 << 24, 700, directed=rng.random() < 0.2)}
    if path == "batch":
        n_min = _log(rng, 64, 1024)
        return {"path": path, "count": _log(rng, 3, 512), "n_min": n_min, "n_max": n_min * rng.randint(2, 60),
                "degree": rng.randint(4, 12)}
    if path == "build":
        directed = rng.random() < 0.3
        return {"path": path, **_draw_graph(rng, 1 << 22, 1 << 26, 4000, directed=directed, hub=rng.random() < 0.5,
                                            wide=rng.random() < 0.15)}
    if path == "graph":
        return {"path": path, "direction": gb.DIR_OPTIMIZING,
                **_draw_graph(rng, 1 << 20, 1 << 22, 1000, directed=rng.random() < 0.3)}
    if path == "scan":
        return {"path": path, "n": _log(rng, 1000, 1 << 28)}
    return {"path": path, "graphs": rng.randint(2, 8), "scale_max": rng.randint(12, 18),
            "side_max": rng.randint(100, 1024), "queries": rng.randint(4, 60), "slots": rng.randint(2, 6)}


# ---- inputs --------------------------------------------------------------------

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand_int(hi: int, size: int, g: torch.Generator) -> torch.Tensor:
    return torch.randint(0, hi, (size,), generator=g, device="cuda", dtype=torch.int64)


def _rmat_pairs(n: int, pairs: int, g: torch.Generator) -> tuple[torch.Tensor, torch.Tensor]:
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(pairs, dtype=torch.int64, device="cuda")
    v = torch.zeros(pairs, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        x = torch.rand(pairs, generator=g, device="cuda")
        bu = x >= 0.76
        bv = ((x >= 0.57) & ~bu) | (x >= 0.95)
        u = 2 * u + bu
        v = 2 * v + bv
    perm = torch.randperm(1 << scale, generator=g, device="cuda")
    # ids scaled from [0, 2^scale) to [0, n): the identity when n is a power of two
    return perm[u] * n >> scale, perm[v] * n >> scale


def _grid_pairs(side: int, g: torch.Generator) -> tuple[torch.Tensor, torch.Tensor]:
    ids = torch.arange(side * side, device="cuda").view(side, side)
    u = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    v = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    extra = u.numel() // 1000
    keep = torch.rand(u.numel(), generator=g, device="cuda") >= 0.1
    u, v = u[keep], v[keep]
    a = _rand_int(side * side, extra, g)
    dx = _rand_int(17, extra, g) - 8
    dy = _rand_int(17, extra, g) - 8
    r, c = a // side + dy, a % side + dx
    ok = (dx.abs() + dy.abs() <= 8) & (r >= 0) & (r < side) & (c >= 0) & (c < side)
    return torch.cat([u, a[ok]]), torch.cat([v, (r * side + c)[ok]])


def _pairs(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """The case's edge list, int64 on the GPU."""
    g = _generator(seed)
    if case["kind"] == "grid":
        return _grid_pairs(case["side"], g)
    if case["kind"] == "rmat":
        return _rmat_pairs(case["n"], case["pairs"], g)
    return _rand_int(case["n"], case["pairs"], g), _rand_int(case["n"], case["pairs"], g)


def _sources(u: torch.Tensor, k: int, seed: int) -> list[int]:
    """k start vertices that have an edge."""
    return u[_rand_int(u.numel(), k, _generator(seed + 7919))].tolist()


def _flags(case: dict) -> int:
    return ((0 if case["directed"] else gb.UNDIRECTED) | (gb.HUB_FIRST if case["hub"] else 0)
            | (gb.WIDE_ROWS if case["wide"] else 0))


def _build(case: dict, u: torch.Tensor, v: torch.Tensor) -> gb.Graph:
    src, dst = u.int(), v.int()
    torch.cuda.synchronize()  # the engine reads them on a stream of its own
    g = gb.Graph.from_edges(case["n"], src, dst, _flags(case))
    if "direction" in case:
        g.set_params(direction=case["direction"])
    return g


def _batch_members(case: dict, seed: int) -> list[tuple[int, torch.Tensor, torch.Tensor]]:
    g = _generator(seed)
    count, ratio = case["count"], case["n_max"] / case["n_min"]
    out = []
    for i in range(count):
        n = int(case["n_min"] * ratio ** (i / max(1, count - 1)))
        pairs = n * case["degree"] // 2
        out.append((n, _rand_int(n, pairs, g), _rand_int(n, pairs, g)))
    return out


def _serve_graphs(case: dict) -> list[dict]:
    """The server's graphs: power-law graphs and grids in turn, spread over the sizes."""
    out = []
    half = (case["graphs"] + 1) // 2
    for i in range(case["graphs"]):
        t = (i // 2 + 1) / half
        if i % 2 == 0:
            n = 1 << (12 + round((case["scale_max"] - 12) * t))
            out.append(_graph("rmat", n, 16 * n))
        else:
            out.append(_grid(int(64 * (case["side_max"] / 64) ** t)))
    return out


def _serve_queries(case: dict, pairs: list, seed: int) -> list[tuple[int, int]]:
    # the graphs are asked in a fixed random order, from start vertices of the seed
    which = np.random.RandomState(5).randint(0, len(pairs), case["queries"]).tolist()
    starts = [_sources(u, case["queries"], seed + i) for i, (u, _) in enumerate(pairs)]
    return [(w, starts[w][q]) for q, w in enumerate(which)]


def prepare(case: dict, seed: int):
    path = case["path"]
    if path == "scan":
        x = torch.randint(0, 64, (case["n"],), generator=_generator(seed), device="cuda", dtype=torch.int32)
        return {"path": path, "x": x}
    if path == "batch":
        members = _batch_members(case, seed)
        host = [(n, u.int().cpu().numpy(), v.int().cpu().numpy()) for n, u, v in members]
        gs = gb.GraphSet.from_edges(host)
        levels = torch.empty(int(gs.offsets[-1]), dtype=torch.int32, device="cuda")
        roots = np.array([int(u[0]) for _, u, _ in host], np.int32)
        ptrs = (ctypes.c_void_p * len(host))(*[levels.data_ptr() + 4 * int(o) for o in gs.offsets[:-1]])
        return {"path": path, "set": gs, "levels": levels, "roots": roots, "ptrs": ptrs}
    if path == "serve":
        graphs = _serve_graphs(case)
        pairs = [_pairs(c, seed + i) for i, c in enumerate(graphs)]
        srv = gb.Server(8 << 30, num_slots=case["slots"], batch_window_us=500, window_pct=10)
        ids = [srv.add_graph(_build(c, u, v)) for c, (u, v) in zip(graphs, pairs)]
        queries = [(ids[w], s, torch.empty(graphs[w]["n"], dtype=torch.int32, pin_memory=True).numpy())
                   for w, s in _serve_queries(case, pairs, seed)]
        return {"path": path, "server": srv, "queries": queries}
    u, v = _pairs(case, seed)
    if path == "graph":
        return {"path": path, "case": case, "src": u.int().cpu().numpy(), "dst": v.int().cpu().numpy(),
                "source": _sources(u, 1, seed)[0]}
    if path == "build":
        row = torch.empty(case["n"] + 1, dtype=torch.int64 if case["wide"] else torch.int32, device="cuda")
        col = torch.full((_capacity(case),), -1, dtype=torch.int32, device="cuda")
        state = {"path": path, "case": case, "src": u.int(), "dst": v.int(), "row": row, "col": col}
        torch.cuda.synchronize()
        return state
    state = {"path": path, "graph": _build(case, u, v), "sources": _sources(u, case.get("k", 1), seed)}
    shape = (case["k"], case["n"]) if path == "multi" else (case["n"],)
    state["levels"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    if path == "parents":
        state["parents"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    return state


# ---- one pass ------------------------------------------------------------------

def _run_build(state: dict):
    case = state["case"]
    g = gb.Graph.from_edges(case["n"], state["src"], state["dst"], _flags(case))
    export = _lib.lib.gbfs_graph_get_csr64 if g.wide else _lib.lib.gbfs_graph_get_csr
    _lib.check(export(g.handle, state["row"].data_ptr(), state["col"].data_ptr()), "gbfs_graph_get_csr")
    g.close()
    return state["row"], state["col"]  # the columns end with -1 where deduplication left fewer


def run(state: dict):
    path = state["path"]
    if path == "bfs":
        return state["graph"].bfs(state["sources"][0], out=state["levels"])
    if path == "parents":
        return state["graph"].bfs_parents(state["sources"][0], levels=state["levels"], parents=state["parents"])
    if path == "multi":
        return state["graph"].bfs_multi(state["sources"], out=state["levels"])
    if path == "batch":
        _lib.check(_lib.lib.gbfs_bfs_batch(state["set"]._h, state["roots"].ctypes.data, state["ptrs"], None),
                   "gbfs_bfs_batch")
        return state["levels"]
    if path == "build":
        return _run_build(state)
    if path == "graph":
        case = state["case"]
        g = gb.Graph.from_edges(case["n"], state["src"], state["dst"], _flags(case))
        g.set_params(direction=case["direction"])
        levels = g.bfs(state["source"])
        g.close()
        return levels
    if path == "scan":
        return gb.exclusive_scan(state["x"])
    srv = state["server"]
    tickets = [srv.submit(gid, source, out) for gid, source, out in state["queries"]]
    return [srv.wait(t)[0] for t in tickets]


# ---- what a pass cannot do without ---------------------------------------------------

def _stored(case: dict) -> int:
    """Stored edges, before deduplication (a dropped grid edge not counted)."""
    pairs = case["pairs"] * 0.9 if case["kind"] == "grid" else case["pairs"]
    return int(pairs if case["directed"] else 2 * pairs)


def _capacity(case: dict) -> int:
    """Room for the stored edges of any seed."""
    return max(1, case["pairs"] * (1 if case["directed"] else 2))


def _csr_bytes(case: dict) -> int:
    return (8 if case["wide"] else 4) * (case["n"] + 1) + 4 * _stored(case)


def work(case: dict) -> dict:
    """Bytes: the CSR (or the edge list) read once and the outputs written once."""
    path = case["path"]
    if path == "scan":
        return {"bytes": 12 * case["n"], "flops": 0}
    if path == "batch":
        count, ratio = case["count"], case["n_max"] / case["n_min"]
        n = sum(int(case["n_min"] * ratio ** (i / max(1, count - 1))) for i in range(count))
        return {"bytes": 8 * n + 4 * n * case["degree"], "flops": 0}
    if path == "serve":
        graphs = _serve_graphs(case)
        mean = sum(_csr_bytes(c) + 4 * c["n"] for c in graphs) / len(graphs)
        return {"bytes": int(mean * case["queries"]), "flops": 0}
    if path == "build":
        return {"bytes": 8 * case["pairs"] + _csr_bytes(case), "flops": 0}
    outputs = {"parents": 2, "multi": case.get("k", 1)}.get(path, 1)
    edges = 8 * case["pairs"] if path == "graph" else 0
    return {"bytes": _csr_bytes(case) + edges + 4 * case["n"] * outputs, "flops": 0}


# ---- the same results in plain torch --------------------------------------------------------

def _directed_edges(case: dict, u: torch.Tensor, v: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    return (u, v) if case.get("directed") else (torch.cat([u, v]), torch.cat([v, u]))


def _levels(n: int, u: torch.Tensor, v: torch.Tensor, starts: list[list[int]]) -> torch.Tensor:
    """Hop counts, one row per list of start vertices (-1: not reached)."""
    order = torch.argsort(u)
    col = v[order]
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
    k = max(1, min(len(starts), 200_000_000 // max(1, u.numel())))
    out = []
    for k0 in range(0, len(starts), k):
        lanes = starts[k0:k0 + k]
        level = torch.full((len(lanes) * n,), -1, dtype=torch.int64, device="cuda")
        claim = torch.empty_like(level)
        front = torch.tensor(sorted({i * n + s for i, l in enumerate(lanes) for s in l}), device="cuda")
        level[front] = 0
        depth = 0
        while front.numel():
            depth += 1
            vert = front % n
            begin = row[vert]
            degree = row[vert + 1] - begin
            ends = torch.cumsum(degree, 0)
            at = torch.repeat_interleave(degree)
            j = torch.arange(at.numel(), device="cuda")
            w = col[begin[at] + j - (ends - degree)[at]] + (front - vert)[at]
            w = w[level[w] < 0]
            level[w] = depth
            j = torch.arange(w.numel(), device="cuda")
            claim[w] = j
            front = w[claim[w] == j]
        out.append(level.view(len(lanes), n).int())
    return torch.cat(out)


def _parents(n: int, u: torch.Tensor, v: torch.Tensor, level: torch.Tensor) -> torch.Tensor:
    tree = (level[u] >= 0) & (level[v] == level[u] + 1)
    best = torch.full((n,), n, dtype=torch.int64, device="cuda")
    best.scatter_reduce_(0, v[tree], u[tree], "amin")
    return torch.where(best == n, -1, best).int()


def _csr(case: dict, u: torch.Tensor, v: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    n = case["n"]
    u, v = _directed_edges(case, u, v)
    key = u * n + v
    key = torch.sort(key).values if case["directed"] else torch.unique(key[u != v])
    at, col = key // n, key % n
    degree = torch.bincount(at, minlength=n)
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(degree, 0)
    if case["hub"]:  # each row's highest-degree entry (the first of several) swapped to its front
        pos = torch.arange(col.numel(), device="cuda") - row[at]
        rank = degree[col] * (1 << 31) + ((1 << 31) - 1 - pos)
        best = torch.zeros(n, dtype=torch.int64, device="cuda").scatter_reduce_(0, at, rank, "amax")
        has = degree > 0
        first = row[:-1][has]
        hub = first + (1 << 31) - 1 - best[has] % (1 << 31)
        a, b = col[first], col[hub]
        col[hub] = a
        col[first] = b
    out = torch.full((_capacity(case),), -1, dtype=torch.int32, device="cuda")
    out[:col.numel()] = col
    return row if case["wide"] else row.int(), out


def exact(case: dict, seed: int):
    path = case["path"]
    if path == "scan":
        x = prepare(case, seed)["x"].long()
        return torch.cumsum(x, 0) - x
    if path == "batch":
        us, vs, roots, base = [], [], [], 0
        for n, u, v in _batch_members(case, seed):
            us.append(u + base)
            vs.append(v + base)
            roots.append(int(u[0]) + base)
            base += n
        return _levels(base, *_directed_edges(case, torch.cat(us), torch.cat(vs)), [roots])[0]
    if path == "serve":
        graphs = _serve_graphs(case)
        pairs = [_pairs(c, seed + i) for i, c in enumerate(graphs)]
        queries = _serve_queries(case, pairs, seed)
        out = [None] * len(queries)
        for w, (c, (u, v)) in enumerate(zip(graphs, pairs)):
            mine = [i for i, (which, _) in enumerate(queries) if which == w]
            if mine:
                found = _levels(c["n"], *_directed_edges(c, u, v), [[queries[i][1]] for i in mine]).cpu().numpy()
                for i, levels in zip(mine, found):
                    out[i] = levels
        return out
    u, v = _pairs(case, seed)
    if path == "build":
        return _csr(case, u, v)
    starts = _sources(u, case.get("k", 1), seed)
    u, v = _directed_edges(case, u, v)
    levels = _levels(case["n"], u, v, [[s] for s in starts])
    if path == "multi":
        return levels
    if path == "parents":
        return levels[0], _parents(case["n"], u, v, levels[0])
    return levels[0].cpu().numpy() if path == "graph" else levels[0]
