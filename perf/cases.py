"""Timed cases of the engine's public entry points (ctypes binding and C ABI).

Four kinds of case:
  update    one call (or one call per phase) that applies update batches of a
            maintained BFS / SSSP / CC state and reads the values back;
  query     multi-source BFS / SSSP on the current graph into device memory;
  pagerank  one update batch of a maintained PageRank and its ranks;
  serve     a burst of updates and queries through the serving loop.

Graphs are R-MAT (a/b/c/d = 0.57/0.19/0.19/0.05, vertex ids permuted, vertex
0 kept as the hub, self-loops and duplicates removed; `vertices` need not be
a power of two) or road-like grids.  A batch deletes edges that are in the
graph and inserts edges that are not: half of them R-MAT (grid) edges, half
uniform pairs (grid: pairs within 3 rows and columns).  So that a pass can
follow another on one state, every batch slot keeps a pool of edge sets, half
of them in the graph at any time; a pass deletes one that is in and inserts
one that is out, both chosen by the state's own generator.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from coincgraph_b200.engine import FLAG_PR_FP64, FLAG_WEIGHT_U255, Engine

POOL = 16  # edge sets per batch slot; half of them are in the graph
MASK = 0xFFFFFFFF
INF = 1 << 40


def listed():
    return [
        # The smallest update: a few dozen edges of a small graph from host arrays; latency and launches.
        _update("bfs-update-1k", algo="bfs", vertices=1000, batch=32, mode="host", cache=1.0),
        # The plain configuration: R-MAT s16, all rows resident, 1,000 deletions and 1,000 insertions.
        _update("bfs-update-s16", algo="bfs", vertices=1 << 16, batch=1000, mode="host", cache=2.0),
        # The benchmark's larger-than-cache SSSP stream at a quarter of its size: four batches in one call.
        _update("sssp-stream-s22", algo="sssp", vertices=1 << 22, batch=25_000, batches=4, mode="stream", cache=0.25),
        # Min-label components of a symmetric graph under batches of uneven size, all in one call.
        _update("cc-uneven-300k", algo="cc", vertices=300_007, symmetric=True, batch=500, batch_max=50_000, batches=6,
                mode="stream", cache=4.0),
        # High diameter: a road-like grid with local insertions, device arrays.
        _update("sssp-road-511", algo="sssp", graph="grid", vertices=511 * 511, batch=251, mode="device", cache=1.0),
        # The reference's own flow: one call per phase, values read after each, every row in host memory.
        _update("sssp-phases-hostrows", algo="sssp_u255", vertices=200_003, batch=2001, mode="phases", cache=0.0),
        # 64 BFS sources as one bitmask wave on a symmetric graph.
        _query("bfs-64-sources-s20", algo="bfs", vertices=1 << 20, symmetric=True, sources=64, width=64),
        # A partly filled wave of SSSP queries, as the serving loop forms them.
        _query("sssp-13-sources-s19", algo="sssp", vertices=1 << 19, sources=13, width=13),
        # One BFS query on a large graph, alone in its wave.
        _query("bfs-1-source-s22", algo="bfs", vertices=1 << 22, sources=1, width=1),
        # PageRank kept up to date in FP32 with compensated sums.
        _pagerank("pagerank-fp32-s18", vertices=1 << 18, batch=2000, fp64=False),
        # PageRank in FP64 on a smaller ragged graph.
        _pagerank("pagerank-fp64-50k", vertices=50_021, batch=501, fp64=True),
        # A burst through the serving loop: queries, an update, queries that see it.
        _serve("serve-mix-s17", vertices=1 << 17, batch=2000, queries=16),
    ]


def draw(rng):
    kind = rng.choice(["update", "update", "update", "query", "query", "pagerank", "serve"])
    if kind == "update":
        algo = rng.choice(["bfs", "sssp", "sssp_u255", "cc"])
        if rng.random() < 0.2:
            side = _log(rng, 40, 511)
            return _update(None, algo=algo, graph="grid", vertices=side * side, batch=_log(rng, 20, max(21, side // 2)),
                           mode=rng.choice(["host", "device", "phases"]), cache=1.0)
        n = _log(rng, 1000, 1 << 21)
        mode = rng.choice(["host", "device", "stream", "phases"])
        small = _log(rng, 20, max(21, min(25_000, n // 40)))
        return _update(None, algo=algo, vertices=n, symmetric=rng.random() < 0.3, batch=small,
                       batch_max=min(50_000, small * rng.choice([1, 1, 8])) if mode == "stream" else 0,
                       batches=rng.randint(2, 6) if mode == "stream" else 1, mode=mode,
                       cache=rng.choice([0.0, 0.01, 0.1, 1.0, 4.0]))
    if kind == "query":
        n = _log(rng, 1000, 1 << 20)
        k = _log(rng, 1, 64)
        return _query(None, algo=rng.choice(["bfs", "bfs", "sssp", "sssp_u255"]), vertices=n,
                      symmetric=rng.random() < 0.5, sources=k, width=rng.choice([k, min(k, 7), 64]))
    if kind == "pagerank":
        n = _log(rng, 1000, 1 << 18)
        return _pagerank(None, vertices=n, batch=_log(rng, 20, max(21, min(2000, n // 40))), fp64=rng.random() < 0.4)
    n = _log(rng, 1000, 1 << 17)
    return _serve(None, vertices=n, batch=_log(rng, 20, max(21, min(2000, n // 40))), queries=2 * rng.randint(2, 12))


def _case(name, **kw):
    return {"name": name, **kw} if name else kw


def _update(name, algo, vertices, batch, mode, cache, graph="rmat", symmetric=False, batch_max=0, batches=1):
    return _case(name, kind="update", algo=algo, graph=graph, vertices=vertices, symmetric=symmetric, batch=batch,
                 batch_max=batch_max, batches=batches, mode=mode, cache=cache)


def _query(name, algo, vertices, sources, width, symmetric=False):
    return _case(name, kind="query", algo=algo, graph="rmat", vertices=vertices, symmetric=symmetric, sources=sources,
                 width=width, cache=4.0)


def _pagerank(name, vertices, batch, fp64):
    return _case(name, kind="pagerank", graph="rmat", vertices=vertices, symmetric=False, batch=batch, batch_max=0,
                 batches=1, fp64=fp64, cache=4.0)


def _serve(name, vertices, batch, queries):
    return _case(name, kind="serve", algo="sssp", graph="rmat", vertices=vertices, symmetric=False, batch=batch,
                 batch_max=0, batches=1, queries=queries, cache=4.0)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---------------------------------------------------------------- inputs


def _slot_sizes(case):
    """Deletions (and as many insertions) of every batch of a pass; even on symmetric graphs."""
    lo, hi, k = case["batch"], max(case["batch"], case["batch_max"]), case["batches"]
    sizes = [int(round(lo * (hi / lo) ** (((i + 1) * 0.6180339887) % 1.0))) for i in range(k)] if hi > lo else [lo] * k
    return [2 * (s // 2) for s in sizes] if case["symmetric"] else sizes


def _pack(u, v):
    return (u << 32) | v


def _rmat(n, gen, symmetric):
    """Sorted distinct edges u << 32 | v of an R-MAT graph (symmetric: u < v only)."""
    bits = max(1, (n - 1).bit_length())
    m = 16 * n
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(bits):
        r = torch.rand(m, device="cuda", generator=gen)
        u = (u << 1) | (r >= 0.76)
        v = (v << 1) | (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(1 << bits, device="cuda", generator=gen)
    zero = (perm == 0).nonzero()[0, 0]
    perm[zero] = perm[0].clone()
    perm[0] = 0
    u, v = perm[u], perm[v]
    if symmetric:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    keep = (u != v) & (u < n) & (v < n)
    return torch.unique(_pack(u[keep], v[keep]))


def _grid(n):
    side = math.isqrt(n)
    at = torch.arange(n, device="cuda")
    i, j = at // side, at % side
    pairs = []
    for di, dj in ((0, 1), (0, -1), (1, 0), (-1, 0)):
        ok = (i + di >= 0) & (i + di < side) & (j + dj >= 0) & (j + dj < side)
        pairs.append(_pack(at[ok], (i + di)[ok] * side + (j + dj)[ok]))
    return torch.cat(pairs).sort().values


def _new_edges(case, keys, count, gen):
    """Distinct edges that are not in the sorted `keys`."""
    n = case["vertices"]
    draws = 2 * count + 256
    u = torch.randint(n, (draws,), device="cuda", generator=gen)
    if case["graph"] == "grid":
        side = math.isqrt(n)
        di, dj = (torch.randint(-3, 4, (draws,), device="cuda", generator=gen) for _ in range(2))
        i, j = u // side + di, u % side + dj
        v = i * side + j
        ok = (i >= 0) & (i < side) & (j >= 0) & (j < side)
    else:
        v = torch.randint(n, (draws,), device="cuda", generator=gen)
        ok = torch.ones_like(v, dtype=torch.bool)
    if case["symmetric"]:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    found = torch.unique(_pack(u, v)[ok & (u != v)])
    at = torch.searchsorted(keys, found).clamp(max=keys.numel() - 1)
    found = found[keys[at] != found]
    return found[torch.randperm(found.numel(), device="cuda", generator=gen)[:count]]


def _edges_of(keys, symmetric):
    u, v = keys >> 32, keys & MASK
    return (torch.cat([u, v]), torch.cat([v, u])) if symmetric else (u, v)


def _inputs(case, seed):
    """(sorted keys in the graph at first, per slot the POOL edge sets; the even ones are in the graph)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    sym = case["symmetric"]
    keys = _grid(case["vertices"]) if case["graph"] == "grid" else _rmat(case["vertices"], gen, sym)
    sizes = [s // 2 if sym else s for s in (_slot_sizes(case) if "batch" in case else [])]
    if not sizes:
        return keys, []
    old = [s // 2 for s in sizes]
    new = [s - o for s, o in zip(sizes, old)]
    picked = torch.randperm(keys.numel(), device="cuda", generator=gen)[: POOL * sum(old)]
    fresh = _new_edges(case, keys, POOL * sum(new), gen)
    slots, a, b = [], 0, 0
    present = torch.ones(keys.numel(), dtype=torch.bool, device="cuda")
    added = []
    for so, sn in zip(old, new):
        sets = []
        for p in range(POOL):
            part = torch.cat([keys[picked[a: a + so]], fresh[b: b + sn]])
            if p % 2:
                present[picked[a: a + so]] = False
            else:
                added.append(fresh[b: b + sn])
            a, b = a + so, b + sn
            sets.append(part[torch.randperm(part.numel(), device="cuda", generator=gen)])
        slots.append(sets)
    return torch.cat([keys[present], *added]).sort().values, slots


def _engine(case, keys, algo, **options):
    n = case["vertices"]
    u, v = _edges_of(keys, case["symmetric"])
    if case["symmetric"]:
        both = _pack(u, v).sort().values
        u, v = both >> 32, both & MASK
    xadj = np.zeros(n + 1, dtype=np.uint64)
    xadj[1:] = torch.bincount(u, minlength=n).cumsum(0).cpu().numpy()
    flags = FLAG_WEIGHT_U255 if case.get("algo") == "sssp_u255" else 0
    sizes = _slot_sizes(case) if "batch" in case else [0]
    # Arena headroom of a long-running stream (blocks left by relocated rows are not reused): up to four slots per
    # inserted edge over a few hundred large to several thousand small passes.
    slots = sum(sizes) * 0.8 / (4e-5 + 4e-9 * sum(sizes))
    eng = Engine(algo, cache_gib=case["cache"], flags=flags | options.pop("flags", 0),
                 headroom_pct=int(25 + 100 * slots / u.numel()), max_batch=max(sizes), **options)
    eng.load_csr(n, xadj, v.to(torch.int32).cpu().numpy().view(np.uint32))
    eng.init()
    return eng


def _batches(slots, symmetric, host):
    """Per slot and set the (u, v) arrays of its edges, on the host (numpy uint32) or the device (int32)."""
    def arrays(keys):
        u, v = (x.to(torch.int32) for x in _edges_of(keys, symmetric))
        return (u.cpu().numpy().view(np.uint32), v.cpu().numpy().view(np.uint32)) if host else (u, v)
    return [[arrays(s) for s in sets] for sets in slots]


def prepare(case, seed):
    keys, slots = _inputs(case, seed)
    rng = random.Random(seed)
    n = case["vertices"]
    state = {"case": case, "rng": rng, "inside": [list(range(0, POOL, 2)) for _ in slots],
             "outside": [list(range(1, POOL, 2)) for _ in slots]}
    if case["kind"] == "update":
        state["eng"] = _engine(case, keys, "sssp" if case["algo"] == "sssp_u255" else case["algo"])
        state["batches"] = _batches(slots, case["symmetric"], case["mode"] in ("host", "phases"))
        state["values"] = [torch.empty(n, dtype=torch.int32, pin_memory=True)
                           for _ in range(2 if case["mode"] == "phases" else 1)]
    elif case["kind"] == "query":
        state["eng"] = _engine(case, keys, "sssp" if case["algo"] == "sssp_u255" else case["algo"])
        state["sources"] = np.array(_sources(keys, rng, case["sources"]), dtype=np.uint32)
        state["out"] = torch.empty((case["sources"], n), dtype=torch.int32, device="cuda")
    elif case["kind"] == "pagerank":
        state["eng"] = _engine(case, keys, "pr", pr_epsilon=1e-9, pr_max_rounds=100_000,
                               flags=FLAG_PR_FP64 if case["fp64"] else 0)
        state["batches"] = _batches(slots, False, True)
        state["rank"] = torch.empty(n, dtype=torch.float64 if case["fp64"] else torch.float32, pin_memory=True)
    else:
        state["eng"] = _engine(case, keys, "sssp")
        state["batches"] = _batches(slots, False, True)
        state["sources"] = _sources(keys, rng, case["queries"])
        state["out"] = np.empty((case["queries"], n), dtype=np.uint32)
        state["eng"].serve_start()
    return state


def _sources(keys, rng, count):
    """Uniform vertices with out-edges."""
    at = torch.tensor([rng.randrange(keys.numel()) for _ in range(count)], device="cuda")
    return (keys[at] >> 32).cpu().tolist()


# ---------------------------------------------------------------- one pass


def _next(state):
    """Per slot the set to delete (in the graph) and the set to insert (not in it)."""
    picks = []
    for sets, inside, outside in zip(state["batches"], state["inside"], state["outside"]):
        i, j = state["rng"].randrange(len(inside)), state["rng"].randrange(len(outside))
        gone, come = inside[i], outside[j]
        inside[i], outside[j] = come, gone
        picks.append((*sets[gone], *sets[come]))
    return picks


def _read_values(eng, out):
    eng._check(eng.lib.cig_get_values(eng.h, ctypes.c_void_p(out.data_ptr())))


def run(state):
    case, eng = state["case"], state["eng"]
    if case["kind"] == "query":
        eng.query_device("bfs" if case["algo"] == "bfs" else "sssp", state["sources"], state["out"],
                         width=case["width"])
        return state["out"]
    picks = _next(state)
    if case["kind"] == "pagerank":
        eng.apply_batch(*picks[0])
        rank = ctypes.c_void_p(state["rank"].data_ptr())
        eng._check((eng.lib.cig_get_pr64 if case["fp64"] else eng.lib.cig_get_pr)(eng.h, rank, None))
        return state["rank"]
    if case["kind"] == "serve":
        tickets = []
        for q, source in enumerate(state["sources"]):
            if 2 * q == len(state["sources"]):
                update = eng.submit_update(*picks[0])
            tickets.append(eng.submit_query(("bfs", "sssp")[q % 2], source, state["out"][q]))
        ok = eng.wait(update)["status"]
        return {"out": state["out"], "status": [ok] + [eng.wait(t)["status"] for t in tickets]}
    values = state["values"]
    if case["mode"] == "phases":
        du, dv, au, av = picks[0]
        stats = [eng.delete_phase(du, dv)]
        _read_values(eng, values[0])
        stats.append(eng.insert_phase(au, av))
        _read_values(eng, values[1])
    elif case["mode"] == "host":
        stats = [eng.apply_batch(*picks[0])]
        _read_values(eng, values[0])
    elif case["mode"] == "device":
        stats = [eng.apply_batch_device(*picks[0]).as_dict()]
        _read_values(eng, values[0])
    else:
        stats = [s.as_dict() for s in eng.apply_batches_device(picks, digests=False)[0]]
        _read_values(eng, values[0])
    return {"values": values, "missing": sum(s["missing_deletes"] for s in stats),
            "invalid": sum(s["invalid_additions"] for s in stats)}


# ---------------------------------------------------------------- work and tolerance


def work(case):
    """What a pass cannot do without: the batch arrays, one word of both adjacencies and of the vertex state per
    changed edge, and the values read back; a query reads every row once; PageRank reads every row and rank once."""
    n = case["vertices"]
    m = n * (4 if case["graph"] == "grid" else 32 if case["symmetric"] else 16)
    changed = 2 * sum(_slot_sizes(case)) if "batch" in case else 0
    update = changed * (8 + 2 * 4 + 8)
    if case["kind"] == "update":
        return {"bytes": update + 4 * n * (2 if case["mode"] == "phases" else 1), "flops": 0}
    if case["kind"] == "query":
        waves = -(-case["sources"] // case["width"])
        return {"bytes": waves * (4 * m + 16 * n) + 4 * n * case["sources"], "flops": 0}
    if case["kind"] == "pagerank":
        word = 8 if case["fp64"] else 4
        return {"bytes": changed * 16 + 4 * m + (16 + 2 * word) * n, "flops": 2 * m}
    return {"bytes": update + 4 * (4 * m + 16 * n) + 4 * n * case["queries"], "flops": 0}


def tolerance(case):
    if case["kind"] != "pagerank":
        return "exact"
    # Measured against exact(): FP64 2e-9 (the residual threshold 1e-9 decides), FP32 5e-8 and at most 3e-7.
    return {"rel": 1e-8, "max": 3e-8} if case["fp64"] else {"rel": 2.5e-7, "max": 1.5e-6}


# ---------------------------------------------------------------- 64-bit results in plain torch


def _weights(algo, u, v):
    if algo == "bfs":
        return torch.ones_like(u)
    if algo == "sssp":
        return (u + v) % 128 + 1
    x = (u * 0x9E3779B1 + v * 0x85EBCA77) & MASK
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & MASK
    x = ((x ^ (x >> 15)) * 0x846CA68B) & MASK
    return 1 + (x ^ (x >> 16)) % 255


def _solve(algo, n, u, v, source):
    """Distances from `source`, or (algo "cc") the smallest id that reaches each vertex."""
    d = torch.arange(n, device="cuda") if algo == "cc" else torch.full((n,), INF, device="cuda")
    w = torch.zeros_like(u) if algo == "cc" else _weights(algo, u, v)
    if algo != "cc":
        d[source] = 0
    while True:
        e = d.scatter_reduce(0, v, d[u] + w, "amin")
        if torch.equal(e, d):
            return torch.where(d >= INF, -1, d).to(torch.int32)
        d = e


def exact(case, seed):
    keys, slots = _inputs(case, seed)
    n, sym = case["vertices"], case["symmetric"]
    rng = random.Random(seed)
    if case["kind"] == "query":
        u, v = _edges_of(keys, sym)
        return torch.stack([_solve(case["algo"], n, u, v, s) for s in _sources(keys, rng, case["sources"])])
    sources = _sources(keys, rng, case["queries"]) if case["kind"] == "serve" else []
    state = {"rng": rng, "batches": [[(s,) for s in sets] for sets in slots],
             "inside": [list(range(0, POOL, 2)) for _ in slots], "outside": [list(range(1, POOL, 2)) for _ in slots]}
    before = keys
    middle = after = keys
    for gone, come in _next(state):
        middle = after[~torch.isin(after, gone)]
        after = torch.cat([middle, come])
    if case["kind"] == "pagerank":
        u, v = _edges_of(after, sym)
        share = 0.85 / torch.bincount(u, minlength=n).clamp(min=1).double()
        x = torch.ones(n, dtype=torch.float64, device="cuda")
        for _ in range(2000):
            y = torch.full_like(x, 0.15).index_add_(0, v, (x * share)[u])
            moved = float((y - x).abs().max() / y.max())
            x = y
            if moved < 1e-15:
                break
        return x
    if case["kind"] == "serve":
        rows = []
        for q, s in enumerate(sources):
            u, v = _edges_of(before if 2 * q < len(sources) else after, sym)
            rows.append(_solve(("bfs", "sssp")[q % 2], n, u, v, s))
        return {"out": torch.stack(rows), "status": [0] * (1 + len(sources))}
    graphs = [middle, after] if case["mode"] == "phases" else [after]
    return {"values": [_solve(case["algo"], n, *_edges_of(g, sym), 0) for g in graphs], "missing": 0, "invalid": 0}
