"""Shared test inputs: seeded R-MAT cases and hand-built adversarial cases.

The adversarial cases cover what the reference's chunk store and repair
paths handle (source_local_chunk_store.h:670-848 and the samples' deletion
rules): parallel edges and deleting one copy, repeated deletion requests,
missing deletes, out-of-range ids, self-loops, empty batches, deleting the
parent edge with and without a tight alternative, rows that outgrow their
block several times, and rows large enough for the block-wide paths
(> 4096 entries) and for multi-segment blocks (> 16384 entries).
"""
from __future__ import annotations

from dataclasses import dataclass, field

import numpy as np

from coincgraph_b200 import gen


@dataclass
class Case:
    name: str
    n: int
    xadj: np.ndarray
    adj: np.ndarray
    batches: list = field(default_factory=list)  # (du, dv, au, av) uint32 arrays
    source: int = 0


def _csr_from_edges(n, src, dst):
    g = gen.graph_from_edges(n, src, dst)
    return g.xadj, g.adj


def rmat_case(scale: int, batches: int, dels: int, adds: int, seed_offset: int = 0, symmetric=False) -> Case:
    g, h = gen.rmat(scale, keep_handle=True, symmetric=symmetric)
    ups = gen.updates(h, [dels] * batches, [adds] * batches, seed=gen.UPDATE_SEED_BASE + 100 + seed_offset,
                      symmetric=symmetric)
    return Case(f"rmat{scale}", g.n, g.xadj, g.adj, [ups.batch(i) for i in range(batches)], source=0)


def _u32(x):
    return np.asarray(x, dtype=np.uint32)


def adversarial_case() -> Case:
    rng = np.random.default_rng(20240611)
    n = 64
    src, dst = [], []
    # a path with a tight alternative and a weak one
    for a, b in [(0, 1), (1, 2), (2, 3), (3, 4), (0, 5), (5, 2), (0, 6), (6, 3), (4, 7), (7, 8)]:
        src.append(a)
        dst.append(b)
    # parallel edges
    for _ in range(3):
        src.append(0)
        dst.append(9)
    src += [9, 9, 10, 11, 12, 12]
    dst += [10, 10, 11, 12, 13, 13]
    # self loops
    src += [13, 14]
    dst += [13, 14]
    # equal-label cycle for CC (20 -> 21 -> 22 -> 20, fed from 15)
    src += [15, 20, 21, 22]
    dst += [20, 21, 22, 20]
    # random filler
    for _ in range(200):
        a, b = rng.integers(0, n, 2)
        src.append(int(a))
        dst.append(int(b))
    xadj, adj = _csr_from_edges(n, src, dst)
    batches = [
        # delete one copy of a parallel edge, a missing edge and an out-of-range id
        (_u32([0, 40, 70]), _u32([9, 41, 1]), _u32([]), _u32([])),
        # empty batch
        (_u32([]), _u32([]), _u32([]), _u32([])),
        # delete the tree path and the parent edge of 2, repeated requests
        (_u32([1, 1, 0, 9, 9, 9]), _u32([2, 2, 1, 10, 10, 10]), _u32([30, 31, 32, 99]), _u32([31, 32, 2, 3])),
        # break the equal-label cycle feed, re-add parallel edges, grow row 30 through several classes
        (_u32([15, 20]), _u32([20, 21]), _u32([30] * 40 + [0, 0]), _u32(list(range(1, 41)) + [9, 9])),
        # insert only
        (_u32([]), _u32([]), _u32([4, 8, 63]), _u32([63, 0, 1])),
    ]
    return Case("adversarial", n, xadj, adj, batches, source=0)


def big_row_case() -> Case:
    """Rows above the warp path (5000 entries) and above one segment (20000)."""
    rng = np.random.default_rng(7)
    n = 30000
    # vertex 5 has 6000 in-edges and its parent edge (0, 5) is deleted in
    # batch 0, so the pull repair meets an in-row above the split threshold
    src = np.concatenate([np.zeros(20000, np.int64), np.ones(5000, np.int64), rng.integers(0, n, 30000),
                          np.arange(100, 6100), [0]])
    dst = np.concatenate([rng.integers(6, n, 20000), rng.integers(2, n, 5000), rng.integers(0, n, 30000),
                          np.full(6000, 5), [5]])
    xadj, adj = _csr_from_edges(n, src, dst)
    row0 = adj[int(xadj[0]):int(xadj[1])]
    row1 = adj[int(xadj[1]):int(xadj[2])]
    batches = []
    for k in range(3):
        pick0 = row0[rng.integers(0, len(row0), 50)]
        pick1 = row1[rng.integers(0, len(row1), 20)]
        extra = 1 if k == 0 else 0
        du = np.concatenate([np.zeros(50, np.uint32), np.ones(20, np.uint32), rng.integers(0, n, 30).astype(np.uint32),
                             np.zeros(extra, np.uint32)])
        dv = np.concatenate([pick0, pick1, rng.integers(0, n, 30), np.full(extra, 5)]).astype(np.uint32)
        # batch 1 pushes row 0 past its 32768-slot block and row 1 past 8192
        au = np.concatenate([np.zeros(13000 * (k == 1), np.uint32), np.ones(4000 * (k == 1), np.uint32),
                             rng.integers(0, n, 100).astype(np.uint32)])
        av = rng.integers(0, n, len(au)).astype(np.uint32)
        batches.append((du, dv, au, av))
    return Case("bigrow", n, xadj, adj, batches, source=0)


def heavy_delete_case() -> Case:
    """Many deletion keys in one row: a 3000-entry row losing 200 entries
    (more than a warp's 32 key registers) and a 12000-entry row losing 3000
    (more than the block path's 2048 shared-memory keys), with parallel edges
    and repeated requests."""
    rng = np.random.default_rng(11)
    n = 9000
    src = np.concatenate([np.full(3000, 0), np.full(12000, 1), rng.integers(0, n, 20000)])
    dst = np.concatenate([rng.integers(2, 400, 3000), rng.integers(2, n, 12000), rng.integers(0, n, 20000)])
    xadj, adj = _csr_from_edges(n, src, dst)
    row0 = adj[int(xadj[0]):int(xadj[1])]
    row1 = adj[int(xadj[1]):int(xadj[2])]
    batches = []
    for k in range(2):
        d0 = row0[rng.integers(0, len(row0), 200)]
        d1 = row1[rng.integers(0, len(row1), 3000)]
        du = np.concatenate([np.zeros(200, np.uint32), np.ones(3000, np.uint32)])
        dv = np.concatenate([d0, d1]).astype(np.uint32)
        au = rng.integers(0, n, 500).astype(np.uint32)
        av = rng.integers(0, n, 500).astype(np.uint32)
        batches.append((du, dv, au, av))
    return Case("heavydelete", n, xadj, adj, batches, source=0)


def full_row_case() -> Case:
    """Rows at and beside the block sizes and worker limits (lane 8, warp 1024
    and 4096, segment 16384) that overflow while they hold tombstones: batch 0
    appends as many entries as it deletes (a full row compacts in place),
    batch 1 outgrows the block (the row moves, tombstones and all where they
    fit), batch 2 repeats batch 0 on the moved rows; some entries are parallel
    edges whose first occurrence goes."""
    rng = np.random.default_rng(23)
    n = 40000
    sizes = [2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 2048, 4095, 4096, 4097,
             16384, 16385]
    rows = [list(rng.integers(0, max(64, 2 * k), k) % n) for k in sizes]
    src = np.repeat(np.arange(len(sizes)), sizes)
    xadj, adj = _csr_from_edges(n, src, np.concatenate(rows))
    batches = []
    for k in range(3):
        du, dv, au, av = [], [], [], []
        for u, row in enumerate(rows):
            gone = max(1, len(row) // 16)
            come = gone + (len(row) if k == 1 and u % 2 else 1 if k == 1 else 0)
            for i in sorted(rng.choice(len(row), gone, replace=False), reverse=True):
                du.append(u)
                dv.append(row[i])
                row.remove(row[i])  # the first occurrence goes
            new = list(rng.integers(0, n, come))
            au += [u] * come
            av += new
            row += new
        batches.append((_u32(du), _u32(dv), _u32(au), _u32(av)))
    return Case("fullrow", n, xadj, adj, batches, source=0)


def grown_row_case() -> Case:
    """Rows that are short when the position index is built and grow past the
    longest row one warp serves (4096): 0 to 40,000 entries (several
    segments), 1 to 6,000, some of them parallel edges; vertex 2's in-row to
    20,000.  Then deletions of a few, many and missing entries, repeated
    requests, and enough for a compaction; the rows go on growing between."""
    rng = np.random.default_rng(53)
    n = 45000
    src = np.concatenate([[0, 0, 1, 1], rng.integers(0, n, 3000)])
    dst = np.concatenate([[5, 6, 7, 8], rng.integers(0, n, 3000)])
    xadj, adj = _csr_from_edges(n, src, dst)
    row0 = list(rng.permutation(np.arange(10, n))[:40000])
    row1 = list(rng.integers(10, 5000, 6000))
    in2 = list(rng.permutation(np.arange(10, n))[:20000])

    def take(row, k):
        got = [row.pop(i) for i in sorted(rng.choice(len(row), k, replace=False), reverse=True)]
        return got

    def batch(d0, d1, d2, a0, a1, extra=()):
        du = [0] * len(d0) + [1] * len(d1) + list(d2) + [e[0] for e in extra]
        dv = list(d0) + list(d1) + [2] * len(d2) + [e[1] for e in extra]
        order = rng.permutation(len(du))
        return (_u32(du)[order], _u32(dv)[order], _u32([0] * len(a0) + [1] * len(a1)), _u32(list(a0) + list(a1)))

    batches = [(_u32([]), _u32([]), _u32([0] * 40000 + [1] * 6000 + in2),
                _u32(row0 + row1 + [2] * 20000))]
    # few keys per row, two of them missing; a lane's worth, 32 and 300 of them
    batches.append(batch(take(row0, 3), [row1[0]], take(in2, 4), [], [], extra=[(0, 1), (1, 4)]))
    batches.append(batch(take(row0, 32), take(row1, 9), take(in2, 300), [11, 12], [13]))
    # repeated requests on both out-rows, and more keys than a group of shared memory holds
    twice = [row1[3], row1[3], row1[5]]
    batches.append(batch(take(row0, 1) * 2, twice, take(in2, 2500), [], row1[:50]))
    # a quarter and more: compactions
    batches.append(batch(take(row0, 12000), sorted(set(row1))[:1500], take(in2, 6000), row0[:100], []))
    batches.append(batch(take(row0, 5), [], take(in2, 5), [], []))
    return Case("grownrow", n, xadj, adj, batches, source=0)


def recurring_case() -> Case:
    """The same edges deleted and inserted again, batch after batch, some of
    them twice in the row and some requested when they are absent, in an
    indexed row of 300 entries and a short one."""
    rng = np.random.default_rng(31)
    n = 500
    src = np.concatenate([np.zeros(300, np.int64), np.ones(10, np.int64), rng.integers(0, n, 2000)])
    dst = rng.integers(0, n, len(src))
    xadj, adj = _csr_from_edges(n, src, dst)
    u = np.concatenate([np.zeros(40, np.uint32), np.ones(4, np.uint32)])
    v = np.concatenate([adj[:40], adj[300:304]])
    batches = [(u, v, u, v)] * 6 + [(u, v, _u32([]), _u32([])), (u, v, u, v), (u, v, u, v)]
    return Case("recurring", n, xadj, adj, batches, source=0)


def admission_case() -> Case:
    """248 neighbours of the source with rows of 16,384 entries (one 64 KiB
    segment each) or 8,192.  Batch 0 appends to the 48 shorter rows, so that
    each moves to a segment of its own; the batches after it only delete and
    insert edges of the source, whose subtrees then read the long rows
    again: no new segments."""
    rng = np.random.default_rng(41)
    n = 40000
    hubs = np.arange(1, 249)
    sizes = np.where(hubs <= 200, 16384, 8192)
    src = np.concatenate([np.zeros(len(hubs), np.int64), np.repeat(hubs, sizes)])
    dst = np.concatenate([hubs, rng.integers(249, n, int(sizes.sum()))])
    xadj, adj = _csr_from_edges(n, src, dst)
    short = _u32(hubs[200:])
    batches = [(_u32([]), _u32([]), short, _u32(rng.integers(249, n, len(short))))]
    for k in range(3):
        gone = _u32(hubs[60 * k:60 * k + 60])
        back = _u32(hubs[60 * (k - 1):60 * k]) if k else _u32([])
        batches.append((np.zeros_like(gone), gone, np.zeros_like(back), back))
    return Case("admission", n, xadj, adj, batches, source=0)


def grid_case(side: int = 48, batches: int = 3, size: int = 150) -> Case:
    """Road-like high-diameter case: a side x side grid, local insertions."""
    g = gen.grid(side)
    ups = gen.local_updates(g, side, [size] * batches, [size] * batches, seed=gen.UPDATE_SEED_BASE + 300)
    return Case(f"grid{side}", g.n, g.xadj, g.adj, [ups.batch(i) for i in range(batches)], source=0)


ORACLE_MODE = {"bfs": 0, "sssp": 1, "cc": 2, "sssp_u255": 3}


def make_engine(algo: str, **kw):
    """Engine for a test algorithm name; "sssp_u255" is SSSP with the
    uniform [1, 255] edge weights (CIG_FLAG_WEIGHT_U255)."""
    from coincgraph_b200 import Engine
    from coincgraph_b200.engine import FLAG_WEIGHT_U255

    if algo == "sssp_u255":
        return Engine("sssp", flags=kw.pop("flags", 0) | FLAG_WEIGHT_U255, **kw)
    return Engine(algo, **kw)


def oracle_trace(case: Case, algo: str):
    """Replay the case on the oracle: per batch the values after the deletion
    phase and after the batch, and the rows after the batch."""
    import oracle

    g = oracle.Graph(case.n, case.xadj, case.adj)
    mode = ORACLE_MODE.get(algo)

    def values():
        if algo == "cc":
            return g.cc()
        return g.sssp(case.source, mode)

    out = {"init": values(), "delete": [], "batch": [], "rows": []}
    for du, dv, au, av in case.batches:
        g.delete(du, dv)
        out["delete"].append(values())
        g.add(au, av)
        out["batch"].append(values())
        out["rows"].append(g.export())
    return out, g
