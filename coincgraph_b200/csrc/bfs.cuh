// bfs.cuh - BFS queries: waves of up to 64 sources as bitmasks, and the
// single-source form as bitmaps.
//
// Both are level-synchronous persistent kernels that switch direction
// (Beamer, Asanovic and Patterson, "Direction-optimizing breadth-first
// search", SC 2012): small frontiers are queues whose out-rows are expanded
// (top-down), large ones are masks that every incomplete vertex gathers over
// its in-row (bottom-up).  A wave keeps per vertex the 64-bit mask of sources
// that reached it and of those that did so in the last round (MS-BFS: Then et
// al., "The More the Merrier: Efficient Multi-Source Graph Traversal", VLDB
// 2014).
//
// Depths of a wave below 16 are kept bit-sliced: plane p of vertex v holds, for
// every source, bit p of its depth, so recording a level for any number of
// sources is one OR per set bit of the level, and the k x n result is written
// once, in rows, from four planes (depths stay below 16 on R-MAT).  A word per
// vertex and source instead took a 4 n k byte fill, scattered 4-byte stores and
// a transpose that read it all again.  Deeper levels, on graphs whose rounds
// carry few sources per vertex, go straight to the result, one word per source,
// and a fifth plane marks them (in further planes a vertex took an OR for every
// set bit of a depth of up to twelve bits).
#pragma once

#include "common.cuh"
#include "expand.cuh"
#include "traverse.cuh"

namespace cig {

constexpr uint32_t kMsWidth = 64;
constexpr int kTpbMs = 256;
constexpr uint32_t kBfsPlanes = 4;      // depth bits of the planes; plane kBfsPlanes marks deeper levels
constexpr uint32_t kBfsDeep = 1u << kBfsPlanes;
constexpr uint32_t kBfsChunk = 1024;     // in-rows of at least this many entries are gathered by several warps
constexpr uint32_t kBfsWarpRow = 256;    // ... of at least this many by a warp, shorter ones by eight lanes

struct MsFrontier {
    uint32_t *q0;
    uint32_t *q1;
    uint32_t *cnt;                // 3 round counters, as for the push closure
    unsigned long long *mask0;    // source masks read in even rounds
    unsigned long long *mask1;    // ... in odd rounds
    uint32_t cap;
};

// Bottom-up rounds: when the frontier holds more than `on` vertices (or, once
// bottom-up, more than `off`), or when its out-rows hold more than `edges_on`
// entries: a few hub vertices are a small frontier whose expansion costs as
// much as the whole graph's (on R-MAT the round after the hubs; a top-down
// edge costs an atomic or two, a bottom-up entry a load).  The chunks of long in-rows (`tasks`, listed
// at the first bottom-up round) are gathered by warps of their own into
// `acc`; the last to arrive completes the vertex.
struct BfsPull {
    AdjView rev;  // in-edges (desc null: no bottom-up)
    uint32_t on, off;
    uint32_t edges_on;
    BigRow *tasks;              // off, len, x = vertex, payload = chunks of the row << 32 | row's place in acc
    uint32_t task_cap;
    unsigned long long *acc;    // cleared with the list, left zero by each round
    uint32_t *arrived;          // cleared with the list, left zero by each round
    uint32_t *bigbits;          // bit v: v's in-row is in `tasks`
    uint32_t *ctl;              // BfsCtl, zero at launch
};
enum BfsCtl : int {
    kBfsTasks = 0,
    kBfsBigRows = 1,
    kBfsFill = 2,
    kBfsRounds = 3,
    kBfsEdges = 4,  // 3 counters
    kBfsGoOn = 7    // bits 0: deep rounds follow, 1: bottom-up, 2: tasks listed
};

// Top-down edge of a wave: the bits that have not reached y do so now.
struct MsBfsOp {
    unsigned long long *visit;
    unsigned long long *mask_out;
    WarpBuf buf;

    __device__ __forceinline__ unsigned long long peek(uint32_t y) const { return __ldcg(visit + y); }
    __device__ __forceinline__ bool edge_peeked(bool valid, uint32_t, unsigned long long m, uint32_t y,
                                                unsigned long long seen) const {
        bool want = false, hit = false;
        const unsigned long long cand = m & ~seen;
        if (valid && cand) {
            const unsigned long long nb = cand & ~atomicOr(visit + y, cand);
            if (nb) {
                hit = true;
                want = atomicOr(mask_out + y, nb) == 0ull;
            }
        }
        buf.add(want, y);
        return hit;
    }
    __device__ __forceinline__ bool edge(bool valid, uint32_t x, unsigned long long m, uint32_t y) const {
        return edge_peeked(valid, x, m, y, valid ? peek(y) : 0ull);
    }
};

// Where a wave's depths go.  DEEP: levels of kBfsDeep and more, whose rounds run
// in a kernel of their own (in one kernel with the others the deep part took
// registers from those: 3 to 8 % on R-MAT).
template <bool DEEP>
struct BfsDepths {
    unsigned long long *planes;
    uint32_t *out;  // source-major result
    uint32_t n;

    __device__ __forceinline__ void deep(uint32_t v, uint32_t level, unsigned long long m) const {
        red_or(planes + static_cast<uint64_t>(kBfsPlanes) * n + v, m);
        for (unsigned long long b = m; b; b &= b - 1)
            out[static_cast<uint64_t>(__ffsll(static_cast<long long>(b)) - 1) * n + v] = level;
    }
    // Depth `level` for the sources in m at vertex v (one thread per vertex), as
    // ORs without a result: each waits for nothing, where a load, an OR and a
    // store per set bit of the level followed one another.
    __device__ __forceinline__ void put(uint32_t v, uint32_t level, unsigned long long m) const {
        if (DEEP && level >= kBfsDeep) {
            deep(v, level, m);
            return;
        }
        for (uint32_t b = level; b; b &= b - 1)
            red_or(planes + static_cast<uint64_t>(__ffs(static_cast<int>(b)) - 1) * n + v, m);
    }
    // The same where a warp's vertices follow one another (bottom-up rounds):
    // the loads and stores of the warp are whole lines.
    __device__ __forceinline__ void record(uint32_t v, uint32_t level, unsigned long long m) const {
        if (DEEP && level >= kBfsDeep) {
            deep(v, level, m);
            return;
        }
        for (uint32_t b = level; b; b &= b - 1)
            planes[static_cast<uint64_t>(__ffs(static_cast<int>(b)) - 1) * n + v] |= m;
    }
};

// Warp-wide OR.
__device__ __forceinline__ unsigned long long warp_or(unsigned long long x) {
    const uint32_t lo = __reduce_or_sync(kFull, static_cast<uint32_t>(x));
    const uint32_t hi = __reduce_or_sync(kFull, static_cast<uint32_t>(x >> 32));
    return (static_cast<unsigned long long>(hi) << 32) | lo;
}

// OR of get(y) over the entries of a row (device-only arena), by one warp,
// 256 entries per step, until it covers `missing`; *read counts the entries.
template <class G>
__device__ __forceinline__ unsigned long long warp_gather(const AdjView &rev, const uint32_t *rp, uint32_t len,
                                                          unsigned long long missing, const G &get, uint32_t *read) {
    const uint32_t lane = lane_id();
    unsigned long long acc = 0;
    for (uint32_t b0 = 0; b0 < len; b0 += 256u) {
        uint4 q[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t k = b0 + 128u * h + 4u * lane;
            q[h] = k < len ? __ldg(reinterpret_cast<const uint4 *>(rp + k)) : make_uint4(kTomb, kTomb, kTomb, kTomb);
        }
        unsigned long long m[8];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t k = b0 + 128u * h + 4u * lane;
            const uint32_t y[4] = {rev.vid(q[h].x), rev.vid(q[h].y), rev.vid(q[h].z), rev.vid(q[h].w)};
#pragma unroll
            for (int j = 0; j < 4; ++j) m[4 * h + j] = k + j < len && y[j] != kTomb ? get(y[j]) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) acc |= m[j];
        *read += lane == 0 ? min(256u, len - b0) : 0u;
        acc = warp_or(acc);
        if ((acc & missing) == missing) break;
    }
    return acc;
}

// OR of get(y) over the first kBfsHead entries of the lane's own row, in
// flight together.
constexpr uint32_t kBfsHead = 8;
template <class G>
__device__ __forceinline__ unsigned long long lane_gather(const AdjView &rev, const uint32_t *rp, uint32_t len,
                                                          const G &get) {
    uint4 q[kBfsHead / 4];
#pragma unroll
    for (uint32_t h = 0; h < kBfsHead / 4; ++h)
        q[h] = 4u * h < len ? __ldg(reinterpret_cast<const uint4 *>(rp + 4u * h))
                            : make_uint4(kTomb, kTomb, kTomb, kTomb);
    unsigned long long acc = 0;
#pragma unroll
    for (uint32_t h = 0; h < kBfsHead / 4; ++h) {
        const uint32_t y[4] = {rev.vid(q[h].x), rev.vid(q[h].y), rev.vid(q[h].z), rev.vid(q[h].w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) acc |= 4u * h + j < len && y[j] != kTomb ? get(y[j]) : 0ull;
    }
    return acc;
}

// The rows of the lanes in `mask`, from entry kBfsHead on: eight lanes per
// row, four rows at a time, 32 entries of each per step (a row per lane left
// the warp waiting for its longest row, a row per warp for one chain of loads
// after another).  ORs into the owners' `acc` until it covers `missing`.
template <class G>
__device__ __forceinline__ void groups_gather(const AdjView &rev, uint32_t mask, const RowDesc &d,
                                              unsigned long long missing, const G &get, unsigned long long &acc,
                                              uint32_t &read) {
    const uint32_t lane = lane_id(), sub = lane & 7u;
    while (mask) {  // warp-uniform
        uint32_t m = mask;
        for (uint32_t k = 0; k < (lane >> 3); ++k) m &= m - 1;
        const bool on = m != 0;
        const uint32_t src = on ? __ffs(m) - 1 : 0u;
        const uint64_t off = __shfl_sync(kFull, static_cast<unsigned long long>(d.off), src);
        const uint32_t len = __shfl_sync(kFull, d.len, src);
        const unsigned long long want = __shfl_sync(kFull, missing, src);
        unsigned long long a = __shfl_sync(kFull, acc, src);
        const uint32_t *rp = rev.at(on ? off : 0ull);
        uint32_t k = kBfsHead;
        bool more = on && k < len;
        while (__any_sync(kFull, more)) {
            unsigned long long got = 0;
            if (more) {
                const uint32_t kk = k + 4u * sub;
                const uint4 q = kk < len ? __ldg(reinterpret_cast<const uint4 *>(rp + kk))
                                         : make_uint4(kTomb, kTomb, kTomb, kTomb);
                const uint32_t y[4] = {rev.vid(q.x), rev.vid(q.y), rev.vid(q.z), rev.vid(q.w)};
#pragma unroll
                for (int j = 0; j < 4; ++j) got |= kk + j < len && y[j] != kTomb ? get(y[j]) : 0ull;
                k += 32u;
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) got |= __shfl_xor_sync(kFull, got, o);
            a |= got;
            more = on && k < len && (a & want) != want;
        }
        // the owner with rank g among the four takes group g's result
        const uint32_t rank = __popc(mask & lanemask_lt());
        const unsigned long long res = __shfl_sync(kFull, a, (rank & 3u) * 8u);
        const uint32_t end = __shfl_sync(kFull, k, (rank & 3u) * 8u);
        if (((mask >> lane) & 1u) && rank < 4u) {
            acc = res;
            read = min(end, d.len);
        }
        for (int t = 0; t < 4; ++t) mask &= mask - 1;  // 0 stays 0
    }
}

// List the chunks of the long in-rows and mark their vertices.  A row's place
// in `acc` and `arrived` is cleared when it is handed out, once per wave: what
// a wave that ended in an error left there, or what the memory held before,
// must not count as chunks that have arrived.  A grid barrier follows.
__device__ __forceinline__ void bfs_list_tasks(const BfsPull &pl, uint32_t n, Status *st) {
    const uint32_t lane = lane_id();
    const uint32_t rounded = (n + 31u) & ~31u;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < rounded; v += gridDim.x * blockDim.x) {
        uint32_t len = 0;
        uint64_t off = 0;
        if (v < n) {
            const RowDesc d = pl.rev.desc[v];
            len = d.len;
            off = d.off;
        }
        uint32_t bigs = __ballot_sync(kFull, len >= kBfsChunk);
        if (lane == 0) pl.bigbits[v >> 5] = bigs;
        while (bigs) {
            const uint32_t l = __ffs(bigs) - 1;
            bigs &= bigs - 1;
            const uint32_t llen = __shfl_sync(kFull, len, l), lv = __shfl_sync(kFull, v, l);
            const uint64_t loff = __shfl_sync(kFull, static_cast<unsigned long long>(off), l);
            const uint32_t chunks = (llen + kBfsChunk - 1) / kBfsChunk;
            uint32_t at = 0, row = 0;
            if (lane == 0) {
                at = atomicAdd(pl.ctl + kBfsTasks, chunks);
                row = atomicAdd(pl.ctl + kBfsBigRows, 1u);
                pl.acc[row] = 0ull;
                pl.arrived[row] = 0u;
                if (at + chunks > pl.task_cap) set_error(st, kErrQueue, at);
            }
            at = __shfl_sync(kFull, at, 0);
            row = __shfl_sync(kFull, row, 0);
            for (uint32_t i = lane; i < chunks; i += 32u)
                if (at + i < pl.task_cap)
                    pl.tasks[at + i] = BigRow{loff + static_cast<uint64_t>(i) * kBfsChunk,
                                              (static_cast<unsigned long long>(chunks) << 32) | row, lv,
                                              min(kBfsChunk, llen - i * kBfsChunk)};
        }
    }
}

// Add the block's new frontier vertices to the round's counter: one atomic
// per block (one per warp queued thousands on one address).  All threads call.
__device__ __forceinline__ void block_add(uint32_t *counter, uint32_t mine, uint32_t *shared) {
    mine = __reduce_add_sync(kFull, mine);
    if (threadIdx.x == 0) *shared = 0;
    __syncthreads();
    if (lane_id() == 0 && mine) atomicAdd(shared, mine);
    __syncthreads();
    if (threadIdx.x == 0 && *shared) atomicAdd(counter, *shared);
}

// Does a top-down round over the queue hold more than pl.edges_on row
// entries?  Looked at for queues of kBfsCount vertices and more (below, a
// round is short anyway).  The sum is made while the vertices are queued
// (WarpBuf), so that the round's own barrier covers it: a counting pass with a
// barrier of its own in every round cost a fifth to two fifths on graphs of
// many short rounds (a 511 x 511 grid, 678 to 841 rounds: one source 6.0 ->
// 7.4 ms, two 7.6 -> 10.7 ms), where no round can pass the limit.
// `edges`: the sum, read together with the round's vertex count.
constexpr uint32_t kBfsCount = 256;
__device__ __forceinline__ bool bfs_many_edges(const BfsPull &pl, uint32_t n_in, uint32_t edges) {
    return pl.rev.desc && n_in >= kBfsCount && edges > pl.edges_on;
}

// Bottom-up round of a wave: every vertex that misses source bits ORs the
// frontier masks of its in-neighbours, stopping once nothing is missing.
// Every in-row's first entries are gathered by its own lane, the rest of rows
// below kBfsWarpRow by eight lanes, below kBfsChunk by a warp, longer ones by a
// warp per chunk.  Bound by the gathers: 8 bytes of a 32-byte L2 sector per
// entry.  Returns the new frontier vertices found by this thread.
template <class D>
__device__ __forceinline__ uint32_t bfs_bottom_up(const BfsPull &pl, uint32_t n, unsigned long long full,
                                                  unsigned long long *visit, const D &depths,
                                                  const unsigned long long *m_in, unsigned long long *m_out,
                                                  uint32_t level, ExpandCounters &cnt, unsigned long long &src_edges) {
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    auto get = [&](uint32_t u) { return m_in[u]; };
    uint32_t found = 0;
    const uint32_t nt = min(ld_volatile(pl.ctl + kBfsTasks), pl.task_cap);
    for (uint32_t i = wid; i < nt; i += warps) {
        const BigRow t = pl.tasks[i];
        const unsigned long long vis = __ldcg(visit + t.x), missing = full & ~vis;
        const uint32_t row = static_cast<uint32_t>(t.payload), chunks = static_cast<uint32_t>(t.payload >> 32);
        uint32_t read = 0;
        const unsigned long long acc =
            missing ? warp_gather(pl.rev, pl.rev.at(t.off), t.deg, missing, get, &read) & missing : 0ull;
        if (lane == 0) {
            cnt.edges += read;
            cnt.edges_cached += read;
            cnt.rows += read ? 1u : 0u;
            src_edges += static_cast<unsigned long long>(__popcll(missing)) * read;
            if (acc) atomicOr(pl.acc + row, acc);
            __threadfence();
            if (atomicAdd(pl.arrived + row, 1u) == chunks - 1u) {
                __threadfence();
                const unsigned long long nb = atomicExch(pl.acc + row, 0ull);
                pl.arrived[row] = 0u;
                m_out[t.x] = nb;
                if (nb) {
                    visit[t.x] = vis | nb;
                    depths.record(t.x, level, nb);
                    ++found;
                    ++cnt.hits;
                }
            }
        }
    }
    // The next tile's masks and descriptors are read while this one's rows are
    // gathered.
    const uint32_t words = (n + 31u) / 32u;
    bool mine_next = false;
    unsigned long long vis_next = full;
    RowDesc d_next{0, 0, 0};
    auto look = [&](uint32_t w) {
        const uint32_t v = 32u * w + lane;
        mine_next = w < words && v < n && !((pl.bigbits[w] >> lane) & 1u);
        vis_next = mine_next ? __ldcg(visit + v) : full;
        d_next = mine_next ? pl.rev.desc[v] : RowDesc{0, 0, 0};
    };
    look(wid);
    for (uint32_t w = wid; w < words; w += warps) {
        const uint32_t v = 32u * w + lane;
        const bool mine = mine_next;
        const unsigned long long vis = vis_next;
        const unsigned long long missing = full & ~vis;
        unsigned long long acc = 0;
        RowDesc d = d_next;
        look(w + warps < words ? w + warps : words);
        if (!missing) d.len = 0;
        uint32_t read = 0;
        if (d.len) {
            acc = lane_gather(pl.rev, pl.rev.at(d.off), d.len, get);
            read = min(d.len, kBfsHead);
        }
        const bool open = (acc & missing) != missing;
        groups_gather(pl.rev, __ballot_sync(kFull, open && d.len > kBfsHead && d.len < kBfsWarpRow), d, missing, get,
                      acc, read);
        uint32_t meds = __ballot_sync(kFull, open && d.len >= kBfsWarpRow);
        while (meds) {
            const uint32_t l = __ffs(meds) - 1;
            meds &= meds - 1;
            const uint64_t loff = __shfl_sync(kFull, static_cast<unsigned long long>(d.off), l);
            const uint32_t llen = __shfl_sync(kFull, d.len, l);
            const unsigned long long lm = __shfl_sync(kFull, missing, l);
            uint32_t r = 0;
            const unsigned long long a = warp_gather(pl.rev, pl.rev.at(loff), llen, lm, get, &r);
            r = __shfl_sync(kFull, r, 0);
            if (lane == l) {
                acc = a;
                read = r;
            }
        }
        cnt.edges += read;
        cnt.edges_cached += read;
        cnt.rows += read ? 1u : 0u;
        src_edges += static_cast<unsigned long long>(__popcll(missing)) * read;
        const unsigned long long nb = acc & missing;
        if (mine) m_out[v] = nb;
        if (nb) {
            visit[v] = vis | nb;
            depths.record(v, level, nb);
            ++found;
            ++cnt.hits;
        }
    }
    return found;
}

// The rounds of a wave: those before the first deep level (true: go on to the
// deep ones), or, DEEP, from there on.
struct BfsLoop {
    uint32_t r = 0;
    bool pull = false, listed = false;  // every block takes the same decisions from the same counts
    ExpandCounters cnt;
    unsigned long long src_edges = 0;
};
struct BfsWaveSmem {
    ExpandSmem<kTpbMs, unsigned long long> expand;
    uint32_t fresh;
    uint32_t buf[kTpbMs / 32][kWarpBuf];
    uint32_t held[kTpbMs / 32];
};
template <bool DEEP>
__device__ __forceinline__ bool bfs_rounds(const AdjView &fwd, uint32_t n, unsigned long long full,
                                           unsigned long long *visit, const BfsDepths<DEEP> &depths,
                                           const MsFrontier &fr, const BigList &big, uint32_t max_rounds,
                                           const BfsPull &pl, BfsWaveSmem &ws, BfsLoop &lp, Status *st) {
    auto &sm = ws.expand;
    uint32_t &s_new = ws.fresh;
    auto &s_buf = ws.buf;
    auto &s_held = ws.held;
    ExpandCounters &cnt = lp.cnt;
    unsigned long long &src_edges = lp.src_edges;
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
    uint32_t &r = lp.r;
    bool &pull = lp.pull, &listed = lp.listed;
    bool was_pull = false;
    for (;; ++r) {
        if (!DEEP && r + 1 == kBfsDeep) return true;
        const uint32_t n_in = ld_volatile(fr.cnt + (r % 3));
        const uint32_t n_edges = ld_volatile(pl.ctl + kBfsEdges + r % 3);
        if (n_in == 0) return false;
        if (r >= max_rounds) {
            if (gtid == 0) set_error(st, kErrRounds, r);
            return false;
        }
        if (gtid == 0) {
            fr.cnt[(r + 2) % 3] = 0;
            big.cnt[(r + 2) % 3] = 0;
            pl.ctl[kBfsEdges + (r + 2) % 3] = 0;
        }
        uint32_t *in = (r & 1) ? fr.q1 : fr.q0;
        uint32_t *out = (r & 1) ? fr.q0 : fr.q1;
        uint32_t *out_cnt = fr.cnt + ((r + 1) % 3);
        unsigned long long *m_in = (r & 1) ? fr.mask1 : fr.mask0;
        unsigned long long *m_out = (r & 1) ? fr.mask0 : fr.mask1;
        const uint32_t level = r + 1;
        if (DEEP && level == kBfsDeep) {  // the first deep level
            unsigned long long *mark = depths.planes + static_cast<uint64_t>(kBfsPlanes) * n;
            for (uint32_t v = gtid; v < n; v += gthreads) mark[v] = 0ull;
            if (!grid_barrier(st)) return false;
        }
        was_pull = pull;
        pull = pl.rev.desc && n_in > (was_pull ? pl.off : pl.on);
        if (!was_pull) pull = pull || bfs_many_edges(pl, n_in, n_edges);
        if (pull) {
            if (!was_pull) {
                // The queued vertices are not popped: record their depth here.
                for (uint32_t i = gtid; i < n_in; i += gthreads) {
                    const uint32_t x = __ldcg(in + i);
                    depths.put(x, r, __ldcg(m_in + x));
                }
                if (!listed) bfs_list_tasks(pl, n, st);
                listed = true;
                if (!grid_barrier(st)) return false;
            }
            const uint32_t found =
                bfs_bottom_up(pl, n, full, visit, depths, m_in, m_out, level, cnt, src_edges);
            block_add(out_cnt, found, &s_new);
            if (!grid_barrier(st)) return false;
            continue;
        }
        if (was_pull) {
            // The frontier is the non-zero masks: queue it, and clear the
            // masks of the round before for this one's.
            const uint32_t rounded = (n + 31u) & ~31u;
            for (uint32_t v = gtid; v < rounded; v += gthreads) {
                bool want = false;
                if (v < n) {
                    want = m_in[v] != 0ull;
                    m_out[v] = 0ull;
                }
                warp_enqueue(want, v, in, pl.ctl + kBfsFill, fr.cap, st);
            }
            if (!grid_barrier(st)) return false;
            if (gtid == 0) pl.ctl[kBfsFill] = 0;
        }
        const Defer df{big.rows, big.cnt + (r % 3), big.cap, big.split};
        const MsBfsOp op{visit, m_out,
                         WarpBuf{s_buf[threadIdx.x >> 5], s_held + (threadIdx.x >> 5), out, out_cnt, fr.cap, st,
                                 fwd.desc, pl.ctl + kBfsEdges + (r + 1) % 3}};
        for (uint32_t base = 0; base < n_in; base += gridDim.x * kTpbMs) {
            const uint32_t i = base + spread_rank<kTpbMs>() * gridDim.x + blockIdx.x;
            bool has = i < n_in;
            uint32_t x = 0, deg = 0;
            uint64_t off = 0;
            unsigned long long m = 0;
            if (has) {
                x = __ldcg(in + i);
                // Nobody writes m_in this round: take the bits and clear them.
                m = __ldcg(m_in + x);
                const RowDesc d = fwd.desc[x];
                m_in[x] = 0ull;
                depths.put(x, r, m);
                deg = d.len;
                off = d.off;
                has = m != 0ull && deg > 0;
                if (has) src_edges += static_cast<unsigned long long>(__popcll(m)) * deg;
            }
            expand_rows<kTpbMs>(fwd, has, x, m, off, deg, op, sm, cnt, df);
        }
        op.buf.flush();
        if (!grid_barrier(st)) return false;
        const uint32_t nbig = min(ld_volatile(big.cnt + (r % 3)), big.cap);
        if (nbig) {
            expand_deferred<kTpbMs, unsigned long long>(fwd, big.rows, nbig, op, cnt);
            op.buf.flush();
            if (!grid_barrier(st)) return false;
        }
    }
}

// Counters at the end of a wave's kernel, which began at round `before`.
__device__ __forceinline__ void bfs_wave_end(const BfsPull &pl, const BfsLoop &lp, uint32_t before, Status *st) {
    flush_counters(st, lp.cnt, kCntPush);
    unsigned long long src_edges = lp.src_edges;
    for (int o = 16; o > 0; o >>= 1) src_edges += __shfl_down_sync(kFull, src_edges, o);
    if (lane_id() == 0 && src_edges) atomicAdd(&st->counters[kCntSrcEdges], src_edges);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        pl.ctl[kBfsRounds] = lp.r;
        atomicAdd(&st->counters[kCntRounds], static_cast<unsigned long long>(lp.r - before));
    }
}

// One wave (cooperative launch), up to the deep levels.  Round r gives depth
// r + 1.  `full`: the wave's source bits.  Planes 0..kBfsPlanes-1 are cleared
// before the launch, the mark of deep levels by the round that reaches them.
// PER_SM blocks per SM: rounds of few vertices wait for their barriers, which
// cost with the blocks, long ones for the gathers in flight.  Two, except for
// waves of more than kBfsFew sources and for graphs of many and long rows
// (bfs_blocks in engine.cu).  511 x 511 grid, 2 / 5 / 13 sources: 7.0 / 8.1 /
// 9.9 ms with two blocks, 8.7 / 9.9 / 11.8 with four; R-MAT s16, 1 / 13 / 64
// sources: 0.094 / 0.147 / 0.160 and 0.115 / 0.175 / 0.160; s22, 1 / 13 / 64:
// 0.36 / 1.23 / 1.35 and 0.30 / 0.94 / 1.35.
constexpr uint32_t kBfsFew = 16;
template <int PER_SM>
__global__ void __launch_bounds__(kTpbMs, PER_SM) bfs_wave(AdjView fwd, uint32_t n, unsigned long long full,
                                                           unsigned long long *visit, unsigned long long *planes,
                                                           MsFrontier fr, BigList big, uint32_t max_rounds,
                                                           BfsPull pl, Status *st) {
    __shared__ BfsWaveSmem ws;
    if (threadIdx.x < kTpbMs / 32) ws.held[threadIdx.x] = 0;
    __syncthreads();
    BfsLoop lp;
    const bool more =
        bfs_rounds(fwd, n, full, visit, BfsDepths<false>{planes, nullptr, n}, fr, big, max_rounds, pl, ws, lp, st);
    bfs_wave_end(pl, lp, 0u, st);
    if (more && blockIdx.x == 0 && threadIdx.x == 0)
        pl.ctl[kBfsGoOn] = 1u | (lp.pull ? 2u : 0u) | (lp.listed ? 4u : 0u);
}

// Source-major depths from the planes: out[j * n + v], four vertices per
// thread and 512-byte stores per warp where the rows are 16-byte aligned (n a
// multiple of 4 and an aligned result), one vertex per thread otherwise; one
// pass over `visit` and the planes in use.  Deep entries are there already.
template <int V, bool DEEP>
__device__ __forceinline__ void bfs_depths_of(const unsigned long long *visit, const unsigned long long *planes,
                                              uint32_t n, uint32_t k, uint32_t used, uint32_t v, uint32_t *out) {
    unsigned long long vis[V], p[kBfsPlanes][V], mark[DEEP ? V : 1];
#pragma unroll
    for (int i = 0; i < V; ++i) vis[i] = visit[v + i];
#pragma unroll
    for (uint32_t b = 0; b < kBfsPlanes; ++b)
#pragma unroll
        for (int i = 0; i < V; ++i) p[b][i] = b < used ? planes[static_cast<uint64_t>(b) * n + v + i] : 0ull;
    if constexpr (DEEP)
#pragma unroll
        for (int i = 0; i < V; ++i) mark[i] = planes[static_cast<uint64_t>(kBfsPlanes) * n + v + i];
    for (uint32_t j = 0; j < k; ++j) {
        uint32_t d[V];
        bool there = false;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            d[i] = 0;
#pragma unroll
            for (uint32_t b = 0; b < kBfsPlanes; ++b) d[i] |= (static_cast<uint32_t>(p[b][i] >> j) & 1u) << b;
            if (!((vis[i] >> j) & 1ull)) d[i] = kInf;
            if constexpr (DEEP) there = there || ((mark[i] >> j) & 1ull);
        }
        uint32_t *to = out + static_cast<uint64_t>(j) * n + v;
        if (DEEP && there) {
#pragma unroll
            for (int i = 0; i < V; ++i)
                if (!((mark[DEEP ? i : 0] >> j) & 1ull)) to[i] = d[i];
        } else if constexpr (V == 4) {
            __stcs(reinterpret_cast<uint4 *>(to), make_uint4(d[0], d[1], d[2], d[3]));
        } else {
            __stcs(to, d[0]);
        }
    }
}

template <bool DEEP>
__device__ __forceinline__ void bfs_depths_all(const unsigned long long *visit, const unsigned long long *planes,
                                               uint32_t n, uint32_t k, uint32_t used, uint32_t *out) {
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
    if ((n & 3u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
        for (uint32_t q = gtid; q < n / 4; q += gthreads)
            bfs_depths_of<4, DEEP>(visit, planes, n, k, used, 4 * q, out);
    } else {
        for (uint32_t v = gtid; v < n; v += gthreads) bfs_depths_of<1, DEEP>(visit, planes, n, k, used, v, out);
    }
}

// Waves without deep levels (the others' depths: bfs_wave_deep).
__global__ void bfs_depths(const unsigned long long *visit, const unsigned long long *planes, uint32_t n, uint32_t k,
                           const uint32_t *ctl, uint32_t *out) {
    if (!ctl[kBfsGoOn]) bfs_depths_all<false>(visit, planes, n, k, 32u - __clz(ctl[kBfsRounds]), out);
}

// The rounds from the first deep level on, if bfs_wave left any, and the depths
// of such a wave: few vertices a round, so two blocks per SM (cooperative
// launch).  511 x 511 grid, 64 sources: 11.5 ms with every level in planes,
// 8.9 so; 2048 x 2048: 264 and 214 ms.
__global__ void __launch_bounds__(kTpbMs, 2) bfs_wave_deep(AdjView fwd, uint32_t n, unsigned long long full,
                                                           unsigned long long *visit, unsigned long long *planes,
                                                           uint32_t *out, uint32_t k, MsFrontier fr, BigList big,
                                                           uint32_t max_rounds, BfsPull pl, Status *st) {
    const uint32_t go_on = pl.ctl[kBfsGoOn];
    if (!go_on) return;
    __shared__ BfsWaveSmem ws;
    if (threadIdx.x < kTpbMs / 32) ws.held[threadIdx.x] = 0;
    __syncthreads();
    BfsLoop lp;
    const uint32_t before = lp.r = kBfsDeep - 1;
    lp.pull = go_on & 2u;
    lp.listed = go_on & 4u;
    bfs_rounds(fwd, n, full, visit, BfsDepths<true>{planes, out, n}, fr, big, max_rounds, pl, ws, lp, st);
    bfs_wave_end(pl, lp, before, st);
    // Every block left the rounds after the same barrier.
    bfs_depths_all<true>(visit, planes, n, k, 32u - __clz(lp.r), out);
}

// ---------------------------------------------------------------- one source
// Visited and frontier vertices are bitmaps (n / 8 bytes: they stay in L2 and
// largely in L1, where 8 bytes per vertex do not), depths go straight to the
// result.
struct OneBfsOp {
    uint32_t *vis;
    uint32_t *depth;
    uint32_t level;
    WarpBuf buf;

    __device__ __forceinline__ uint32_t peek(uint32_t y) const { return __ldcg(vis + (y >> 5)); }
    __device__ __forceinline__ bool edge_peeked(bool valid, uint32_t, uint32_t, uint32_t y, uint32_t word) const {
        const uint32_t bit = 1u << (y & 31u);
        bool want = false;
        if (valid && !(word & bit)) want = !(atomicOr(vis + (y >> 5), bit) & bit);
        if (want) depth[y] = level;
        buf.add(want, y);
        return want;
    }
    __device__ __forceinline__ bool edge(bool valid, uint32_t x, uint32_t p, uint32_t y) const {
        return edge_peeked(valid, x, p, y, valid ? peek(y) : 0u);
    }
};

__global__ void bfs_one_seed(const uint32_t *source, uint32_t *depth, uint32_t *vis, uint32_t *q0, uint32_t *cnt) {
    const uint32_t s = source[0];
    depth[s] = 0u;
    vis[s >> 5] = 1u << (s & 31u);
    q0[0] = s;
    cnt[0] = 1u;
}

// Single-source BFS (cooperative launch); `vis` cleared and `depth` filled
// with kInf before it, `bm0` / `bm1` the frontier bitmaps of bottom-up rounds
// ((n + 31) / 32 words each).  PER_SM blocks per SM as for bfs_wave.
template <int PER_SM>
__global__ void __launch_bounds__(kTpbMs, PER_SM) bfs_one(AdjView fwd, uint32_t n, uint32_t *depth, uint32_t *vis,
                                                     uint32_t *bm0, uint32_t *bm1, MsFrontier fr, BigList big,
                                                     uint32_t max_rounds, BfsPull pl, Status *st) {
    __shared__ ExpandSmem<kTpbMs> sm;
    __shared__ uint32_t s_new;
    __shared__ uint32_t s_buf[kTpbMs / 32][kWarpBuf];
    __shared__ uint32_t s_held[kTpbMs / 32];
    if (threadIdx.x < kTpbMs / 32) s_held[threadIdx.x] = 0;
    __syncthreads();
    ExpandCounters cnt;
    bool pull = false, was_pull = false;
    const uint32_t lane = lane_id();
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
    const uint32_t warps = gthreads >> 5, wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t words = (n + 31u) / 32u;
    uint32_t r = 0;
    for (;; ++r) {
        const uint32_t n_in = ld_volatile(fr.cnt + (r % 3));
        const uint32_t n_edges = ld_volatile(pl.ctl + kBfsEdges + r % 3);
        if (n_in == 0) break;
        if (r >= max_rounds) {
            if (gtid == 0) set_error(st, kErrRounds, r);
            break;
        }
        if (gtid == 0) {
            fr.cnt[(r + 2) % 3] = 0;
            big.cnt[(r + 2) % 3] = 0;
            pl.ctl[kBfsEdges + (r + 2) % 3] = 0;
        }
        uint32_t *in = (r & 1) ? fr.q1 : fr.q0;
        uint32_t *out = (r & 1) ? fr.q0 : fr.q1;
        uint32_t *out_cnt = fr.cnt + ((r + 1) % 3);
        uint32_t *cur = (r & 1) ? bm1 : bm0;
        uint32_t *next = (r & 1) ? bm0 : bm1;
        was_pull = pull;
        pull = pl.rev.desc && n_in > (was_pull ? pl.off : pl.on);
        if (!was_pull) pull = pull || bfs_many_edges(pl, n_in, n_edges);
        if (pull) {
            if (!was_pull) {  // the queue as a bitmap
                for (uint32_t w = gtid; w < words; w += gthreads) cur[w] = 0u;
                if (!grid_barrier(st)) break;
                for (uint32_t i = gtid; i < n_in; i += gthreads) {
                    const uint32_t x = __ldcg(in + i);
                    atomicOr(cur + (x >> 5), 1u << (x & 31u));
                }
                if (!grid_barrier(st)) break;
            }
            auto get = [&](uint32_t u) { return static_cast<unsigned long long>((cur[u >> 5] >> (u & 31u)) & 1u); };
            uint32_t found = 0;
            // The next words' vertices and descriptors are read while this
            // one's rows are looked through.
            uint32_t seen_next = 0xFFFFFFFFu;
            RowDesc d_next{0, 0, 0};
            auto look = [&](uint32_t w) {
                seen_next = 0xFFFFFFFFu;
                if (w < words) seen_next = __ldcg(vis + w);
                const bool open = w < words && 32u * w + lane < n && !((seen_next >> lane) & 1u);
                d_next = open ? pl.rev.desc[32u * w + lane] : RowDesc{0, 0, 0};
            };
            look(wid);
            for (uint32_t w = wid; w < words; w += warps) {
                const uint32_t seen = seen_next;
                const uint32_t v = 32u * w + lane;
                const RowDesc d = d_next;
                look(w + warps < words ? w + warps : words);
                uint32_t read = 0;
                unsigned long long hit = 0;
                // Most vertices that have a parent in the frontier find one
                // among the first entries.
                if (d.len) {
                    hit = lane_gather(pl.rev, pl.rev.at(d.off), d.len, get);
                    read = min(d.len, kBfsHead);
                }
                const bool open = !hit;
                groups_gather(pl.rev, __ballot_sync(kFull, open && d.len > kBfsHead && d.len < kBfsWarpRow), d, 1ull,
                              get, hit, read);
                uint32_t rest = __ballot_sync(kFull, open && d.len >= kBfsWarpRow);
                while (rest) {
                    const uint32_t l = __ffs(rest) - 1;
                    rest &= rest - 1;
                    const uint64_t loff = __shfl_sync(kFull, static_cast<unsigned long long>(d.off), l);
                    const uint32_t llen = __shfl_sync(kFull, d.len, l);
                    uint32_t rd = 0;
                    const unsigned long long a = warp_gather(pl.rev, pl.rev.at(loff), llen, 1ull, get, &rd);
                    rd = __shfl_sync(kFull, rd, 0);
                    if (lane == l) {
                        hit = a;
                        read += rd;
                    }
                }
                cnt.edges += read;
                cnt.edges_cached += read;
                cnt.rows += read ? 1u : 0u;
                if (hit) {
                    depth[v] = r + 1;
                    ++cnt.hits;
                    ++found;
                }
                const uint32_t nb = __ballot_sync(kFull, hit != 0ull);
                if (lane == 0) {
                    next[w] = nb;
                    if (nb) vis[w] = seen | nb;
                }
            }
            block_add(out_cnt, found, &s_new);
            if (!grid_barrier(st)) break;
            continue;
        }
        if (was_pull) {  // the bitmap as a queue
            for (uint32_t w = wid; w < words; w += warps) {
                const uint32_t bits = cur[w];
                warp_enqueue((bits >> lane) & 1u, 32u * w + lane, in, pl.ctl + kBfsFill, fr.cap, st);
            }
            if (!grid_barrier(st)) break;
            if (gtid == 0) pl.ctl[kBfsFill] = 0;
        }
        const Defer df{big.rows, big.cnt + (r % 3), big.cap, big.split};
        const OneBfsOp op{vis, depth, r + 1,
                          WarpBuf{s_buf[threadIdx.x >> 5], s_held + (threadIdx.x >> 5), out, out_cnt, fr.cap, st,
                                  fwd.desc, pl.ctl + kBfsEdges + (r + 1) % 3}};
        for (uint32_t base = 0; base < n_in; base += gridDim.x * kTpbMs) {
            const uint32_t i = base + spread_rank<kTpbMs>() * gridDim.x + blockIdx.x;
            bool has = i < n_in;
            uint32_t x = 0, deg = 0;
            uint64_t off = 0;
            if (has) {
                x = __ldcg(in + i);
                const RowDesc d = fwd.desc[x];
                deg = d.len;
                off = d.off;
                has = deg > 0;
            }
            expand_rows<kTpbMs>(fwd, has, x, 0u, off, deg, op, sm, cnt, df);
        }
        op.buf.flush();
        if (!grid_barrier(st)) break;
        const uint32_t nbig = min(ld_volatile(big.cnt + (r % 3)), big.cap);
        if (nbig) {
            expand_deferred<kTpbMs>(fwd, big.rows, nbig, op, cnt);
            op.buf.flush();
            if (!grid_barrier(st)) break;
        }
    }
    flush_counters(st, cnt, kCntPush);
    const uint32_t edges = __reduce_add_sync(kFull, cnt.edges);  // one source: source edges = edges
    if (lane == 0 && edges) atomicAdd(&st->counters[kCntSrcEdges], static_cast<unsigned long long>(edges));
    if (gtid == 0) atomicAdd(&st->counters[kCntRounds], static_cast<unsigned long long>(r));
}

}  // namespace cig
