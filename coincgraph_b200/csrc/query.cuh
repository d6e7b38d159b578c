// query.cuh - multi-source SSSP with 64-wide bitmask frontiers, and the
// output side of the query waves (BFS: bfs.cuh).
//
// One wave serves up to 64 sources.  Per vertex the wave keeps a 64-bit mask
// of the sources whose value at that vertex changed in the last round, so a
// row is read once per round for all of those sources (the "MS-BFS" idea of
// Then et al., "The More the Merrier: Efficient Multi-Source Graph
// Traversal", VLDB 2014, applied to label-correcting SSSP).  Values
// are stored vertex-major, 4 to 64 words per vertex (the wave's sources padded
// to a power of two), so the sources of one vertex share cache lines; a
// transpose kernel writes the k x n source-major result.
//
// The reference answers one source per engine run (BFS/SSSP Start,
// include/framework/framework.cuh:1151-1182); these queries give the same
// depths and distances (the values are unique) for many sources at once,
// over the same adjacency (cache or zero-copy rows) and edge weights.
#pragma once

#include "bfs.cuh"
#include "common.cuh"
#include "expand.cuh"
#include "traverse.cuh"

namespace cig {

// One source (a wave of one: one word per vertex, the result itself).
template <int A>
struct MsRelaxOp {
    uint32_t *dist;
    unsigned long long *mask_out;
    uint32_t *q_out;
    uint32_t *q_count;
    uint32_t q_cap;
    Status *st;

    __device__ __forceinline__ uint32_t peek(uint32_t y) const { return __ldcg(dist + y); }
    __device__ __forceinline__ bool edge_peeked(bool valid, uint32_t x, uint32_t dx, uint32_t y, uint32_t dy) const {
        const uint32_t nd = dx + edge_weight<A>(x, y);
        const bool improved = valid && nd < dy && nd < atomicMin(dist + y, nd);
        const bool want = improved && atomicOr(mask_out + y, 1ull) == 0ull;
        warp_enqueue(want, y, q_out, q_count, q_cap, st);
        return improved;
    }
    __device__ __forceinline__ bool edge(bool valid, uint32_t x, uint32_t dx, uint32_t y) const {
        return edge_peeked(valid, x, dx, y, valid ? peek(y) : 0u);
    }
};

// Seeds of one wave: source j of the wave gets bit j, value 0 (`dist`: SSSP)
// or its visited bit (`visit`: BFS), and its vertex is queued once (several
// bits may share a vertex).
__global__ void ms_seed(const uint32_t *sources, uint32_t k, uint32_t *dist, uint32_t width,
                        unsigned long long *visit, MsFrontier fr, Status *st) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= k) return;
    const uint32_t s = sources[j];
    if (dist) dist[static_cast<uint64_t>(s) * width + j] = 0u;
    if (visit) atomicOr(visit + s, 1ull << j);
    if (atomicOr(fr.mask0 + s, 1ull << j) == 0ull) {
        const uint32_t pos = atomicAdd(fr.cnt + 0, 1u);
        if (pos < fr.cap)
            fr.q0[pos] = s;
        else
            set_error(st, kErrQueue, pos);
    }
}

// Single-source closure (cooperative launch): round r expands the vertices
// queued in round r-1.
template <int A>
__global__ void __launch_bounds__(kTpbMs, 4) ms_closure(AdjView fwd, uint32_t *dist, MsFrontier fr, BigList big,
                                                        uint32_t max_rounds, Status *st) {
    __shared__ ExpandSmem<kTpbMs> sm;
    ExpandCounters cnt;
    uint32_t r = 0;
    for (;; ++r) {
        const uint32_t n_in = ld_volatile(fr.cnt + (r % 3));
        if (n_in == 0) break;
        if (r >= max_rounds) {
            if (blockIdx.x == 0 && threadIdx.x == 0) set_error(st, kErrRounds, r);
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fr.cnt[(r + 2) % 3] = 0;
            big.cnt[(r + 2) % 3] = 0;
        }
        const uint32_t *in = (r & 1) ? fr.q1 : fr.q0;
        uint32_t *out = (r & 1) ? fr.q0 : fr.q1;
        unsigned long long *m_in = (r & 1) ? fr.mask1 : fr.mask0;
        unsigned long long *m_out = (r & 1) ? fr.mask0 : fr.mask1;
        const Defer df{big.rows, big.cnt + (r % 3), big.cap, big.split};
        const MsRelaxOp<A> op{dist, m_out, out, fr.cnt + ((r + 1) % 3), fr.cap, st};
        for (uint32_t base = 0; base < n_in; base += gridDim.x * kTpbMs) {
            const uint32_t i = base + spread_rank<kTpbMs>() * gridDim.x + blockIdx.x;
            bool has = i < n_in;
            uint32_t x = 0, dx = 0, deg = 0;
            uint64_t off = 0;
            if (has) {
                x = __ldcg(in + i);
                m_in[x] = 0ull;  // nobody writes m_in this round
                dx = __ldcg(dist + x);
                const RowDesc d = fwd.desc[x];
                deg = d.len;
                off = d.off;
                has = deg > 0;
            }
            expand_rows<kTpbMs>(fwd, has, x, dx, off, deg, op, sm, cnt, df);
        }
        if (!grid_barrier(st)) break;
        const uint32_t nbig = min(ld_volatile(big.cnt + (r % 3)), big.cap);
        if (nbig) {
            expand_deferred<kTpbMs>(fwd, big.rows, nbig, op, cnt);
            if (!grid_barrier(st)) break;
        }
    }
    flush_counters(st, cnt, kCntPush);
    warp_count(&st->counters[kCntSrcEdges], cnt.edges);  // one source
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&st->counters[kCntRounds], static_cast<unsigned long long>(r));
}

// Waves of several sources.  A distance row holds the wave's sources padded to
// `4 * LPE` words, so LPE lanes relax an edge with one 16-byte load of either
// end's row each, and several edges' loads of a warp are in flight together.
// (One lane relaxing an edge's sources in turn waited for two dependent loads
// per source.)  While many vertices changed in the last round the frontier is
// the non-zero masks: a round scans them, and an improved bit is an OR without
// a result.  With a queue in those rounds too, the appends' atomics on its one
// counter and the wait for every mask's old value took most of the time
// (2.9 ms for 13 sources on R-MAT s19, 6 % of the L2's throughput).
// Short chunks and three blocks per SM with two edges per lane in flight keep
// the warps even: 13 sources on s19 take 1.37 ms with 256-entry chunks and four
// edges in two blocks, 1.13 with 128 and 1.05 with 64 entries.
constexpr uint32_t kMsChunk = 64;  // rows of at least this many entries are expanded by the whole grid
constexpr int kMsGroup = 2;        // edges per lane whose loads are in flight together
// A scan round hands out n / 32 tiles whatever it finds in them, so few
// improvements are better queued (511 x 511 grid, 13 sources: 12.3 ms with
// scans from n / 64 on, 9.2 from n / 16; R-MAT s19: 1.31, 1.30).
constexpr uint32_t kMsScan = 16;  // rounds after more than n / kMsScan improvements scan the masks

// Chunks of long rows met in a round (three counters, as for the frontier),
// and the entries of a queue rebuilt from the masks (three counters).  A warp
// per chunk: short, since the longest warp decides a round's time.  What finds
// no place in the list is relaxed by the warp that met it.
struct MsChunks {
    BigRow *rows;
    uint32_t *cnt;
    uint32_t cap;
    uint32_t *fill;
    uint32_t *tiles;  // three counters (TileFeed)
};

template <int A, int LPE>
struct MsWave {
    uint32_t *dist;
    unsigned long long *mask_out;
    bool queue;  // append improved vertices
    WarpBuf buf;

    // N 16-byte pieces of edges per lane: sources 4 quad .. 4 quad + 3 of edge
    // xs -> ys, those of `bits` (0: none).  xs's row is read through L1 (a
    // value lowered meanwhile is relaxed again next round), ys's from L2: a
    // stale row of a hub costs an atomic for every source, all of them on one
    // sector.
    template <int N>
    __device__ __forceinline__ uint32_t pieces(const uint32_t (&xs)[N], const uint32_t (&ys)[N],
                                               const uint32_t (&quad)[N], const uint32_t (&bits)[N]) const {
        constexpr uint64_t kRow = 4 * LPE;
        uint4 dx[N], dy[N];
        uint32_t hits = 0;
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (bits[j]) {
                dx[j] = *reinterpret_cast<const uint4 *>(dist + xs[j] * kRow + 4u * quad[j]);
                dy[j] = __ldcg(reinterpret_cast<const uint4 *>(dist + ys[j] * kRow + 4u * quad[j]));
            }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            uint32_t add = 0;
            if (bits[j]) {
                const uint32_t w = edge_weight<A>(xs[j], ys[j]);
                const uint32_t nd[4] = {dx[j].x + w, dx[j].y + w, dx[j].z + w, dx[j].w + w};
                const uint32_t od[4] = {dy[j].x, dy[j].y, dy[j].z, dy[j].w};
                uint32_t *row = dist + ys[j] * kRow + 4u * quad[j];
                uint32_t old[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    old[i] = ((bits[j] >> i) & 1u) && nd[i] < od[i] ? atomicMin(row + i, nd[i]) : 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i) add |= nd[i] < old[i] ? 1u << i : 0u;
                hits += add ? 1u : 0u;
            }
            const unsigned long long add64 = static_cast<unsigned long long>(add) << (4u * quad[j]);
            if (queue)
                buf.add(add && atomicOr(mask_out + ys[j], add64) == 0ull, ys[j]);
            else if (add)
                red_or(mask_out + ys[j], add64);
        }
        return hits;
    }

    // Relax 32 edges, one per lane (x -> y for the sources in m; m = 0: none).
    __device__ __forceinline__ uint32_t relax(uint32_t x, uint32_t y, unsigned long long m) const {
        constexpr int kPer = 32 / LPE;                            // edges per step
        constexpr int N = LPE < kMsGroup ? LPE : kMsGroup;        // steps in flight
        const uint32_t lane = lane_id();
        // Few sources per edge (high-diameter graphs: one or two of 64): the
        // pieces that hold any are dealt out instead of all of them, up to
        // half of what the steps would go through (511 x 511 grid, 64
        // sources: 31.4 -> 16.0 ms, with kMsScan; R-MAT s20: 9.4 -> 8.4).
        // Rows of up to four pieces are two such steps.
        constexpr bool kDeal = LPE >= 8;
        unsigned long long nz = 0;
        uint32_t excl = 0, total = 0;
        bool deal = false;
        if constexpr (kDeal) {
            nz = m | (m >> 1);
            nz = (nz | (nz >> 2)) & 0x1111111111111111ull;
            const uint32_t mine = __popcll(nz);
            total = __reduce_add_sync(kFull, mine);
            deal = total <= 16u * LPE;
            if (deal) {
                uint32_t incl = mine;
#pragma unroll
                for (uint32_t o = 1; o < 32u; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += t;
                }
                excl = incl - mine;
            }
        }
        const int steps = deal ? static_cast<int>((total + 31u) / 32u) : LPE;
        uint32_t hits = 0;
#pragma unroll(kDeal ? 1 : LPE)
        for (int s0 = 0; s0 < steps; s0 += N) {
            uint32_t xs[N], ys[N], bits[N], quad[N];
#pragma unroll
            for (int j = 0; j < N; ++j) {
                uint32_t src = LPE == 1 ? lane : (s0 + j) * kPer + lane / LPE;
                const uint32_t e = 32u * (s0 + j) + lane;
                quad[j] = lane % LPE;
                if (kDeal && deal) {
                    uint32_t lo = 0, hi = 32;  // the last lane whose pieces start at or before e
#pragma unroll
                    for (int step = 0; step < 5; ++step) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (__shfl_sync(kFull, excl, mid) <= e)
                            lo = mid;
                        else
                            hi = mid;
                    }
                    src = lo;
                    unsigned long long z = __shfl_sync(kFull, nz, src);
                    for (uint32_t k = e - __shfl_sync(kFull, excl, src); k && z; --k) z &= z - 1;
                    quad[j] = z ? static_cast<uint32_t>(__ffsll(static_cast<long long>(z)) - 1) >> 2 : 0u;
                }
                xs[j] = LPE == 1 ? x : __shfl_sync(kFull, x, src);
                ys[j] = LPE == 1 ? y : __shfl_sync(kFull, y, src);
                const unsigned long long ms = LPE == 1 ? m : __shfl_sync(kFull, m, src);
                bits[j] = kDeal && deal && e >= total ? 0u : static_cast<uint32_t>(ms >> (4u * quad[j])) & 15u;
            }
            hits += pieces<N>(xs, ys, quad, bits);
        }
        return hits;
    }
};

// The entries of a chunk (it lies in one segment) of x's row for the sources
// in m, by one warp; the next step's are read while this one's are relaxed.
template <int A, int LPE>
__device__ __forceinline__ uint32_t ms_chunk(const AdjView &fwd, const MsWave<A, LPE> &op, uint64_t off, uint32_t len,
                                             uint32_t x, unsigned long long m) {
    const uint32_t lane = lane_id();
    const uint32_t *rp = fwd.at(off);
    uint32_t hits = 0;
    uint32_t y_next = lane < len ? __ldg(rp + lane) : kTomb;
    for (uint32_t e0 = 0; e0 < len; e0 += 32u) {
        const uint32_t y = fwd.vid(y_next);
        y_next = e0 + 32u + lane < len ? __ldg(rp + e0 + 32u + lane) : kTomb;
        const bool live = y != kTomb;
        hits += op.relax(x, live ? y : 0u, live ? m : 0ull);
    }
    return hits;
}

template <int A, int LPE>
__global__ void __launch_bounds__(kTpbMs, 3) ms_wave(AdjView fwd, uint32_t n, uint32_t *dist, MsFrontier fr,
                                                     MsChunks ch, uint32_t max_rounds, Status *st) {
    __shared__ uint32_t s_scan[kTpbMs];
    __shared__ uint32_t s_x[kTpbMs];
    __shared__ unsigned long long s_m[kTpbMs];
    __shared__ const uint32_t *s_ptr[kTpbMs];
    __shared__ uint32_t s_buf[kTpbMs / 32][kWarpBuf];
    __shared__ uint32_t s_held[kTpbMs / 32];
    __shared__ uint32_t s_new;
    if (threadIdx.x < kTpbMs / 32) s_held[threadIdx.x] = 0;
    __syncthreads();
    ExpandCounters cnt;
    unsigned long long src_edges = 0;
    const uint32_t lane = lane_id(), wb = threadIdx.x & ~31u;
    const uint32_t warps = (gridDim.x * kTpbMs) >> 5;
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    bool scan = false;  // every block takes the same decisions from the same counts
    uint32_t r = 0;
    for (;; ++r) {
        uint32_t n_in = ld_volatile(fr.cnt + (r % 3));  // queued vertices, or improvements of a scan round
        if (n_in == 0) break;
        if (r >= max_rounds) {
            if (blockIdx.x == 0 && threadIdx.x == 0) set_error(st, kErrRounds, r);
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fr.cnt[(r + 2) % 3] = 0;
            ch.cnt[(r + 2) % 3] = 0;
            ch.fill[(r + 1) % 3] = 0;
            ch.tiles[(r + 1) % 3] = 0;
        }
        uint32_t *in = (r & 1) ? fr.q1 : fr.q0;
        uint32_t *out_cnt = fr.cnt + ((r + 1) % 3);
        unsigned long long *m_in = (r & 1) ? fr.mask1 : fr.mask0;
        unsigned long long *m_out = (r & 1) ? fr.mask0 : fr.mask1;
        uint32_t *ch_cnt = ch.cnt + r % 3;
        const bool was_scan = scan;
        scan = n_in > n / kMsScan;
        if (was_scan && !scan) {  // the masks as a queue
            const uint32_t rounded = (n + 31u) & ~31u;
            for (uint32_t v = blockIdx.x * kTpbMs + threadIdx.x; v < rounded; v += gridDim.x * kTpbMs)
                warp_enqueue(v < n && m_in[v] != 0ull, v, in, ch.fill + r % 3, fr.cap, st);
            if (!grid_barrier(st)) break;
            n_in = ld_volatile(ch.fill + r % 3);
        }
        const MsWave<A, LPE> op{dist, m_out, !scan,
                                WarpBuf{s_buf[threadIdx.x >> 5], s_held + (threadIdx.x >> 5), (r & 1) ? fr.q0 : fr.q1,
                                        out_cnt, fr.cap, st}};
        const uint32_t items = scan ? n : n_in;
        uint32_t hits = 0;
        uint32_t tile = 32;  // items per warp and step: few items spread over all warps
        while (tile > (scan ? 8u : 1u) && items <= static_cast<uint64_t>(warps) * (scan ? 4u : 1u) * (tile / 2))
            tile >>= 1;
        // A round whose tiles go round once asks for no further ones: a
        // thousand warps' requests on one counter take as long as their work.
        const bool more = items > static_cast<uint64_t>(warps) * tile;
        TileFeed feed(ch.tiles + r % 3, warps);
        for (uint64_t t = wid; t * tile < items; t = more ? feed.take() : items) {
            if (more) feed.ask();
            const uint64_t i = t * tile + lane;
            uint32_t x = 0, deg = 0;
            uint64_t off = 0;
            unsigned long long m = 0;
            if (lane < tile && i < items) {
                x = scan ? static_cast<uint32_t>(i) : __ldcg(in + i);
                // Nobody writes m_in this round: take the bits and clear them.
                m = __ldcg(m_in + x);
                if (m) {
                    m_in[x] = 0ull;
                    const RowDesc d = fwd.desc[x];
                    deg = d.len;
                    off = d.off;
                    if (deg) {
                        src_edges += static_cast<unsigned long long>(__popcll(m)) * deg;
                        cnt.rows += 1;
                        cnt.edges += deg;
                        if (fwd.cached(off)) cnt.edges_cached += deg;
                    }
                }
            }
            uint32_t bigs = __ballot_sync(kFull, deg >= kMsChunk);
            while (bigs) {
                const uint32_t l = __ffs(bigs) - 1;
                bigs &= bigs - 1;
                const uint32_t ldeg = __shfl_sync(kFull, deg, l), lx = __shfl_sync(kFull, x, l);
                const uint64_t loff = __shfl_sync(kFull, static_cast<unsigned long long>(off), l);
                const unsigned long long lm = __shfl_sync(kFull, m, l);
                const uint32_t k = (ldeg + kMsChunk - 1) / kMsChunk;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(ch_cnt, k);
                at = __shfl_sync(kFull, at, 0);
                const uint32_t fit = at < ch.cap ? min(k, ch.cap - at) : 0u;
                for (uint32_t c = lane; c < fit; c += 32u)
                    ch.rows[at + c] = BigRow{loff + static_cast<uint64_t>(c) * kMsChunk, lm, lx,
                                             min(kMsChunk, ldeg - c * kMsChunk)};
                if (lane == l) {
                    off += static_cast<uint64_t>(fit) * kMsChunk;
                    deg = fit < k ? deg - fit * kMsChunk : 0u;
                }
            }
            // What is left of the warp's rows concatenated (short rows; of
            // rows that found no place in the list a chunk at a time, which
            // lies in one segment), 32 edges per step; the next step's entries
            // are read while this one's are relaxed.
            while (__any_sync(kFull, deg != 0u)) {
                const uint32_t mine = min(deg, kMsChunk);
                uint32_t incl = mine;
#pragma unroll
                for (uint32_t o = 1; o < 32u; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += t;
                }
                const uint32_t total = __shfl_sync(kFull, incl, 31);
                s_scan[wb + lane] = incl - mine;
                s_x[wb + lane] = x;
                s_m[wb + lane] = m;
                s_ptr[wb + lane] = mine ? fwd.at(off) : nullptr;
                deg -= mine;
                off += mine;
                __syncwarp();
                auto fetch = [&](uint32_t e, uint32_t &owner) -> uint32_t {
                    owner = 0;
                    if (e >= total) return kTomb;
                    uint32_t lo = 0, hi = 32;  // the last lane whose edges start at or before e
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (s_scan[wb + mid] <= e)
                            lo = mid;
                        else
                            hi = mid;
                    }
                    owner = lo;
                    return __ldg(s_ptr[wb + lo] + (e - s_scan[wb + lo]));
                };
                uint32_t o_next, y_next = fetch(lane, o_next);
                for (uint32_t e0 = 0; e0 < total; e0 += 32u) {
                    const uint32_t y = fwd.vid(y_next), o = o_next;
                    y_next = fetch(e0 + 32u + lane, o_next);
                    const bool live = y != kTomb;
                    hits += op.relax(s_x[wb + o], live ? y : 0u, live ? s_m[wb + o] : 0ull);
                }
                __syncwarp();
            }
        }
        op.buf.flush();
        if (scan) block_add(out_cnt, min(hits, 1024u), &s_new);
        cnt.hits += hits;
        if (!grid_barrier(st)) break;
        const uint32_t nch = min(ld_volatile(ch_cnt), ch.cap);
        if (nch) {
            hits = 0;
            for (uint32_t i = wid; i < nch; i += warps) {
                const BigRow c = ch.rows[i];
                hits += ms_chunk(fwd, op, c.off, c.deg, c.x, c.payload);
            }
            op.buf.flush();
            if (scan) block_add(out_cnt, min(hits, 1024u), &s_new);
            cnt.hits += hits;
            if (!grid_barrier(st)) break;
        }
    }
    flush_counters(st, cnt, kCntPush);
    for (int o = 16; o > 0; o >>= 1) src_edges += __shfl_down_sync(kFull, src_edges, o);
    if (lane == 0 && src_edges) atomicAdd(&st->counters[kCntSrcEdges], src_edges);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&st->counters[kCntRounds], static_cast<unsigned long long>(r));
}

// Source-major output: out[j * n + v] = dist[v * 4 LPE + j] for j < k, through
// a shared-memory tile: 16-byte reads, 128-byte stores.
template <int LPE>
__global__ void __launch_bounds__(256) ms_transpose(const uint32_t *dist, uint32_t n, uint32_t k, uint32_t *out) {
    constexpr uint32_t kRow = 4 * LPE, kRows = 512 / LPE;
    __shared__ uint32_t tile[kRows][kRow + 1];
    const uint32_t v0 = blockIdx.x * kRows;
    const uint32_t rows = min(kRows, n - v0);
    for (uint32_t e = threadIdx.x; e < rows * LPE; e += 256u) {
        const uint32_t v = e / LPE, q = e % LPE;
        const uint4 d = *reinterpret_cast<const uint4 *>(dist + static_cast<uint64_t>(v0 + v) * kRow + 4u * q);
        tile[v][4 * q] = d.x;
        tile[v][4 * q + 1] = d.y;
        tile[v][4 * q + 2] = d.z;
        tile[v][4 * q + 3] = d.w;
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < kRows * k; e += 256u) {
        const uint32_t j = e / kRows, v = e % kRows;
        if (v < rows) __stcs(out + static_cast<uint64_t>(j) * n + v0 + v, tile[v][j]);
    }
}

// Digest of every row of a k x n result (the function of value_digest, so a
// query row and a maintained state with the same values agree).
__global__ void ms_row_digest(const uint32_t *rows, uint32_t n, unsigned long long *out) {
    const uint32_t j = blockIdx.y;
    const uint32_t *row = rows + static_cast<uint64_t>(j) * n;
    unsigned long long acc = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t d = row[v];
        if (d != kInf) acc += digest_mix((static_cast<unsigned long long>(v) << 32) | d);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane_id() == 0 && acc) atomicAdd(out + j, acc);
}

}  // namespace cig
