// pr.cuh - incremental PageRank by signed residual push.
//
// Same fixed point as the reference (samples/hybrid_pr/README.md: x[v] =
// 0.15 + 0.85 * sum x[u]/outdeg(u), parallel edges counted, dangling vertices
// send nothing) and the same residual protocol as include/framework/
// pr_residual.cuh:16-188: a vertex whose |residual| exceeds epsilon is
// consumed into its rank and pushes 0.85*r/deg to its out-neighbours; a batch
// first withdraws the old contributions of every touched source over its old
// row, mutates the topology, then re-adds them over the new row.
//
// Differences: one persistent cooperative kernel converges (no host count
// read per round): queue rounds while few vertices hold a residual above
// epsilon, sweeps over all vertices once many do (pr_converge); the rank is
// FP32 with a per-vertex Kahan compensation term (or FP64 throughout); the
// batch reports the FP64 L1 norm of the residual.
//
// FP32 residuals lose precision where many contributions pile up between two
// consumptions: a vertex with in-degree k takes up to k atomic adds per round,
// and the rounding of each (half an ulp of the running sum) adds up to about
// 6e-8 * sqrt(k) of its residual.  So in FP32 mode vertices whose in-degree
// was at least kPrHubInDeg at load keep their residual in an FP64 slot;
// everything else stays FP32.  The hub set is a bitmap (n/8 bytes) with a
// per-word prefix count (slot = prefix + rank in the word), small enough to
// stay in L2, since every scattered edge looks its destination up.
#pragma once

#include "common.cuh"
#include "expand.cuh"
#include "traverse.cuh"  // BigList

namespace cig {

constexpr float kAlphaF = 0.85f;
constexpr double kAlphaD = 0.85;

constexpr uint32_t kPrHubInDeg = 256;
// Sweeps spread the adds to a hub over this many copies of its slot, by block:
// adds to one address are served one after the other (16 thousand per sweep at
// the largest hub of R-MAT s18), and the consumer sums the copies.
constexpr uint32_t kHubCopies = 8;

template <class T>
struct PrArrays {
    T *rank;
    T *res;
    const uint32_t *hub_bits;    // FP32 mode: bit v set when v has an FP64 residual slot
    const uint32_t *hub_prefix;  // slots before word w of hub_bits
    double *res_hub;
    double *hub_more;  // kHubCopies - 1 further copies of res_hub, zero outside sweeps
    uint32_t hubs;
    float *comp;       // Kahan compensation of rank (FP32 mode only)
    uint32_t *queued;
    uint32_t *q0;
    uint32_t *q1;
    uint32_t *cnt;     // 3 round counters
    T *contrib;        // per queued item: alpha * r / deg (or 0)
    uint32_t *final_round;
    uint32_t cap;
};

template <class T>
__device__ __forceinline__ T pr_abs(T x) { return x < T(0) ? -x : x; }

template <class T>
__device__ __forceinline__ bool pr_finite(T x) { return isfinite(x); }

template <class T>
__device__ __forceinline__ int32_t hub_slot(const PrArrays<T> &a, uint32_t v) {
    if (sizeof(T) != 4 || !a.hub_bits) return -1;
    const uint32_t w = __ldg(a.hub_bits + (v >> 5));
    const uint32_t b = 1u << (v & 31u);
    if (!(w & b)) return -1;
    return static_cast<int32_t>(__ldg(a.hub_prefix + (v >> 5)) + __popc(w & (b - 1u)));
}

template <class T>
__device__ __forceinline__ T res_get(const PrArrays<T> &a, uint32_t v) {
    const int32_t h = hub_slot(a, v);
    return h >= 0 ? static_cast<T>(__ldcg(a.res_hub + h)) : __ldcg(a.res + v);
}

template <class T>
__device__ __forceinline__ void res_set(const PrArrays<T> &a, uint32_t v, double x) {
    const int32_t h = hub_slot(a, v);
    if (h >= 0)
        a.res_hub[h] = x;
    else
        a.res[v] = static_cast<T>(x);
}

// Threshold tests are made in the precision the residual is stored in, so
// that "crossed epsilon" (queue the vertex) and "above epsilon" (consume it)
// always agree; a residual left above epsilon but unqueued would never be
// consumed again.

// Atomic add of c; true when |res| went from <= eps to > eps.
template <class T>
__device__ __forceinline__ bool res_add_crossed(const PrArrays<T> &a, uint32_t v, T c, T eps, bool &finite) {
    const int32_t h = hub_slot(a, v);
    if (h >= 0) {
        const double old = atomicAdd(a.res_hub + h, static_cast<double>(c));
        const double nv = old + static_cast<double>(c);
        const double e = static_cast<double>(eps);
        finite = isfinite(nv);
        return fabs(old) <= e && fabs(nv) > e;
    }
    const T old = atomicAdd(a.res + v, c);
    const T nv = old + c;
    finite = pr_finite(nv);
    return pr_abs(old) <= eps && pr_abs(nv) > eps;
}

// Consume: if |res| > eps, return true with `taken` = the whole residual
// (FP64 slots keep their full value) and clear it.
template <class T>
__device__ __forceinline__ bool res_take(const PrArrays<T> &a, uint32_t v, T eps, double &taken, bool &finite) {
    const int32_t h = hub_slot(a, v);
    if (h >= 0) {
        const double r = __ldcg(a.res_hub + h);
        finite = isfinite(r);
        if (!(fabs(r) > static_cast<double>(eps))) return false;
        taken = r;
        a.res_hub[h] = 0.0;
        return true;
    }
    const T r = __ldcg(a.res + v);
    finite = pr_finite(r);
    if (!(pr_abs(r) > eps)) return false;
    taken = static_cast<double>(r);
    a.res[v] = T(0);
    return true;
}

template <class T>
__device__ __forceinline__ T rank_value(const PrArrays<T> &a, uint32_t v) {
    if (sizeof(T) == 4)
        return static_cast<T>(static_cast<double>(__ldcg(a.rank + v)) - static_cast<double>(__ldcg(a.comp + v)));
    return __ldcg(a.rank + v);
}

template <class T>
__device__ __forceinline__ void rank_add(const PrArrays<T> &a, uint32_t v, T r) {
    if (sizeof(T) == 4) {
        // Kahan summation: comp holds the negated low-order bits lost so far.
        const float y = static_cast<float>(r) - __ldcg(a.comp + v);
        const float s = static_cast<float>(__ldcg(a.rank + v));
        const float t = __fadd_rn(s, y);
        a.comp[v] = __fsub_rn(__fsub_rn(t, s), y);
        a.rank[v] = static_cast<T>(t);
    } else {
        a.rank[v] = __ldcg(a.rank + v) + r;
    }
}

// Frontier::Add (pr_residual.cuh:16-31): add to the residual and queue the
// vertex once when its magnitude crosses epsilon.
template <class T>
struct PrPushOp {
    PrArrays<T> a;
    uint32_t *queued;
    const T *contrib;
    T eps;
    uint32_t *q_out;
    uint32_t *q_cnt;
    uint32_t cap;
    Status *st;

    __device__ __forceinline__ bool edge(bool valid, uint32_t, uint32_t item, uint32_t y) const {
        bool want = false;
        if (valid) {
            bool finite = true;
            if (res_add_crossed(a, y, contrib[item], eps, finite) && __ldcg(queued + y) == 0u)
                want = atomicCAS(queued + y, 0u, 1u) == 0u;
            if (!finite) set_error(st, kErrNonFinite, y);
        }
        warp_enqueue(want, y, q_out, q_cnt, cap, st);
        return valid;
    }
};

template <class T>
__global__ void pr_init(PrArrays<T> a, uint32_t n) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        a.rank[v] = T(0);
        res_set(a, v, 0.15);
        if (a.comp) a.comp[v] = 0.f;
        a.queued[v] = 1u;
        a.q0[v] = v;
    }
}

constexpr int kTpbPr = 256;

// Sweep payload: the contribution's bits, in a word of its own width.
template <class T>
struct PrBits;
template <>
struct PrBits<float> {
    using type = uint32_t;
    static __device__ __forceinline__ type to(float c) { return __float_as_uint(c); }
    static __device__ __forceinline__ float from(type b) { return __uint_as_float(b); }
};
template <>
struct PrBits<double> {
    using type = unsigned long long;
    static __device__ __forceinline__ type to(double c) { return static_cast<type>(__double_as_longlong(c)); }
    static __device__ __forceinline__ double from(type b) { return __longlong_as_double(static_cast<long long>(b)); }
};

// Add in memory without a result (an atomicAdd whose result is unused was
// still issued as one that returns it).
__device__ __forceinline__ void red_add(float *p, float x) {
    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p), "f"(x) : "memory");
}
__device__ __forceinline__ void red_add(double *p, double x) {
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(p), "d"(x) : "memory");
}

// Sweeps: add to the residual, with no result to wait for (the sweep over
// the vertices finds what crossed epsilon).  The hub lookups of a thread's
// entries are in flight together (peek).
template <class T>
struct PrSweepOp {
    PrArrays<T> a;
    double *hub;  // this block's copy of the hubs' residuals
    __device__ __forceinline__ explicit PrSweepOp(const PrArrays<T> &arr) : a(arr), hub(arr.res_hub) {
        const uint32_t copy = blockIdx.x % kHubCopies;
        if (copy && a.hub_more) hub = a.hub_more + static_cast<uint64_t>(copy - 1) * a.hubs;
    }
    __device__ __forceinline__ int32_t peek(uint32_t y) const { return hub_slot(a, y); }
    __device__ __forceinline__ bool edge_peeked(bool valid, uint32_t, typename PrBits<T>::type c, uint32_t y,
                                                int32_t h) const {
        if (valid) {
            if (h >= 0)
                red_add(hub + h, static_cast<double>(PrBits<T>::from(c)));
            else
                red_add(a.res + y, PrBits<T>::from(c));
        }
        return valid;
    }
    __device__ __forceinline__ bool edge(bool valid, uint32_t x, typename PrBits<T>::type c, uint32_t y) const {
        return edge_peeked(valid, x, c, y, valid ? peek(y) : -1);
    }
};

// v's residual while others add to it.
template <class T>
__device__ __forceinline__ double res_look(const PrArrays<T> &a, uint32_t v, int32_t h) {
    if (h < 0) return static_cast<double>(__ldcg(a.res + v));
    double r = __ldcg(a.res_hub + h);
#pragma unroll
    for (uint32_t c = 0; c + 1 < kHubCopies; ++c) r += __ldcg(a.hub_more + static_cast<uint64_t>(c) * a.hubs + h);
    return r;
}

// Take it, leaving zero.
template <class T>
__device__ __forceinline__ double res_exchange(const PrArrays<T> &a, uint32_t v, int32_t h) {
    using B = typename PrBits<T>::type;
    if (h < 0) return static_cast<double>(PrBits<T>::from(atomicExch(reinterpret_cast<B *>(a.res + v), B{0})));
    auto take = [](double *p) {
        return __longlong_as_double(static_cast<long long>(atomicExch(reinterpret_cast<unsigned long long *>(p), 0ull)));
    };
    double r = take(a.res_hub + h);
#pragma unroll
    for (uint32_t c = 0; c + 1 < kHubCopies; ++c) r += take(a.hub_more + static_cast<uint64_t>(c) * a.hubs + h);
    return r;
}

// After the sweeps: what is left in the copies joins the hubs' own slots.
template <class T>
__device__ __forceinline__ void fold_hub_copies(const PrArrays<T> &a) {
    if (!a.hub_more) return;
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < a.hubs; h += gridDim.x * blockDim.x) {
        double r = __ldcg(a.res_hub + h);
        for (uint32_t c = 0; c + 1 < kHubCopies; ++c) {
            double *p = a.hub_more + static_cast<uint64_t>(c) * a.hubs + h;
            r += __ldcg(p);
            *p = 0.0;
        }
        a.res_hub[h] = r;
    }
}

// An FP64 residual enters an FP32 rank as two compensated adds (its float
// part and the rest), so nothing of it is lost.  Returns alpha * r / deg.
template <class T>
__device__ __forceinline__ T rank_consume(const PrArrays<T> &a, uint32_t v, double r, uint32_t deg) {
    const T hi = static_cast<T>(r);
    rank_add(a, v, hi);
    if (sizeof(T) == 4) {
        const T lo = static_cast<T>(r - static_cast<double>(hi));
        if (lo != T(0)) rank_add(a, v, lo);
    }
    return deg ? static_cast<T>(kAlphaD * r / static_cast<double>(deg)) : T(0);
}

// Rows of at least this many entries are pushed by the whole grid, a warp
// per chunk of as many entries (262k vertices, FP32: 512 takes 5.28 ms, 256
// 4.93, 128 4.77; 50k vertices, FP64: 1.59, 1.55, 1.56).
constexpr uint32_t kPrChunk = 128;

// Sweeps stop below epsilon: with epsilon itself as their threshold they left
// FP64 ranks at 50k vertices 2.5e-9 off (relative 2-norm, epsilon 1e-9) where
// queue rounds leave 2.2e-9 (8k vertices: 2.5e-9, 2.55e-9); with 0.7 of it
// 1.8e-9 at either size, for 3 % more time at a million vertices.
constexpr double kPrSweepEps = 0.7;

// The chunks a sweep leaves to the whole grid; what finds no place in the
// list is pushed by the warp that met it.
struct PrChunks {
    BigRow *rows;
    uint32_t *cnt;  // 3 counters
    uint32_t cap;
};

// Share of the vertices above which a round's queue is left for sweeps.
constexpr uint32_t kPrSweepShare = 16;

// Sweeps over all vertices until none holds a residual above epsilon.  Every
// vertex above it is consumed and pushed in one go, its residual taken with
// an exchange while other vertices add to it: what reaches a vertex before
// its turn is pushed on in the same sweep (Gauss-Seidel rather than Jacobi
// order), which needs about 0.6 of the pushes and half the rounds.  Against
// the queue rounds a push is an add without a result (no threshold test,
// queue claim or append per edge), and the consume pass with its barrier is
// gone.  Warps take tiles of vertices and push their rows without waiting for
// one another; the chunks of rows of kPrChunk entries and more are pushed by
// the whole grid after a barrier, in sweeps that have any.  (With block-wide
// rows inside the sweep nearly half of all warp time was spent at block
// barriers.)  Tiles shrink with n so that every warp gets a few.
// (Tiles handed out by a counter instead: no faster at 262k vertices, a fifth
// slower at 50k.)
// `act` (vertices consumed) and `ch.cnt`: three counters each (sweep s uses s
// mod 3, clears (s+1) mod 3, which was last read before the previous barrier).
// Returns false on a barrier error; `done` tells whether it converged.
template <class T>
__device__ __forceinline__ bool pr_sweeps(const AdjView &fwd, const PrArrays<T> &a, T eps, uint32_t n,
                                          uint32_t max_sweeps, const PrChunks &ch, uint32_t *act, uint32_t *seg_hot,
                                          ExpandSmem<kTpbPr, typename PrBits<T>::type> &sm, ExpandCounters &cnt,
                                          uint32_t &sweeps, bool &done, Status *st) {
    using B = typename PrBits<T>::type;
    const PrSweepOp<T> op{a};
    eps *= static_cast<T>(kPrSweepEps);
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * kTpbPr) >> 5;
    const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    uint32_t tile = 32;
    while (tile > 8 && n < 4ull * warps * tile) tile >>= 1;
    done = false;
    for (sweeps = 0;; ++sweeps) {
        if (sweeps && ld_volatile(act + (sweeps + 2) % 3) == 0) {
            done = true;
            return true;
        }
        if (sweeps >= max_sweeps) return true;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            act[(sweeps + 1) % 3] = 0;
            ch.cnt[(sweeps + 1) % 3] = 0;
        }
        uint32_t *ch_cnt = ch.cnt + sweeps % 3;
        uint32_t mine = 0;
        // The next tile's residuals are read while this one's rows are pushed.
        int32_t h_next = -1;
        double r_next = 0.0;
        auto look = [&](uint64_t t) {
            const uint64_t at = t * tile + lane;
            r_next = 0.0;
            if (lane < tile && at < n) {
                h_next = hub_slot(a, static_cast<uint32_t>(at));
                r_next = res_look(a, static_cast<uint32_t>(at), h_next);
            }
        };
        look(wid);
        for (uint64_t t = wid; t * tile < n; t += warps) {
            const uint32_t v = static_cast<uint32_t>(t * tile + lane);
            const int32_t h = h_next;
            const double seen = r_next;
            look(t + warps);
            uint32_t deg = 0;
            uint64_t off = 0;
            T c = T(0);
            if (!isfinite(seen)) set_error(st, kErrNonFinite, v);
            // (the threshold in the precision the residual is stored in)
            bool has = h >= 0 ? fabs(seen) > static_cast<double>(eps) : pr_abs(static_cast<T>(seen)) > eps;
            if (has) {
                const RowDesc d = fwd.desc[v];
                ++mine;
                c = rank_consume(a, v, res_exchange(a, v, h), rd_live(d));
                deg = d.len;
                off = d.off;
                has = deg > 0 && c != T(0);
                if (has) {
                    cnt.rows += 1;
                    cnt.edges += deg;
                    if (fwd.cached(off)) cnt.edges_cached += deg;
                    if (seg_hot && sweeps == 0) atomicAdd(seg_hot + (off >> kSegShift), deg);
                }
            }
            uint32_t bigs = __ballot_sync(kFull, has && deg >= kPrChunk);
            while (bigs) {
                const uint32_t l = __ffs(bigs) - 1;
                bigs &= bigs - 1;
                const uint32_t ldeg = __shfl_sync(kFull, deg, l), lv = __shfl_sync(kFull, v, l);
                const uint64_t loff = __shfl_sync(kFull, static_cast<unsigned long long>(off), l);
                const B lc = __shfl_sync(kFull, PrBits<T>::to(c), l);
                const uint32_t k = (ldeg + kPrChunk - 1) / kPrChunk;
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(ch_cnt, k);
                at = __shfl_sync(kFull, at, 0);
                const uint32_t fit = at < ch.cap ? min(k, ch.cap - at) : 0u;
                for (uint32_t i = lane; i < fit; i += 32u)
                    ch.rows[at + i] = BigRow{loff + static_cast<uint64_t>(i) * kPrChunk,
                                             static_cast<unsigned long long>(lc), lv,
                                             min(kPrChunk, ldeg - i * kPrChunk)};
                for (uint32_t i = fit; i < k; ++i)
                    sweep_row<32u>(fwd, fwd.at(loff + static_cast<uint64_t>(i) * kPrChunk),
                                   min(kPrChunk, ldeg - i * kPrChunk), lane, lv, lc, op, cnt);
            }
            expand_rows_warp<kTpbPr>(fwd, has && deg < kPrChunk, v, PrBits<T>::to(c), off, deg, op, sm, cnt);
        }
        mine = __reduce_add_sync(kFull, mine);
        if (lane == 0 && mine) atomicAdd(act + sweeps % 3, mine);
        if (!grid_barrier(st)) return false;
        const uint32_t nch = min(ld_volatile(ch_cnt), ch.cap);
        if (nch) {
            for (uint32_t i = wid; i < nch; i += warps) {
                const BigRow r = ch.rows[i];
                // A chunk starts a multiple of kPrChunk into a block that covers
                // whole segments or lies in one: it never straddles two.
                sweep_row<32u>(fwd, fwd.at(r.off), r.deg, lane, r.x, static_cast<B>(r.payload), op, cnt);
            }
            if (!grid_barrier(st)) return false;
        }
    }
}

// Persistent converge loop (Runtime::Converge, pr_residual.cuh:171-187).
// Queue rounds: each consumes the queued residuals (Consume, :54-71), then
// scatters them (Scatter, :74-100); the queue of round r is q[r&1] with
// cnt[r%3].  A queue of more than n / kPrSweepShare vertices is left for
// sweeps (pr_sweeps), which run to the end.  On exit `final_round` holds the
// round whose queue is still pending.
template <class T>
__global__ void __launch_bounds__(kTpbPr, 4) pr_converge(AdjView fwd, PrArrays<T> a, T eps, uint32_t n,
                                                      uint32_t max_rounds, PrChunks ch, uint32_t *act,
                                                      uint32_t *seg_hot, Status *st) {
    using B = typename PrBits<T>::type;
    __shared__ union {
        ExpandSmem<kTpbPr> rounds;
        ExpandSmem<kTpbPr, B> sweeps;
    } sm;
    ExpandCounters cnt;
    uint32_t r = 0, sweeps = 0;
    for (;; ++r) {
        const uint32_t n_in = ld_volatile(a.cnt + (r % 3));
        if (n_in == 0 || r >= max_rounds) break;
        const uint32_t *in = (r & 1) ? a.q1 : a.q0;
        if (n_in > n / kPrSweepShare) {
            for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in; i += gridDim.x * blockDim.x)
                a.queued[__ldcg(in + i)] = 0u;
            bool done = false;
            if (!pr_sweeps(fwd, a, eps, n, max_rounds - r, ch, act, seg_hot, sm.sweeps, cnt, sweeps, done, st)) break;
            fold_hub_copies(a);
            // The pending queue: empty, or (round bound) rebuilt in q0.
            if (blockIdx.x == 0 && threadIdx.x < 3) a.cnt[threadIdx.x] = 0;
            if (!done) {
                if (!grid_barrier(st)) break;
                const uint32_t rounded = (n + 31u) & ~31u;
                for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < rounded; v += gridDim.x * blockDim.x) {
                    bool want = false;
                    if (v < n) {
                        const int32_t h = hub_slot(a, v);
                        want = h >= 0 ? fabs(__ldcg(a.res_hub + h)) > static_cast<double>(eps)
                                      : pr_abs(__ldcg(a.res + v)) > eps;
                        if (want) a.queued[v] = 1u;
                    }
                    warp_enqueue(want, v, a.q0, a.cnt, a.cap, st);
                }
            }
            sweeps += r;
            r = 0;
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) a.cnt[(r + 2) % 3] = 0;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in; i += gridDim.x * blockDim.x) {
            const uint32_t v = __ldcg(in + i);
            a.queued[v] = 0u;
            T c = T(0);
            double r64 = 0.0;
            bool finite = true;
            if (res_take(a, v, eps, r64, finite)) c = rank_consume(a, v, r64, rd_live(fwd.desc[v]));
            if (!finite) set_error(st, kErrNonFinite, v);
            a.contrib[i] = c;
        }
        if (!grid_barrier(st)) break;
        PrPushOp<T> op{a, a.queued, a.contrib, eps, (r & 1) ? a.q0 : a.q1, a.cnt + ((r + 1) % 3), a.cap, st};
        for (uint32_t base = 0; base < n_in; base += gridDim.x * kTpbPr) {
            const uint32_t i = base + spread_rank<kTpbPr>() * gridDim.x + blockIdx.x;
            bool has = i < n_in;
            uint32_t v = 0, deg = 0;
            uint64_t off = 0;
            if (has) {
                v = __ldcg(in + i);
                const RowDesc d = fwd.desc[v];
                deg = d.len;
                off = d.off;
                has = deg > 0 && __ldcg(a.contrib + i) != T(0);
                if (has && seg_hot) atomicAdd(seg_hot + (off >> kSegShift), deg);
            }
            expand_rows<kTpbPr>(fwd, has, v, i, off, deg, op, sm.rounds, cnt);
        }
        if (!grid_barrier(st)) break;
    }
    flush_counters(st, cnt, kCntPr);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.final_round = r;
        atomicAdd(&st->counters[kCntPrRounds], static_cast<unsigned long long>(r + sweeps));
    }
}

// Move the pending queue of round `final_round` to (q0, cnt[0]) so that the
// next batch's amendments append to it (Runtime::BeginBatch, :140-156).
template <class T>
__global__ void pr_normalize_frontier(PrArrays<T> a) {
    const uint32_t r = *a.final_round;
    const uint32_t n = ld_volatile(a.cnt + (r % 3));
    const uint32_t *src = (r & 1) ? a.q1 : a.q0;
    if (src != a.q0)
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a.q0[i] = src[i];
}

template <class T>
__global__ void pr_set_counts(PrArrays<T> a) {
    const uint32_t r = *a.final_round;
    const uint32_t n = a.cnt[r % 3];
    a.cnt[0] = n;
    a.cnt[1] = 0;
    a.cnt[2] = 0;
    *a.final_round = 0;
}

// Unique touched sources of a batch (deletion and addition sources).
__global__ void collect_touched(const uint32_t *du, uint32_t nd, const uint32_t *au, uint32_t na, uint32_t n,
                                uint32_t *stamp, uint32_t epoch, uint32_t *list, uint32_t *count, uint32_t cap,
                                Status *st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t total = nd + na;
    bool want = false;
    uint32_t u = 0;
    if (i < total) {
        u = i < nd ? du[i] : au[i - nd];
        if (u < n && __ldcg(stamp + u) != epoch) want = atomicExch(stamp + u, epoch) != epoch;
    }
    if (__any_sync(kFull, i < total)) warp_enqueue(want, u, list, count, cap, st);
}

// contrib[i] = sign * alpha * rank[s] / deg(s) for every touched source
// (CombineValueBufferAmend, samples/hybrid_pr/hybrid_pr.cu:77-83).
template <class T>
__global__ void pr_amend_contrib(const RowDesc *desc, PrArrays<T> a, const uint32_t *list, const uint32_t *count,
                                 T sign, T *contrib) {
    const uint32_t n = *count;
    const T alpha = sizeof(T) == 4 ? T(kAlphaF) : T(kAlphaD);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t s = list[i];
        const uint32_t deg = rd_live(desc[s]);
        contrib[i] = deg ? sign * alpha * rank_value(a, s) / static_cast<T>(deg) : T(0);
    }
}

template <class T>
__global__ void __launch_bounds__(kTpbPr, 4) pr_amend_scatter(AdjView fwd, PrArrays<T> a, const uint32_t *list,
                                                           const uint32_t *count, const T *contrib, T eps,
                                                           Status *st) {
    __shared__ ExpandSmem<kTpbPr> sm;
    ExpandCounters cnt;
    const uint32_t n = *count;
    PrPushOp<T> op{a, a.queued, contrib, eps, a.q0, a.cnt, a.cap, st};
    for (uint32_t base = 0; base < n; base += gridDim.x * kTpbPr) {
        const uint32_t i = base + spread_rank<kTpbPr>() * gridDim.x + blockIdx.x;
        bool has = i < n;
        uint32_t s = 0, deg = 0;
        uint64_t off = 0;
        if (has) {
            s = list[i];
            const RowDesc d = fwd.desc[s];
            deg = d.len;
            off = d.off;
            has = deg > 0 && contrib[i] != T(0);
        }
        expand_rows<kTpbPr>(fwd, has, s, i, off, deg, op, sm, cnt);
    }
    flush_counters(st, cnt, kCntPr);
}

// FP32 mode: a batch's amend (-old contributions over the old rows, +new
// over the new rows) accumulates per vertex in FP64 and the net change is
// rounded into the FP32 residual once (pr_amend_fold).  Added straight into
// FP32 residuals, the two large, mostly cancelling contributions of a hub
// source leave a rounding residue of ~1e-7 of the contribution behind, which
// then converges into the ranks as a real error.
template <class T>
__global__ void pr_amend_contrib64(const RowDesc *desc, PrArrays<T> a, const uint32_t *list, const uint32_t *count,
                                   double sign, double *contrib) {
    const uint32_t n = *count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t s = list[i];
        const uint32_t deg = rd_live(desc[s]);
        contrib[i] = deg ? sign * kAlphaD * static_cast<double>(rank_value(a, s)) / static_cast<double>(deg) : 0.0;
    }
}

struct PrAmendOp {
    double *acc;
    const double *contrib;
    __device__ __forceinline__ bool edge(bool valid, uint32_t, uint32_t item, uint32_t y) const {
        if (valid) atomicAdd(acc + y, contrib[item]);
        return valid;
    }
};

template <class T>
__global__ void __launch_bounds__(kTpbPr, 4) pr_amend_scatter64(AdjView fwd, const uint32_t *list, const uint32_t *count,
                                                             const double *contrib, double *acc, Status *st) {
    __shared__ ExpandSmem<kTpbPr> sm;
    ExpandCounters cnt;
    const uint32_t n = *count;
    const PrAmendOp op{acc, contrib};
    for (uint32_t base = 0; base < n; base += gridDim.x * kTpbPr) {
        const uint32_t i = base + spread_rank<kTpbPr>() * gridDim.x + blockIdx.x;
        bool has = i < n;
        uint32_t s = 0, deg = 0;
        uint64_t off = 0;
        if (has) {
            s = list[i];
            const RowDesc d = fwd.desc[s];
            deg = d.len;
            off = d.off;
            has = deg > 0 && contrib[i] != 0.0;
        }
        expand_rows<kTpbPr>(fwd, has, s, i, off, deg, op, sm, cnt);
    }
    flush_counters(st, cnt, kCntPr);
}

// Round the accumulated amend into the residuals and queue the vertices
// whose residual crossed epsilon (Frontier::Add, pr_residual.cuh:16-31).
template <class T>
__global__ void pr_amend_fold(PrArrays<T> a, double *acc, uint32_t n, T eps, Status *st) {
    const uint32_t rounded = (n + 31u) & ~31u;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < rounded; v += gridDim.x * blockDim.x) {
        bool want = false;
        if (v < n) {
            const double d = acc[v];
            if (d != 0.0) {
                acc[v] = 0.0;
                // one thread per vertex: a plain add, crossing tested as in res_add_crossed
                const int32_t h = hub_slot(a, v);
                bool crossed, finite;
                if (h >= 0) {
                    const double old = a.res_hub[h], nv = old + d, e = static_cast<double>(eps);
                    a.res_hub[h] = nv;
                    finite = isfinite(nv);
                    crossed = fabs(old) <= e && fabs(nv) > e;
                } else {
                    const T old = a.res[v];
                    const T nv = static_cast<T>(static_cast<double>(old) + d);
                    a.res[v] = nv;
                    finite = pr_finite(nv);
                    crossed = pr_abs(old) <= eps && pr_abs(nv) > eps;
                }
                if (!finite) set_error(st, kErrNonFinite, v);
                if (crossed && a.queued[v] == 0u) {
                    a.queued[v] = 1u;
                    want = true;
                }
            }
        }
        warp_enqueue(want, v, a.q0, a.cnt, a.cap, st);
    }
}

// FP32 mode, after the static solve: the residual that the ranks really leave,
// 0.15 + alpha P^T x - x in FP64, takes the place of the FP32 one (one step of
// iterative refinement).  The solve starts from 0.15 rounded to FP32 (4e-8 off
// at every vertex) and adds equal contributions up in FP32, whose roundings
// have one sign; sweeps add up more between two consumptions than queue
// rounds, which made the ranks of a 262k-vertex R-MAT 3.1e-8 off instead of
// 2.8e-8 (relative 2-norm), and of smaller ones up to 1.2e-7.
__device__ __forceinline__ double rank_exact(const PrArrays<float> &a, uint32_t v) {
    return static_cast<double>(__ldcg(a.rank + v)) - static_cast<double>(__ldcg(a.comp + v));
}

struct PrRefineOp {
    double *acc;
    __device__ __forceinline__ bool edge(bool valid, uint32_t, unsigned long long c, uint32_t y) const {
        if (valid) red_add(acc + y, PrBits<double>::from(c));
        return valid;
    }
};

// acc += alpha P^T x.
__global__ void __launch_bounds__(kTpbPr, 4) pr_refine_scatter(AdjView fwd, PrArrays<float> a, uint32_t n, double *acc,
                                                               Status *st) {
    __shared__ ExpandSmem<kTpbPr, unsigned long long> sm;
    ExpandCounters cnt;
    const PrRefineOp op{acc};
    for (uint32_t base = 0; base < n; base += gridDim.x * kTpbPr) {
        const uint32_t v = base + spread_rank<kTpbPr>() * gridDim.x + blockIdx.x;
        RowDesc d{0, 0, 0};
        unsigned long long c = 0;
        if (v >= base && v < n) {
            d = fwd.desc[v];
            const uint32_t deg = rd_live(d);
            if (deg) c = PrBits<double>::to(kAlphaD * rank_exact(a, v) / static_cast<double>(deg));
        }
        expand_rows<kTpbPr>(fwd, d.len > 0u, v, c, d.off, d.len, op, sm, cnt);
    }
    flush_counters(st, cnt, kCntPr);
}

// acc = 0.15 + acc - x - r: what the residual lacks, for pr_amend_fold.
__global__ void pr_refine_diff(PrArrays<float> a, uint32_t n, double *acc) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int32_t h = hub_slot(a, v);
        const double r = h >= 0 ? a.res_hub[h] : static_cast<double>(a.res[v]);
        acc[v] = 0.15 + acc[v] - rank_exact(a, v) - r;
    }
}

// FP64 L1 norm of the residual.
template <class T>
__global__ void pr_residual_l1(PrArrays<T> a, uint32_t n, double *out) {
    double acc = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int32_t h = hub_slot(a, v);
        acc += fabs(h >= 0 ? a.res_hub[h] : static_cast<double>(a.res[v]));
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
    if (lane_id() == 0 && acc != 0.0) atomicAdd(out, acc);
}

template <class T>
__global__ void pr_export(PrArrays<T> a, uint32_t n, float *rank, float *res, double *rank64, double *res64) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const T x = rank_value(a, v);
        if (rank) rank[v] = static_cast<float>(x);
        if (res) res[v] = static_cast<float>(res_get(a, v));
        if (rank64) rank64[v] = static_cast<double>(x);
        if (res64) res64[v] = static_cast<double>(res_get(a, v));
    }
}

}  // namespace cig
