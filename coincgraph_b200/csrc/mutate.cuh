// mutate.cuh - GPU batch maintenance of an adjacency arena.
//
// Semantics follow the reference's source-local chunk store exactly
// (include/groute/graphs/source_local_chunk_store.h:219-391, 670-848) so that
// rows stay identical, element for element:
//   deletion phase: for every source, a destination requested k times loses
//     its first min(k, present) occurrences; survivors keep their order
//     (BuildDeletionPlan / ShouldDelete / CompactSourceInPlace);
//   addition phase: destinations are appended in input order; a row that
//     outgrows its power-of-two block moves to a larger block
//     (RewriteSourceToNewBlock).
// The batch is grouped by source with a device radix sort of 64-bit keys
// (source << 32 | destination) for deletions and (source << 32 | input index)
// for additions; the latter keeps input order inside a source, as the
// reference's stable radix sort does (effective_update_batch.h:48-73).
//
// Design differences from the reference (same rows):
//   - a deleted entry is overwritten with a tombstone instead of shifting
//     the rest of the row; the scan of a row stops once every requested
//     deletion of that row has been found, so a batch reads about half of
//     each touched row and writes one word per deletion;
//   - a row is compacted (tombstones dropped, order kept) when tombstones
//     reach a quarter of its length, or when its block would overflow: in
//     place if the live entries then fit, else into the larger block (which
//     it enters as it is, tombstones and all, where they fit);
//   - grouping, matching, allocation and appends all run on the GPU.
#pragma once

#include <cub/block/block_radix_sort.cuh>
#include <cub/block/block_scan.cuh>

#include "cache.cuh"
#include "common.cuh"
#include "posindex.cuh"

namespace cig {

constexpr uint32_t kKeyShift = 32;
constexpr unsigned long long kKeyNone = ~0ull;
constexpr uint32_t kWarpRowMax = 4096;  // larger rows use the block path
constexpr int kMutWarps = 8;            // warps per block of the warp-path kernels
constexpr int kTpbMut = 256;            // threads per block of the block-path kernels

__device__ __forceinline__ uint32_t key_src(unsigned long long k) { return static_cast<uint32_t>(k >> kKeyShift); }
__device__ __forceinline__ uint32_t key_low(unsigned long long k) { return static_cast<uint32_t>(k); }

// Device-side block allocator: per class a partially used segment
// [cur_next, cur_end) and a global bump pointer over whole segments.
// Blocks left by relocation are not reused.
struct ArenaAlloc {
    unsigned long long seg_bump;
    unsigned long long seg_total;
    unsigned long long cur_next[kNumClasses];
    unsigned long long cur_end[kNumClasses];
    unsigned long long base_cur[kNumClasses];
    unsigned long long base_new[kNumClasses];
    uint32_t demand[kNumClasses];
    uint32_t avail[kNumClasses];
};

__device__ __forceinline__ uint32_t class_for(uint32_t deg) {
    if (deg <= (1u << kMinClass)) return kMinClass;
    return 32u - __clz(deg - 1u);
}

__device__ __forceinline__ unsigned long long alloc_offset(const ArenaAlloc *al, uint32_t cls, uint32_t rank) {
    if (cls <= kSegShift && rank < al->avail[cls])
        return al->base_cur[cls] + (static_cast<unsigned long long>(rank) << cls);
    const uint32_t r = cls <= kSegShift ? rank - al->avail[cls] : rank;
    return al->base_new[cls] + (static_cast<unsigned long long>(r) << cls);
}

// Keys for the deletion phase.  Invalid records (id out of range) sort last;
// they remove nothing and are reported as missing deletes.
__global__ void make_keys_del(const uint32_t *du, const uint32_t *dv, uint32_t nd, uint32_t n,
                              unsigned long long *kf, unsigned long long *kr, Status *) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nd) return;
    const uint32_t u = du[i], v = dv[i];
    if (u < n && v < n) {
        kf[i] = (static_cast<unsigned long long>(u) << kKeyShift) | v;
        kr[i] = (static_cast<unsigned long long>(v) << kKeyShift) | u;
    } else {
        kf[i] = kKeyNone;
        kr[i] = kKeyNone;
    }
}

// Keys for the addition phase: (source << 32 | index) keeps input order.
__global__ void make_keys_add(const uint32_t *au, const uint32_t *av, uint32_t na, uint32_t n,
                              unsigned long long *kf, unsigned long long *kr, Status *st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= na) return;
    const uint32_t u = au[i], v = av[i];
    if (u < n && v < n) {
        kf[i] = (static_cast<unsigned long long>(u) << kKeyShift) | i;
        kr[i] = (static_cast<unsigned long long>(v) << kKeyShift) | i;
    } else {
        kf[i] = kKeyNone;
        kr[i] = kKeyNone;
        atomicAdd(&st->counters[kCntInvalid], 1ull);
    }
}

// Source groups of a sorted key array, in key order: group g spans keys
// [start[g], end[g]).  Built by group_flags, a device exclusive scan of the
// flags and group_scatter, so a group's end is one load away.
struct Groups {
    const uint32_t *start;
    const uint32_t *end;
    const uint32_t *count;
};

__global__ void group_flags(const unsigned long long *keys, uint32_t m, uint32_t *flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const unsigned long long k = keys[i];
    flags[i] = (k != kKeyNone && (i == 0 || key_src(keys[i - 1]) != key_src(k))) ? 1u : 0u;
}

__global__ void group_scatter(const unsigned long long *keys, uint32_t m, const uint32_t *flags, const uint32_t *pos,
                              uint32_t *start, uint32_t *end, uint32_t *count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const unsigned long long k = keys[i];
    if (k == kKeyNone) return;
    if (flags[i]) {
        start[pos[i]] = i;
        if (pos[i] > 0) end[pos[i] - 1] = i;
    }
    if (i + 1 == m || keys[i + 1] == kKeyNone) {  // last valid key closes the last group
        end[pos[i] + flags[i] - 1] = i + 1;
        *count = pos[i] + flags[i];
    }
}

// ---------------------------------------------------------------- one sort per batch
// The four key sets of a whole batch (forward and reverse deletion keys,
// forward and reverse addition keys) are packed into one array and sorted
// by one radix sort: key = set << 2F | first << F | second with F bits per
// field (2^F > n and > the phase sizes), so the sort has 2 + 2F significant
// bits instead of four sorts of 32 + log2(n) bits.  An invalid record gets
// all-ones fields and sorts to the end of its set.  Sets occupy [0, nd),
// [nd, 2nd), [2nd, 2nd+na), [2nd+na, 2nd+2na).
struct PackedSets {
    uint32_t off[5];
    uint32_t f;  // field width F
};

// Packed key of record i; counts a rejected addition once.
__device__ __forceinline__ unsigned long long packed_key(const uint32_t *du, const uint32_t *dv, const uint32_t *au,
                                                         const uint32_t *av, uint32_t n, const PackedSets &ps,
                                                         uint32_t i, Status *st) {
    const uint32_t f = ps.f;
    const unsigned long long none = (1ull << f) - 1;
    uint32_t set, first, second;
    bool ok;
    if (i < ps.off[2]) {
        set = i < ps.off[1] ? 0u : 1u;
        const uint32_t j = i - (set ? ps.off[1] : 0u);
        const uint32_t u = du[j], v = dv[j];
        ok = u < n && v < n;
        first = set == 0 ? u : v;
        second = set == 0 ? v : u;
    } else {
        set = i < ps.off[3] ? 2u : 3u;
        const uint32_t j = i - (set == 3 ? ps.off[3] : ps.off[2]);
        const uint32_t u = au[j], v = av[j];
        ok = u < n && v < n;
        first = set == 2 ? u : v;
        second = j;
        if (!ok && set == 2) atomicAdd(&st->counters[kCntInvalid], 1ull);
    }
    const unsigned long long a = ok ? first : none, b = ok ? second : none;
    return (static_cast<unsigned long long>(set) << (2 * f)) | (a << f) | b;
}

__global__ void make_keys_batch(const uint32_t *du, const uint32_t *dv, const uint32_t *au, const uint32_t *av,
                                uint32_t n, PackedSets ps, unsigned long long *out, Status *st) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ps.off[4]) out[i] = packed_key(du, dv, au, av, n, ps, i, st);
}

// Sorted packed keys -> the usual (first << 32 | second) keys of each set,
// and group flags (first key of every source run inside its set).
__global__ void unpack_keys_batch(const unsigned long long *sorted, PackedSets ps, unsigned long long *k0,
                                  unsigned long long *k1, unsigned long long *k2, unsigned long long *k3,
                                  uint32_t *flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ps.off[4]) return;
    const uint32_t f = ps.f;
    const unsigned long long mask = (1ull << f) - 1;
    const unsigned long long k = sorted[i];
    const uint32_t set = static_cast<uint32_t>(k >> (2 * f)) & 3u;
    const unsigned long long a = (k >> f) & mask, b = k & mask;
    const bool ok = a != mask;
    unsigned long long *dst = set == 0 ? k0 : set == 1 ? k1 : set == 2 ? k2 : k3;
    dst[i - ps.off[set]] = ok ? ((a << kKeyShift) | b) : kKeyNone;
    flags[i] = (ok && (i == ps.off[set] || (sorted[i - 1] >> f) != (k >> f))) ? 1u : 0u;
}

// Groups of the four sets from one exclusive scan of the flags; group
// indices and key positions are relative to the set.
struct SetGroups {
    uint32_t *start[4];
    uint32_t *end[4];
    uint32_t *count[4];
};

__global__ void group_scatter_batch(const unsigned long long *sorted, PackedSets ps, const uint32_t *flags,
                                    const uint32_t *pos, SetGroups sg) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ps.off[4]) return;
    const uint32_t f = ps.f;
    const unsigned long long mask = (1ull << f) - 1;
    const unsigned long long k = sorted[i];
    if (((k >> f) & mask) == mask) return;  // invalid record
    const uint32_t set = static_cast<uint32_t>(k >> (2 * f)) & 3u;
    const uint32_t s0 = ps.off[set], s1 = ps.off[set + 1];
    const uint32_t base = pos[s0];
    const uint32_t local = i - s0;
    const uint32_t g = pos[i] - base;
    if (flags[i]) {
        sg.start[set][g] = local;
        if (g > 0) sg.end[set][g - 1] = local;
    }
    if (i + 1 == s1 || ((sorted[i + 1] >> f) & mask) == mask) {  // last valid key of the set
        sg.end[set][g + flags[i] - 1] = local + 1;
        *sg.count[set] = g + flags[i];
    }
}

// Small batches (at most kSmallSortKeys packed keys): one block does all of it,
// the phase's begin included.  (The device-wide sort and the kernels around it
// are eight launches of a few microseconds each, and its passes as many
// again; a block sort between five of those launches took 45 us on 4,000
// keys.)
constexpr int kSmallSortItems = 8;
constexpr uint32_t kSmallSortKeys = 512 * kSmallSortItems;

struct SmallBatch {
    const uint32_t *du, *dv, *au, *av;
    unsigned long long *keys[4];  // sorted keys of each set
    uint32_t *epoch;              // phase_begin's work
    uint32_t *counters;
    unsigned long long mask;
    uint32_t *seg_ctl;
};

template <int THREADS>
__global__ void __launch_bounds__(THREADS) small_batch(SmallBatch sb, uint32_t n, PackedSets ps, SetGroups sg,
                                                       Status *st) {
    using Sort = cub::BlockRadixSort<unsigned long long, THREADS, kSmallSortItems>;
    using Scan = cub::BlockScan<uint32_t, THREADS>;
    constexpr uint32_t kItems = THREADS * kSmallSortItems;
    __shared__ union {
        typename Sort::TempStorage sort;
        unsigned long long sorted[kItems];
    } sm;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ uint32_t s_base[4];
    begin_phase(sb.epoch, sb.counters, sb.mask, sb.seg_ctl);
    if (threadIdx.x < 4) *sg.count[threadIdx.x] = 0u;
    const uint32_t total = ps.off[4], f = ps.f;
    const uint32_t i0 = threadIdx.x * kSmallSortItems;
    unsigned long long k[kSmallSortItems];
#pragma unroll
    for (int j = 0; j < kSmallSortItems; ++j)  // ~0 sorts behind every key of 2 + 2 f < 64 bits
        k[j] = i0 + j < total ? packed_key(sb.du, sb.dv, sb.au, sb.av, n, ps, i0 + j, st) : ~0ull;
    Sort(sm.sort).Sort(k, 0, 2 + 2 * static_cast<int>(f));
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallSortItems; ++j) sm.sorted[i0 + j] = k[j];
    __syncthreads();
    const unsigned long long mask = (1ull << f) - 1;
    uint32_t flags = 0;
#pragma unroll
    for (int j = 0; j < kSmallSortItems; ++j) {
        const uint32_t i = i0 + j;
        const uint32_t set = i < ps.off[2] ? (i < ps.off[1] ? 0u : 1u) : (i < ps.off[3] ? 2u : 3u);
        const uint32_t s0 = set == 0 ? 0u : set == 1 ? ps.off[1] : set == 2 ? ps.off[2] : ps.off[3];
        const unsigned long long a = (k[j] >> f) & mask, b = k[j] & mask;
        const bool ok = i < total && a != mask;
        const unsigned long long prev = i == 0 ? ~k[j] : j ? k[j ? j - 1 : 0] : sm.sorted[i - 1];
        if (ok && (i == s0 || (prev >> f) != (k[j] >> f))) flags |= 1u << j;
        unsigned long long *dst = set == 0 ? sb.keys[0] : set == 1 ? sb.keys[1] : set == 2 ? sb.keys[2] : sb.keys[3];
        if (i < total) dst[i - s0] = ok ? ((a << kKeyShift) | b) : kKeyNone;
    }
    uint32_t pos;
    Scan(scan_tmp).ExclusiveSum(static_cast<uint32_t>(__popc(flags)), pos);
#pragma unroll
    for (int j = 0; j < kSmallSortItems; ++j) {
        const uint32_t at = pos + __popc(flags & ((1u << j) - 1u));
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (i0 + j == ps.off[t]) s_base[t] = at;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSmallSortItems; ++j) {
        const uint32_t i = i0 + j;
        if (i >= total || ((k[j] >> f) & mask) == mask) continue;  // pad or invalid record
        const uint32_t set = i < ps.off[2] ? (i < ps.off[1] ? 0u : 1u) : (i < ps.off[3] ? 2u : 3u);
        const uint32_t s0 = set == 0 ? 0u : set == 1 ? ps.off[1] : set == 2 ? ps.off[2] : ps.off[3];
        const uint32_t s1 = set == 0 ? ps.off[1] : set == 1 ? ps.off[2] : set == 2 ? ps.off[3] : total;
        uint32_t *start = set == 0 ? sg.start[0] : set == 1 ? sg.start[1] : set == 2 ? sg.start[2] : sg.start[3];
        uint32_t *end = set == 0 ? sg.end[0] : set == 1 ? sg.end[1] : set == 2 ? sg.end[2] : sg.end[3];
        uint32_t *count = set == 0 ? sg.count[0] : set == 1 ? sg.count[1] : set == 2 ? sg.count[2] : sg.count[3];
        const uint32_t head = (flags >> j) & 1u;
        const uint32_t g = pos + __popc(flags & ((1u << j) - 1u)) - s_base[set];
        if (head) {
            start[g] = i - s0;
            if (g > 0) end[g - 1] = i - s0;
        }
        const unsigned long long next = j + 1 < kSmallSortItems ? k[j + 1 < kSmallSortItems ? j + 1 : j]
                                        : i + 1 < kItems        ? sm.sorted[i + 1]
                                                                : ~0ull;
        if (i + 1 == s1 || ((next >> f) & mask) == mask) {  // last valid key of the set
            end[g + head - 1] = i - s0 + 1;
            *count = g + head;
        }
    }
}

// Deletion run of key `key` inside the group [gs, ge): the index of the
// run's first key (a unique run id) and its requested count.
__device__ __forceinline__ bool find_run(const unsigned long long *keys, uint32_t gs, uint32_t ge,
                                         unsigned long long key, uint32_t &run, uint32_t &req) {
    uint32_t lo = gs, hi = ge;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (keys[mid] < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    if (lo >= ge || keys[lo] != key) return false;
    uint32_t e = lo + 1;
    while (e < ge && keys[e] == key) ++e;
    run = lo;
    req = e - lo;
    return true;
}

__device__ __forceinline__ void write_slot(const AdjView &view, unsigned long long off, uint32_t value) {
    *view.wptr(off) = value;
}

// Rows to compact, in one array: rows a warp serves from the front, longer
// ones (kWarpMove) from the back, so that each kind is dealt to workers of its
// own width without reading the other's descriptors.
constexpr uint32_t kWarpMove = 1024;  // survivors of rows up to this length are moved by one warp
struct CompactList {
    uint32_t *rows;
    uint32_t *count;      // from the front
    uint32_t *big_count;  // from the back
    uint32_t cap;
};

// Record the tombstones a row received; queue it for compaction when they
// reach a quarter of its length.
__device__ __forceinline__ void finish_row(RowDesc *desc, uint32_t u, const RowDesc &d, uint32_t removed,
                                           const CompactList &cl) {
    if (!removed) return;
    const uint32_t tombs = rd_tombs(d) + removed;
    desc[u].meta = rd_meta(rd_cls(d), tombs);
    if (4ull * tombs >= d.len || tombs >= kMaxTombs / 2) {
        if (d.len <= kWarpMove)
            cl.rows[atomicAdd(cl.count, 1u)] = u;
        else
            cl.rows[cl.cap - 1u - atomicAdd(cl.big_count, 1u)] = u;
    }
}

// ---------------------------------------------------------------- deletion

// Rows of at most kWarpRowMax slots, at most 32 keys: lane j holds key j;
// run multiplicities and matched counts live in the run-head lanes.
// Returns the number of tombstones written.
__device__ __forceinline__ uint32_t warp_tomb_regs(const AdjView &view, const RowDesc &d,
                                                   const unsigned long long *keys, uint32_t gs, uint32_t m) {
    const uint32_t lane = lane_id();
    const bool kvalid = lane < m;
    const uint32_t kd = kvalid ? key_low(keys[gs + lane]) : 0u;
    const uint32_t vmask = __ballot_sync(kFull, kvalid);
    const uint32_t peers = __match_any_sync(kFull, kd) & vmask;
    const uint32_t req_here = kvalid ? __popc(peers) : 0u;
    uint32_t mcount = 0;
    uint32_t left = m;  // requests not yet satisfied (uniform)
    const uint32_t *src = view.at(d.off);
    uint32_t *dst = nullptr;
    uint4 q = make_uint4(0, 0, 0, 0);
    if (4u * lane < d.len) q = *reinterpret_cast<const uint4 *>(src + 4u * lane);
    for (uint32_t base = 0; base < d.len && left; base += 128u) {
        const uint32_t k0 = base + 4u * lane;
        const uint32_t e[4] = {q.x, q.y, q.z, q.w};
        // prefetch the next chunk while this one is matched
        if (base + 128u + 4u * lane < d.len) q = *reinterpret_cast<const uint4 *>(src + base + 128u + 4u * lane);
        int run[4] = {-1, -1, -1, -1};
        for (uint32_t j = 0; j < m; ++j) {
            const uint32_t kj = __shfl_sync(kFull, kd, j);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                if (run[s] < 0 && k0 + s < d.len && e[s] == kj) run[s] = static_cast<int>(j);
        }
        uint32_t cm[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) cm[s] = __ballot_sync(kFull, run[s] >= 0);
        uint32_t any = cm[0] | cm[1] | cm[2] | cm[3];
        bool del[4] = {false, false, false, false};
        while (any) {  // position order: lane-major, then s
            const uint32_t l = __ffs(any) - 1;
            any &= any - 1;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if ((cm[s] >> l) & 1u) {
                    const uint32_t r = static_cast<uint32_t>(__shfl_sync(kFull, run[s], l));
                    const uint32_t req = __shfl_sync(kFull, req_here, r);
                    const uint32_t seen = __shfl_sync(kFull, mcount, r);
                    if (lane == r) mcount = seen + 1;
                    if (seen < req) {
                        --left;
                        if (lane == l) del[s] = true;
                    }
                }
            }
        }
        if (del[0] | del[1] | del[2] | del[3]) {
            if (!dst) dst = view.wptr(d.off);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                if (del[s]) dst[k0 + s] = kTomb;
        }
        __syncwarp();
    }
    return m - left;
}

// Any number of keys: binary search in the sorted group keys in global
// memory; matched[run] counts the occurrences of a run seen so far.
__device__ __forceinline__ uint32_t warp_tomb_global(const AdjView &view, const RowDesc &d, uint32_t u,
                                                     const unsigned long long *keys, uint32_t gs, uint32_t ge,
                                                     uint32_t *matched) {
    const uint32_t lane = lane_id();
    const unsigned long long uhi = static_cast<unsigned long long>(u) << kKeyShift;
    uint32_t left = ge - gs, done = 0;
    for (uint32_t base = 0; base < d.len && left; base += 32u) {
        const uint32_t k = base + lane;
        const bool valid = k < d.len;
        const uint32_t x = valid ? *view.at(d.off + k) : kTomb;
        uint32_t run = 0xFFFFFFFFu, req = 0;
        const bool cand = x != kTomb && find_run(keys, gs, ge, uhi | x, run, req);
        bool del = false;
        if (__ballot_sync(kFull, cand)) {
            const uint32_t peers = __match_any_sync(kFull, run);
            const uint32_t before = __popc(peers & lanemask_lt());
            uint32_t seen = 0;
            if (cand) seen = matched[run];
            del = cand && seen + before < req;
            __syncwarp();
            if (cand && before == 0) matched[run] = seen + __popc(peers);
            __syncwarp();
        }
        const uint32_t dm = __ballot_sync(kFull, del);
        if (del) write_slot(view, d.off + k, kTomb);
        left -= __popc(dm);
        done += __popc(dm);
    }
    return done;
}

// Deletion phase, one warp per source group; rows above kWarpRowMax go to
// the block path.  Launched with kMutWarps * 32 threads per block.
__global__ void __launch_bounds__(kMutWarps * 32)
    mutate_delete(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr, const uint32_t *list,
                  const uint32_t *list_count, uint32_t *matched, uint32_t *big, uint32_t *big_count,
                  CompactList cl, unsigned long long *stats, Status *st) {
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nl = *list_count;
    unsigned long long removed = 0, changed = 0;
    for (uint32_t li = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; li < nl; li += warps) {
        const uint32_t g = list[li];
        const uint32_t gs = gr.start[g];
        const uint32_t ge = gr.end[g];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        if (d.len > kWarpRowMax) {
            if (lane == 0) big[atomicAdd(big_count, 1u)] = g;
            continue;
        }
        const uint32_t done = (ge - gs <= 32u) ? warp_tomb_regs(view, d, keys, gs, ge - gs)
                                               : warp_tomb_global(view, d, u, keys, gs, ge, matched);
        if (lane == 0) {
            finish_row(desc, u, d, done, cl);
            removed += done;
            changed += done != 0;
        }
    }
    if (lane == 0 && stats) {
        if (removed) atomicAdd(&stats[kCntRemoved], removed);
        if (changed) atomicAdd(&stats[kCntChanged], changed);
    }
}

// Rows above kWarpRowMax: one block per row, tiles of kTpbMut x 8 slots
// (two 16-byte loads per thread), the group's keys and matched counts in
// shared memory (up to kBigKeys keys, beyond that in global memory), a
// 4096-bit filter in front of the key search; candidates resolved in
// position order by one thread; the scan stops once every request of the
// row is satisfied.
constexpr int kBigItems = 8;
constexpr uint32_t kBigKeys = 2048;
constexpr uint32_t kFilterBits = 4096;

__device__ __forceinline__ uint32_t filter_hash(uint32_t x) { return (x * 0x9E3779B1u) >> 20; }  // 12 bits

struct OrderedSmem {
    uint32_t skey[kBigKeys];
    uint32_t scount[kBigKeys];
    uint32_t filter[kFilterBits / 32];
    uint8_t cand_bits[kTpbMut];
    uint8_t del_bits[kTpbMut];
    uint16_t cand_run[kTpbMut * kBigItems];
    uint32_t g_run[kTpbMut * kBigItems];
    uint32_t cand_warp[kTpbMut / 32];
    uint32_t left;
};

// One row by one block; returns the tombstones written (all threads call;
// `matched` of a group above kBigKeys must be zero).
__device__ __forceinline__ uint32_t block_tomb_ordered(const AdjView &view, const RowDesc &d, uint32_t u,
                                                       const unsigned long long *keys, uint32_t gs, uint32_t ge,
                                                       uint32_t *matched, OrderedSmem &sm) {
    const uint32_t tid = threadIdx.x;
    const uint32_t gm = ge - gs;
    const bool in_smem = gm <= kBigKeys;
    const unsigned long long uhi = static_cast<unsigned long long>(u) << kKeyShift;
    for (uint32_t i = tid; i < kFilterBits / 32; i += kTpbMut) sm.filter[i] = 0;
    if (tid == 0) sm.left = gm;
    __syncthreads();
    for (uint32_t j = tid; j < gm; j += kTpbMut) {
        const uint32_t x = key_low(keys[gs + j]);
        if (in_smem) {
            sm.skey[j] = x;
            sm.scount[j] = 0;
        }
        const uint32_t h = filter_hash(x);
        atomicOr(&sm.filter[h >> 5], 1u << (h & 31u));
    }
    __syncthreads();
    for (uint32_t base = 0; base < d.len; base += kTpbMut * kBigItems) {
        const uint32_t k0 = base + tid * kBigItems;
        uint32_t e[kBigItems];
#pragma unroll
        for (int h = 0; h < kBigItems; h += 4) {
            if (k0 + h < d.len) {
                const uint4 q = *reinterpret_cast<const uint4 *>(view.at(d.off + k0 + h));
                e[h] = q.x;
                e[h + 1] = q.y;
                e[h + 2] = q.z;
                e[h + 3] = q.w;
            } else {
                e[h] = e[h + 1] = e[h + 2] = e[h + 3] = kTomb;
            }
        }
        uint32_t cb = 0;
#pragma unroll
        for (int s = 0; s < kBigItems; ++s) {
            if (k0 + s >= d.len || e[s] == kTomb) continue;
            const uint32_t h = filter_hash(e[s]);
            if (!((sm.filter[h >> 5] >> (h & 31u)) & 1u)) continue;
            if (in_smem) {
                uint32_t lo = 0, hi = gm;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (sm.skey[mid] < e[s])
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                if (lo < gm && sm.skey[lo] == e[s]) {
                    cb |= 1u << s;
                    sm.cand_run[tid * kBigItems + s] = static_cast<uint16_t>(lo);
                }
            } else {
                uint32_t run, req;
                if (find_run(keys, gs, ge, uhi | e[s], run, req)) {
                    cb |= 1u << s;
                    sm.g_run[tid * kBigItems + s] = run;
                }
            }
        }
        sm.cand_bits[tid] = static_cast<uint8_t>(cb);
        sm.del_bits[tid] = 0;
        const uint32_t wmask = __ballot_sync(kFull, cb != 0);
        if ((tid & 31u) == 0) sm.cand_warp[tid >> 5] = wmask;
        if (__syncthreads_or(cb != 0)) {
            if (tid == 0) {
                // Visit only the threads that hold candidates, in position order.
                uint32_t l = sm.left;
                for (uint32_t wi = 0; wi < kTpbMut / 32; ++wi) {
                    for (uint32_t tm = sm.cand_warp[wi]; tm; tm &= tm - 1) {
                        const uint32_t t = wi * 32 + __ffs(tm) - 1;
                        uint32_t b = sm.cand_bits[t];
                        uint32_t dbits = 0;
                        while (b) {
                            const uint32_t s = __ffs(b) - 1;
                            b &= b - 1;
                            bool del;
                            if (in_smem) {
                                const uint32_t r = sm.cand_run[t * kBigItems + s];
                                uint32_t e2 = r + 1;
                                while (e2 < gm && sm.skey[e2] == sm.skey[r]) ++e2;
                                del = sm.scount[r] < e2 - r;
                                sm.scount[r] += 1;
                            } else {
                                const uint32_t r = sm.g_run[t * kBigItems + s];
                                uint32_t e2 = r + 1;
                                while (e2 < ge && keys[e2] == keys[r]) ++e2;
                                del = matched[r] < e2 - r;
                                matched[r] += 1;
                            }
                            if (del) {
                                dbits |= 1u << s;
                                --l;
                            }
                        }
                        sm.del_bits[t] = static_cast<uint8_t>(dbits);
                    }
                }
                sm.left = l;
            }
            __syncthreads();
            const uint32_t db = sm.del_bits[tid];
#pragma unroll
            for (int s = 0; s < kBigItems; ++s)
                if ((db >> s) & 1u) write_slot(view, d.off + k0 + s, kTomb);
        }
        __syncthreads();
        if (sm.left == 0) break;
    }
    return gm - sm.left;
}

__global__ void __launch_bounds__(kTpbMut)
    mutate_delete_big(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr, const uint32_t *big,
                      const uint32_t *big_count, uint32_t *matched, CompactList cl, unsigned long long *stats,
                      Status *st) {
    __shared__ OrderedSmem sm;
    const uint32_t nb = *big_count;
    for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const uint32_t gs = gr.start[big[b]];
        const uint32_t ge = gr.end[big[b]];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        const uint32_t done = block_tomb_ordered(view, d, u, keys, gs, ge, matched, sm);
        if (threadIdx.x == 0) {
            finish_row(desc, u, d, done, cl);
            if (done && stats) {
                atomicAdd(&stats[kCntRemoved], static_cast<unsigned long long>(done));
                atomicAdd(&stats[kCntChanged], 1ull);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- flat deletion
//
// When no destination is requested twice for the same source in a batch
// (every run has one key), the entry to tombstone for a key is simply the
// first live occurrence, i.e. the minimum matching position, which an
// atomicMin finds in any order.  Such rows are scanned in 512-entry warp
// chunks spread evenly over the whole grid (a hub row no longer serialises
// on one block); rows with repeated requests keep the position-ordered
// kernels above.
constexpr uint32_t kDelChunk = 512;
constexpr uint32_t kSmemKeys = 256;

// Classify groups: chunk count for flat rows, ordered list for the rest.
// `chunks` must be zero beyond the group count (it is scanned whole).
// Kinds of deletion groups: rows with repeated requests take the ordered
// kernels; rows with distinct requests the flat scan, or the position index
// when the row is indexed (posindex.cuh).
enum : uint8_t { kGroupOrdered = 0, kGroupChunked = 1, kGroupIndexed = 2 };

// Also clears the phase's per-key arrays (the scan chunk counts past the
// groups, the first-match positions, the ordered path's match counts) for
// the m keys, in place of three memsets.
__global__ void del_classify(const RowDesc *desc, const unsigned long long *keys, Groups gr, uint32_t *chunks,
                             uint8_t *gtype, uint32_t *ordered, uint32_t *ordered_count, PosIndex ix,
                             uint32_t *indexed, uint32_t *indexed_count, uint32_t m, uint32_t *firstpos,
                             uint32_t *matched) {
    const uint32_t ng = *gr.count;
    const uint32_t rounded = (ng + 31u) & ~31u;
    const uint32_t lane = lane_id();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        firstpos[i] = kInf;
        matched[i] = 0u;
        if (i >= ng) chunks[i] = 0u;
    }
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < rounded; g += gridDim.x * blockDim.x) {
        bool dup = false, by_index = false;
        uint32_t gs = 0, ge = 0;
        if (g < ng) {
            gs = gr.start[g];
            ge = gr.end[g];
            // Repeated requests are adjacent in the sorted keys; a lane checks
            // its own group when it is short, the warp checks long ones (hub
            // rows draw hundreds of deletions) together below.
            if (ge - gs <= 32u)
                for (uint32_t i = gs; i + 1 < ge && !dup; ++i) dup = keys[i] == keys[i + 1];
        }
        uint32_t longs = __ballot_sync(kFull, g < ng && ge - gs > 32u);
        while (longs) {
            const int l = __ffs(longs) - 1;
            longs &= longs - 1;
            const uint32_t ls = __shfl_sync(kFull, gs, l);
            const uint32_t le = __shfl_sync(kFull, ge, l);
            bool any = false;
            for (uint32_t i = ls + lane; i + 1 < le; i += 32u) any |= keys[i] == keys[i + 1];
            any = __any_sync(kFull, any);
            if (lane == static_cast<uint32_t>(l)) dup = any;
        }
        if (g < ng) {
            const uint32_t u = key_src(keys[gs]);
            by_index = !dup && idx_row(ix, u);
            gtype[g] = dup ? kGroupOrdered : by_index ? kGroupIndexed : kGroupChunked;
            chunks[g] = (dup || by_index) ? 0u : (desc[u].len + kDelChunk - 1) / kDelChunk;
        }
        warp_enqueue(dup, g, ordered, ordered_count, 0xFFFFFFFFu, nullptr);
        warp_enqueue(by_index, g, indexed, indexed_count, 0xFFFFFFFFu, nullptr);
    }
}

// Indexed rows with distinct requests: the first live position of every key
// from the index; the entry loses one occurrence and, when more remain, moves
// to the next one (a scan from the deleted position on, rare: parallel
// edges).  The tombstone is written here at once (the position is final),
// and the position is recorded with kApplied set so that del_apply skips
// it.  A warp deals the keys of its groups of up to kLaneKeys keys one per
// lane (del_index); larger groups get a warp each, and groups of more than
// kHugeKeys keys the whole grid (del_index_wide).
constexpr uint32_t kLaneKeys = 4;
constexpr uint32_t kHugeKeys = 256;
constexpr uint32_t kApplied = 0x80000000u;  // firstpos flag: tombstone already written

// One occurrence of v, found in slot s with entry e, is deleted: its
// tombstone, and the entry moves to the next occurrence or is dropped.
__device__ __forceinline__ uint32_t del_index_take(const AdjView &view, const RowDesc &d, uint32_t v,
                                                   unsigned long long s, const uint2 &e, const PosIndex &ix,
                                                   Status *st) {
    if (e.y == 0u || e.x >= d.len) {
        if (e.y != 0u) set_error(st, kErrInternal, 0x1d2u);
        return 0u;
    }
    write_slot(view, d.off + e.x, kTomb);
    if (e.y == 1u) {
        ix.val[s] = make_uint2(kInf, 0u);  // the key keeps its slot for the next time it is inserted
    } else {
        uint32_t q = e.x + 1;
        while (q < d.len && *view.at(d.off + q) != v) ++q;
        if (q >= d.len) set_error(st, kErrInternal, 0x1d3u);
        ix.val[s] = make_uint2(q < d.len ? q : kInf, e.y - 1u);
    }
    return 1u;
}

// Returns 1 when (u, v) was in the row; *pos is its position.
__device__ __forceinline__ uint32_t del_index_key(const AdjView &view, const RowDesc &d, uint32_t u, uint32_t v,
                                                  const PosIndex &ix, Status *st, uint32_t *pos = nullptr) {
    const unsigned long long s = idx_find(ix, (static_cast<unsigned long long>(u) << 32) | v);
    if (s == ~0ull) return 0u;  // not in the row: a missing delete
    const uint2 e = ix.val[s];
    if (!del_index_take(view, d, v, s, e, ix, st)) return 0u;
    if (pos) *pos = e.x | kApplied;
    return 1u;
}

// The keys of one lane, N at a time (live[j]: key j is served): the key,
// descriptor, first index probe and its value slot of every key are read
// before any of them is used, so the lane waits for one chain of dependent
// loads instead of N.  The first probe almost always decides (the tables
// stay at most half full); a collision continues with idx_find_from.
template <int N>
__device__ __forceinline__ uint32_t del_index_keys(const AdjView &view, RowDesc *desc,
                                                   const unsigned long long *keys, const uint32_t (&ks)[N],
                                                   const bool (&live)[N], uint32_t *firstpos, const PosIndex &ix,
                                                   Status *st) {
    unsigned long long key[N], slot[N], seen[N];
    RowDesc d[N];
    uint2 e[N];
#pragma unroll
    for (int j = 0; j < N; ++j) key[j] = live[j] ? keys[ks[j]] : 0ull;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t u = key_src(key[j]);
        if (live[j]) d[j] = desc[u];
        key[j] = (static_cast<unsigned long long>(u) << 32) | key_low(key[j]);
        slot[j] = idx_mix(key[j]) & ix.mask;
        seen[j] = kIdxEmpty + 0ull;
        if (live[j]) seen[j] = *reinterpret_cast<volatile unsigned long long *>(ix.keys + slot[j]);
        e[j] = live[j] ? ix.val[slot[j]] : make_uint2(0u, 0u);
    }
    uint32_t removed = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (!live[j]) continue;
        if (seen[j] != key[j]) {
            if (seen[j] == kIdxEmpty) continue;  // not in the row: a missing delete
            slot[j] = idx_find_from(ix, key[j], (slot[j] + 1) & ix.mask, 1);
            if (slot[j] == ~0ull) continue;
            e[j] = ix.val[slot[j]];
        }
        const uint32_t u = static_cast<uint32_t>(key[j] >> 32), v = static_cast<uint32_t>(key[j]);
        if (!del_index_take(view, d[j], v, slot[j], e[j], ix, st)) continue;
        firstpos[ks[j]] = e[j].x | kApplied;
        atomicAdd(&desc[u].meta, 1u << 6);
        ++removed;
    }
    return removed;
}

__global__ void __launch_bounds__(256, 4)
    del_index(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr,
                          const uint32_t *list, const uint32_t *count, uint32_t *firstpos, PosIndex ix,
                          uint32_t *wide, uint32_t *wide_count, uint32_t *huge, uint32_t *huge_count,
                          unsigned long long *stats, Status *st) {
    const uint32_t lane = lane_id();
    uint32_t removed = 0;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nl = *count;
    for (uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u; base < nl; base += warps * 32u) {
        const uint32_t i = base + lane;
        uint32_t g = 0, gs = 0, nk = 0;
        if (i < nl) {
            g = list[i];
            gs = gr.start[g];
            nk = gr.end[g] - gs;
        }
        // The warp's small groups (up to kLaneKeys keys) are concatenated (a
        // warp scan of their sizes) and their keys dealt one per lane, at
        // most kLaneKeys steps; distinct keys of a row are independent.
        const bool small_g = i < nl && nk <= kLaneKeys;
        const uint32_t mine = small_g ? nk : 0u;
        uint32_t incl = mine;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        const uint32_t excl = incl - mine;
        const uint32_t total = __shfl_sync(kFull, incl, 31);  // at most 32 * kLaneKeys
        uint32_t ks[kLaneKeys];
        bool live[kLaneKeys];
#pragma unroll
        for (int j = 0; j < static_cast<int>(kLaneKeys); ++j) {
            const uint32_t e = 32u * j + lane;
            ks[j] = 0;
            live[j] = false;
            if (32u * j < total) {  // warp-uniform
                uint32_t lo = 0, hi = 32;  // the last lane whose keys start at or before e
#pragma unroll
                for (int step = 0; step < 5; ++step) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (__shfl_sync(kFull, excl, mid) <= e)
                        lo = mid;
                    else
                        hi = mid;
                }
                ks[j] = __shfl_sync(kFull, gs, lo) + (e - __shfl_sync(kFull, excl, lo));
                live[j] = e < total;
            }
        }
        removed += del_index_keys<kLaneKeys>(view, desc, keys, ks, live, firstpos, ix, st);
        // Larger groups go to del_index_wide: up to kHugeKeys keys one warp
        // per group, more (hub rows, where uniform deletions over the edges
        // concentrate) across the whole grid in 32-key chunks.
        warp_enqueue(i < nl && nk > kLaneKeys && nk <= kHugeKeys, g, wide, wide_count, nl, st);
        warp_enqueue(i < nl && nk > kHugeKeys, g, huge, huge_count, nl, st);
    }
    if (stats) warp_count(&stats[kCntRemoved], removed);
}

__global__ void del_index_wide(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr,
                               const uint32_t *wide, const uint32_t *wide_count, const uint32_t *huge,
                               const uint32_t *huge_count, uint32_t *firstpos, PosIndex ix,
                               unsigned long long *stats, Status *st) {
    const uint32_t lane = lane_id();
    uint32_t removed = 0;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = *wide_count;
    for (uint32_t i = wid; i < nw; i += warps) {
        const uint32_t g = wide[i];
        const uint32_t gs = gr.start[g];
        const uint32_t nk = gr.end[g] - gs;
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        uint32_t tombs = 0;
        for (uint32_t j = lane; j < nk; j += 32u)
            tombs += del_index_key(view, d, u, key_low(keys[gs + j]), ix, st, firstpos + gs + j);
        tombs = __reduce_add_sync(kFull, tombs);
        if (lane == 0 && tombs) atomicAdd(&desc[u].meta, tombs << 6);
        removed += lane == 0 ? tombs : 0u;
    }
    // Huge groups: chunk c of the concatenated 32-key chunks goes to warp
    // c mod warps; every warp walks the (short) list in the same order.
    const uint32_t nh = *huge_count;
    uint64_t prefix = 0;
    for (uint32_t h = 0; h < nh; ++h) {
        const uint32_t g = huge[h];
        const uint32_t gs = gr.start[g];
        const uint32_t nk = gr.end[g] - gs;
        const uint64_t chunks = (nk + 31u) / 32u;
        uint64_t c = prefix + (wid + warps - static_cast<uint32_t>(prefix % warps)) % warps;
        if (c < prefix + chunks) {
            const uint32_t u = key_src(keys[gs]);
            const RowDesc d = desc[u];
            uint32_t tombs = 0;
            for (; c < prefix + chunks; c += warps) {
                const uint32_t j = static_cast<uint32_t>(c - prefix) * 32u + lane;
                if (j < nk)
                    tombs += del_index_key(view, d, u, key_low(keys[gs + j]), ix, st, firstpos + gs + j);
            }
            tombs = __reduce_add_sync(kFull, tombs);
            if (lane == 0 && tombs) atomicAdd(&desc[u].meta, tombs << 6);
            removed += lane == 0 ? tombs : 0u;
        }
        prefix += chunks;
    }
    if (stats) warp_count(&stats[kCntRemoved], removed);
}

// After the ordered kernels: the entries of every key of an ordered group on
// an indexed row are recounted from the row (rare: repeated requests).
__global__ void idx_fix_ordered(AdjView view, const RowDesc *desc, const unsigned long long *keys, Groups gr,
                                const uint32_t *ordered, const uint32_t *ordered_count, PosIndex ix, Status *st) {
    const uint32_t no = *ordered_count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < no; i += gridDim.x * blockDim.x) {
        const uint32_t g = ordered[i];
        const uint32_t gs = gr.start[g];
        const uint32_t ge = gr.end[g];
        const uint32_t u = key_src(keys[gs]);
        if (!idx_row(ix, u)) continue;
        const RowDesc d = desc[u];
        for (uint32_t j = gs; j < ge; ++j) {
            if (j > gs && keys[j] == keys[j - 1]) continue;  // one pass per distinct key
            const uint32_t v = key_low(keys[j]);
            const unsigned long long s = idx_find(ix, (static_cast<unsigned long long>(u) << 32) | v);
            if (s == ~0ull) continue;
            uint32_t first = kInf, live = 0;
            for (uint32_t q = 0; q < d.len; ++q)
                if (*view.at(d.off + q) == v) {
                    if (first == kInf) first = q;
                    ++live;
                }
            ix.val[s] = make_uint2(first, live);
        }
    }
}

// Chunk runs are dealt round-robin to the warps: run r (kDelRun consecutive
// 512-entry chunks) goes to warp r mod warps, so the chunks of one long row
// spread over the whole grid while a warp still reuses a row's keys for a
// few chunks.  `chunk_map[c]` is the group of chunk c (del_chunk_map);
// `chunk_end` is the inclusive prefix sum of `chunks` over scan_n entries.
// Each chunk records the first live match of every key (atomicMin).
//
// Membership test per row entry, by the row's number of requests: up to
// kDelCmpKeys, compare against the keys held in lanes (about 9 instructions
// per request per 4 entries, no divergence); beyond, a per-warp bit filter in
// shared memory (32 bits per request rounded up to a power of two,
// 1024..16384 bits, one multiplicative hash) built once per group, and a
// binary search on a filter hit.  (Filters for rows of 3..8 requests, in
// shared memory or in a 64-bit register, measured 40-50 % slower on the
// whole scan: their hits diverge inside the warp.)
constexpr uint32_t kDelCmpKeys = 8;
constexpr uint32_t kDelFilterWords = 512;

__device__ __forceinline__ uint32_t del_hash(uint32_t y, uint32_t shift) { return (y * 2654435761u) >> shift; }

constexpr uint32_t kDelRun = 4;

// chunk_map[c] = group of chunk c; one warp per group, lanes over its chunks.
__global__ void del_chunk_map(Groups gr, const uint32_t *chunk_end, uint32_t *chunk_map) {
    const uint32_t ng = *gr.count;
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ng; g += warps) {
        const uint32_t c0 = g ? chunk_end[g - 1] : 0u, c1 = chunk_end[g];
        for (uint32_t c = c0 + lane; c < c1; c += 32u) chunk_map[c] = g;
    }
}

// The chunks [0, total) of a scan; chunk c belongs to group map[c], whose first
// chunk is base(g).  kMutWarps warps per block; `sk` and `filt` are the warp's
// shared memory.
template <class B>
__device__ __forceinline__ void del_scan_chunks(const AdjView &view, const RowDesc *desc,
                                                const unsigned long long *keys, const Groups &gr, const B &base,
                                                const uint32_t *chunk_map, uint32_t total, uint32_t *firstpos,
                                                uint32_t *sk, uint32_t *filt, unsigned long long *stats,
                                                uint32_t *seg_hot) {
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t g_ready = ~0u;  // group whose keys are loaded in kd / filt / sk
    uint32_t gs = 0, ge = 0, nk = 0, kd = 0, fshift = 18;
    RowDesc d{};
    unsigned long long uhi = 0;
    uint32_t scanned = 0, scanned_cached = 0;
    for (uint32_t c = wid * kDelRun; c < total; c += (c % kDelRun == kDelRun - 1) ? (warps - 1) * kDelRun + 1 : 1) {
        const uint32_t g = chunk_map[c];
        if (g != g_ready) {
            __syncwarp();
            g_ready = g;
            gs = gr.start[g];
            ge = gr.end[g];
            nk = ge - gs;
            const uint32_t u = key_src(keys[gs]);
            d = desc[u];
            uhi = static_cast<unsigned long long>(u) << kKeyShift;
            kd = lane < nk ? key_low(keys[gs + lane]) : 0u;
            if (nk > kDelCmpKeys) {
                // words = nk rounded up to a power of two in [32, 512]
                const uint32_t words = min(kDelFilterWords, max(32u, 1u << (32 - __clz(nk - 1))));
                fshift = 32u - (5u + (31u - __clz(words)));  // hash -> log2(32 * words) bits
                for (uint32_t j = lane; j < words; j += 32u) filt[j] = 0u;
                __syncwarp();
                for (uint32_t j = lane; j < nk; j += 32u) {
                    const uint32_t y = key_low(keys[gs + j]);
                    const uint32_t h = del_hash(y, fshift);
                    atomicOr(filt + (h >> 5), 1u << (h & 31u));
                    if (nk <= kSmemKeys) sk[j] = y;
                }
            }
            __syncwarp();
        }
        const uint32_t k0 = (c - base(g)) * kDelChunk;
        // A 512-entry chunk never straddles a segment (segments hold 2^14).
        const uint32_t *src = view.at(d.off + k0);
        const uint32_t len_here = min(kDelChunk, d.len - k0);
        scanned += len_here;
        if (view.cached(d.off + k0)) scanned_cached += len_here;
        if (seg_hot && lane == 0) atomicAdd(seg_hot + ((d.off + k0) >> kSegShift), len_here);
        // Short rows (most groups) end after one or two 128-entry steps.
        const uint32_t steps = (len_here + 127u) / 128u;
        uint4 q[kDelChunk / 128u];
#pragma unroll
        for (uint32_t s = 0; s < kDelChunk / 128u; ++s) {
            const uint32_t kk = k0 + 128u * s + 4u * lane;
            q[s] = (s < steps && kk < d.len) ? *reinterpret_cast<const uint4 *>(src + 128u * s + 4u * lane)
                                             : make_uint4(kTomb, kTomb, kTomb, kTomb);
        }
#pragma unroll
        for (uint32_t s = 0; s < kDelChunk / 128u; ++s) {
            if (s >= steps) continue;  // warp-uniform; keeps the loop unrolled (q[] in registers)
            const uint32_t kk = k0 + 128u * s + 4u * lane;
            uint32_t e[4] = {q[s].x, q[s].y, q[s].z, q[s].w};
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (kk + t >= d.len) e[t] = kTomb;
            if (nk <= kDelCmpKeys) {
                int hit[4] = {-1, -1, -1, -1};
                for (uint32_t j = 0; j < nk; ++j) {
                    const uint32_t kj = __shfl_sync(kFull, kd, j);
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (e[t] == kj) hit[t] = static_cast<int>(j);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (hit[t] >= 0 && e[t] != kTomb) atomicMin(firstpos + gs + hit[t], kk + t);
            } else {
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (e[t] == kTomb) continue;
                    const uint32_t h = del_hash(e[t], fshift);
                    if (!((filt[h >> 5] >> (h & 31u)) & 1u)) continue;
                    int hit = -1;
                    if (nk <= kSmemKeys) {
                        uint32_t a = 0, b = nk;
                        while (a < b) {
                            const uint32_t mid = (a + b) >> 1;
                            if (sk[mid] < e[t])
                                a = mid + 1;
                            else
                                b = mid;
                        }
                        if (a < nk && sk[a] == e[t]) hit = static_cast<int>(a);
                    } else {
                        uint32_t run, req;
                        if (find_run(keys, gs, ge, uhi | e[t], run, req)) hit = static_cast<int>(run - gs);
                    }
                    if (hit >= 0) atomicMin(firstpos + gs + hit, kk + t);
                }
            }
        }
    }
    if (stats) {
        // lane 0 of every warp holds the warp's totals (all lanes counted the same chunks)
        if (lane == 0 && scanned) atomicAdd(&stats[kCntDelScanned], static_cast<unsigned long long>(scanned));
        if (lane == 0 && scanned_cached)
            atomicAdd(&stats[kCntDelScannedCached], static_cast<unsigned long long>(scanned_cached));
    }
}

__global__ void __launch_bounds__(kMutWarps * 32)
    del_scan(AdjView view, const RowDesc *desc, const unsigned long long *keys, Groups gr, const uint32_t *chunk_end,
             const uint32_t *chunk_map, uint32_t scan_n, uint32_t *firstpos, unsigned long long *stats,
             uint32_t *seg_hot) {
    __shared__ uint32_t skeys[kMutWarps][kSmemKeys];
    __shared__ uint32_t sfilt[kMutWarps][kDelFilterWords];
    const uint32_t warp = threadIdx.x >> 5;
    del_scan_chunks(view, desc, keys, gr, [&](uint32_t g) { return g ? chunk_end[g - 1] : 0u; }, chunk_map,
                    scan_n ? chunk_end[scan_n - 1] : 0u, firstpos, skeys[warp], sfilt[warp], stats, seg_hot);
}

// Tombstone the first match of every key found by del_scan.
__global__ void del_apply(AdjView view, RowDesc *desc, const unsigned long long *keys, uint32_t m,
                          const uint32_t *firstpos, unsigned long long *stats) {
    uint32_t removed = 0;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t rounded = (m + 31u) & ~31u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rounded; i += stride) {
        if (i < m) {
            const uint32_t p = firstpos[i];
            if (p != kInf && !(p & kApplied)) {
                const uint32_t u = key_src(keys[i]);
                write_slot(view, desc[u].off + p, kTomb);
                atomicAdd(&desc[u].meta, 1u << 6);
                ++removed;
            }
        }
    }
    if (stats) warp_count(&stats[kCntRemoved], removed);
}

// Queue flat rows whose tombstones reached a quarter of their length.
__global__ void del_finish(const RowDesc *desc, const unsigned long long *keys, Groups gr, const uint8_t *gtype,
                           const uint32_t *firstpos, CompactList cl, unsigned long long *stats) {
    const uint32_t ng = *gr.count;
    const uint32_t rounded = (ng + 31u) & ~31u;
    uint32_t changed = 0;
    // Warp-aggregated appends and counts: ~10^5 rows per batch would
    // otherwise queue on one counter address.
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < rounded; g += gridDim.x * blockDim.x) {
        bool want = false, big = false;
        uint32_t u = 0;
        if (g < ng && gtype[g] != kGroupOrdered) {  // flat group (scanned or indexed)
            const uint32_t gs = gr.start[g];
            const uint32_t ge = gr.end[g];
            bool any = false;
            for (uint32_t i = gs; i < ge && !any; ++i) any = firstpos[i] != kInf;
            if (any) {
                ++changed;
                u = key_src(keys[gs]);
                const RowDesc d = desc[u];
                const uint32_t tombs = rd_tombs(d);
                want = 4ull * tombs >= d.len || tombs >= kMaxTombs / 2;
                big = want && d.len > kWarpMove;
                want = want && !big;
            }
        }
        warp_enqueue(want, u, cl.rows, cl.count, 0xFFFFFFFFu, nullptr);
        if (big) cl.rows[cl.cap - 1u - atomicAdd(cl.big_count, 1u)] = u;
    }
    if (stats) warp_count(&stats[kCntChanged], changed);
}

// ---------------------------------------------------------------- moving survivors
// The live entries of a row of `len` slots at `src_off` move, in order, to the
// front of the block at `dst_off` (the same block: compaction in place), and
// the position index follows (idx_move_n) where an entry's position changes.
// Return the number of survivors.
//
// One warp, rows inside one segment: 256 entries per step, the row loads of
// the next step in flight while this step is scanned, stored and indexed (in
// place, this step's stores lie below the next step's loads).
__device__ __forceinline__ uint32_t warp_move_live(const AdjView &view, const PosIndex &ix, uint32_t u,
                                                   uint64_t src_off, uint32_t len, uint64_t dst_off, Status *st) {
    if (!len) return 0u;
    const uint32_t lane = lane_id();
    const uint4 tomb4 = make_uint4(kTomb, kTomb, kTomb, kTomb);
    const uint32_t *src = view.at(src_off);
    uint32_t *dst = view.wptr(dst_off);
    const bool indexed = idx_row(ix, u);
    uint32_t w = 0;
    uint4 next[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t k = 128u * h + 4u * lane;
        next[h] = k < len ? *reinterpret_cast<const uint4 *>(src + k) : tomb4;
    }
    for (uint32_t b0 = 0; b0 < len; b0 += 256u) {
        uint4 cur[2] = {next[0], next[1]};
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t k = b0 + 256u + 128u * h + 4u * lane;
            next[h] = k < len ? *reinterpret_cast<const uint4 *>(src + k) : tomb4;
        }
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t k = b0 + 128u * h + 4u * lane;
            const uint32_t v[4] = {cur[h].x, cur[h].y, cur[h].z, cur[h].w};
            bool live[4];
            uint32_t c = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                live[j] = k + j < len && v[j] != kTomb;
                c += live[j] ? 1u : 0u;
            }
            uint32_t incl = c;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += t;
            }
            uint32_t pos = w + incl - c;
            uint32_t p[4], q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                p[j] = k + j;
                q[j] = pos;
                if (live[j]) {
                    dst[pos++] = v[j];
                    live[j] = p[j] != q[j];
                }
            }
            if (indexed) idx_move_n<4>(ix, u, v, p, q, live, st);
            w += __shfl_sync(kFull, incl, 31);
        }
    }
    __syncwarp();
    return w;
}

// One block, rows of any length: tiles of kTpbMut x 8 slots, block scan,
// survivors staged in shared memory and stored with coalesced writes.
struct MoveSmem {
    typename cub::BlockScan<uint32_t, kTpbMut>::TempStorage scan;
    uint32_t stage[kTpbMut * kBigItems];
};

__device__ __forceinline__ uint32_t block_move_live(const AdjView &view, const PosIndex &ix, uint32_t u,
                                                    uint64_t src_off, uint32_t len, uint64_t dst_off, MoveSmem &sm,
                                                    Status *st) {
    using BlockScan = cub::BlockScan<uint32_t, kTpbMut>;
    const uint32_t tid = threadIdx.x;
    const bool indexed = idx_row(ix, u);
    uint32_t w = 0;
    for (uint32_t base = 0; base < len; base += kTpbMut * kBigItems) {
        const uint32_t k0 = base + tid * kBigItems;
        uint32_t e[kBigItems];
#pragma unroll
        for (int h = 0; h < kBigItems; h += 4) {
            if (k0 + h < len) {
                const uint4 q = *reinterpret_cast<const uint4 *>(view.at(src_off + k0 + h));
                e[h] = q.x;
                e[h + 1] = q.y;
                e[h + 2] = q.z;
                e[h + 3] = q.w;
            } else {
                e[h] = e[h + 1] = e[h + 2] = e[h + 3] = kTomb;
            }
        }
        uint32_t kc = 0;
#pragma unroll
        for (int s = 0; s < kBigItems; ++s) {
            if (k0 + s >= len) e[s] = kTomb;
            kc += e[s] != kTomb ? 1u : 0u;
        }
        uint32_t prefix, total;
        BlockScan(sm.scan).ExclusiveSum(kc, prefix, total);
        uint32_t pos = prefix;
        uint32_t q[kBigItems];
#pragma unroll
        for (int s = 0; s < kBigItems; ++s) {
            q[s] = w + pos;
            if (e[s] != kTomb) sm.stage[pos++] = e[s];
        }
        __syncthreads();  // every load of this tile is done before any store
        const uint32_t tile = min(static_cast<uint32_t>(kTpbMut * kBigItems), len - base);
        if (src_off != dst_off || w != base || total != tile) {
            for (uint32_t i = tid; i < total; i += kTpbMut) write_slot(view, dst_off + w + i, sm.stage[i]);
            if (indexed) {
#pragma unroll
                for (int h = 0; h < kBigItems; h += 4) {
                    const uint32_t v4[4] = {e[h], e[h + 1], e[h + 2], e[h + 3]};
                    const uint32_t p4[4] = {k0 + h, k0 + h + 1, k0 + h + 2, k0 + h + 3};
                    const uint32_t q4[4] = {q[h], q[h + 1], q[h + 2], q[h + 3]};
                    bool moved[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) moved[j] = v4[j] != kTomb && p4[j] != q4[j];
                    idx_move_n<4>(ix, u, v4, p4, q4, moved, st);
                }
            }
        }
        w += total;
        __syncthreads();
    }
    return w;
}

// ---------------------------------------------------------------- compaction

// Drop the tombstones of the queued rows in place (order kept): a warp per
// row of up to kWarpMove slots (nearly all of them: a row of four entries
// compacts at its first deletion), a block per longer row.  A block for
// every row left 255 of 256 threads idle on the short ones.
__device__ __forceinline__ void compact_listed(const AdjView &view, RowDesc *desc, const CompactList &cl,
                                               const PosIndex &ix, MoveSmem &sm, Status *st) {
    const uint32_t nb = *cl.big_count;
    for (uint32_t c = blockIdx.x; c < nb; c += gridDim.x) {
        const uint32_t u = cl.rows[cl.cap - 1u - c];
        const RowDesc d = desc[u];
        const uint32_t w = block_move_live(view, ix, u, d.off, d.len, d.off, sm, st);
        if (threadIdx.x == 0) desc[u] = RowDesc{d.off, w, rd_meta(rd_cls(d), 0)};
        __syncthreads();
    }
    const uint32_t nc = *cl.count;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < nc; c += warps) {
        const uint32_t u = cl.rows[c];
        const RowDesc d = desc[u];
        const uint32_t w = warp_move_live(view, ix, u, d.off, d.len, d.off, st);
        if (lane_id() == 0) desc[u] = RowDesc{d.off, w, rd_meta(rd_cls(d), 0)};
    }
}

__global__ void __launch_bounds__(kTpbMut) compact_rows(AdjView view, RowDesc *desc, CompactList cl, PosIndex ix,
                                                         Status *st) {
    __shared__ MoveSmem sm;
    compact_listed(view, desc, cl, ix, sm, st);
}

// ---------------------------------------------------------------- indexed deletion
// Deletion phase of an arena whose position index covers every row above
// kIdxCls at its last build: three kernels in a chain.  (The flat scan of an
// unindexed arena takes thirteen; on small batches their launches were most
// of the phase.)
//   del_lane: a lane per group.  Indexed rows take the positions of up to
//     kLaneKeys distinct keys from the index; rows of up to kLaneDelRow slots
//     are read into registers, lose the requested entries and are written
//     back without tombstones.  The rest is listed for
//   del_wide: a warp per group: more keys on an indexed row (hub groups of
//     more than kHugeKeys: the whole grid), repeated requests, and unindexed
//     rows (ones that grew since the build) of up to kWarpRowMax slots, in
//     position order; the warp compacts its row when it is due.  Longer
//     unindexed rows are scanned by the whole grid in chunks, as by del_scan (a
//     block per row, in position order: 3.3 ms for 2,000 deletions from a row
//     grown to 900,000 entries, 21.5 ms for 20,000).
//   del_rest: the tombstones of those rows, a block per long row with repeated
//     requests, then the queued compactions.
constexpr uint32_t kLaneDelRow = 16;

// Work lists of the phase (each as long as the arena's groups).
struct DelLists {
    uint32_t *wide;
    uint32_t *wide_count;
    uint32_t *huge;
    uint32_t *huge_count;
    uint32_t *big;
    uint32_t *big_count;
    // Long unindexed rows with distinct requests: their groups, and the chunks
    // of the scan (group per chunk; a group's first chunk in `first`).
    uint32_t *scan;
    uint32_t *scan_count;
    uint32_t *chunk_map;
    uint32_t *chunk_count;
    uint32_t *first;
    uint32_t *firstpos;  // per key: position of its first live occurrence
};

__device__ __forceinline__ bool warp_has_repeats(const unsigned long long *keys, uint32_t gs, uint32_t ge) {
    bool any = false;
    for (uint32_t i = gs + lane_id(); i + 1 < ge; i += 32u) any |= keys[i] == keys[i + 1];
    return __any_sync(kFull, any);
}

__global__ void __launch_bounds__(256, 4)
    del_lane(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr, PosIndex ix, DelLists dl,
             CompactList cl, uint32_t *matched, uint32_t *seg_hot, unsigned long long *stats, unsigned long long *scan_stats, Status *st) {
    const uint32_t ng = *gr.count;
    const uint32_t rounded = (ng + 31u) & ~31u;
    uint32_t removed = 0, changed = 0, scanned = 0, scanned_cached = 0;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < rounded; g += gridDim.x * blockDim.x) {
        bool wide = false, huge = false, compact = false, compact_big = false, scan = false;
        uint32_t u = 0, gs = 0, nk = 0, row_len = 0;
        if (g < ng) {
            gs = gr.start[g];
            nk = gr.end[g] - gs;
            uint32_t v[kLaneKeys];
            bool dup = false;
#pragma unroll
            for (uint32_t j = 0; j < kLaneKeys; ++j) {
                const unsigned long long k = j < nk ? keys[gs + j] : 0ull;
                if (j == 0) u = key_src(k);
                v[j] = key_low(k);
                if (j && j < nk) dup |= v[j] == v[j - 1];
            }
            const RowDesc d = desc[u];
            const bool indexed = idx_row(ix, u);
            if (nk > kLaneKeys || (indexed ? dup : d.len > kLaneDelRow)) {
                huge = indexed && nk > kHugeKeys;  // del_wide looks for repeated requests before it uses the index
                scan = !indexed && d.len > kWarpRowMax;
                wide = !huge && !scan;
                row_len = d.len;
                if (huge) matched[gs] = rd_tombs(d);  // for del_rest: did the row lose any
            } else if (indexed) {
                unsigned long long slot[kLaneKeys], seen[kLaneKeys];
                uint2 e[kLaneKeys];
#pragma unroll
                for (uint32_t j = 0; j < kLaneKeys; ++j) {
                    const unsigned long long key = (static_cast<unsigned long long>(u) << 32) | v[j];
                    slot[j] = idx_mix(key) & ix.mask;
                    seen[j] = kIdxEmpty;
                    if (j < nk) {
                        seen[j] = *reinterpret_cast<volatile unsigned long long *>(ix.keys + slot[j]);
                        e[j] = ix.val[slot[j]];
                    }
                }
                uint32_t tombs = 0;
#pragma unroll
                for (uint32_t j = 0; j < kLaneKeys; ++j) {
                    if (j >= nk) continue;
                    const unsigned long long key = (static_cast<unsigned long long>(u) << 32) | v[j];
                    if (seen[j] != key) {
                        if (seen[j] == kIdxEmpty) continue;  // not in the row: a missing delete
                        slot[j] = idx_find_from(ix, key, (slot[j] + 1) & ix.mask, 1);
                        if (slot[j] == ~0ull) continue;
                        e[j] = ix.val[slot[j]];
                    }
                    tombs += del_index_take(view, d, v[j], slot[j], e[j], ix, st);
                }
                if (tombs) {
                    const uint32_t t = rd_tombs(d) + tombs;
                    desc[u].meta = rd_meta(rd_cls(d), t);
                    compact = 4ull * t >= d.len || t >= kMaxTombs / 2;
                    compact_big = compact && d.len > kWarpMove;
                    compact = compact && !compact_big;
                    removed += tombs;
                    ++changed;
                }
            } else if (d.len) {
                // A block of at most one segment.
                uint32_t e[kLaneDelRow];
                const uint32_t *src = view.at(d.off);
#pragma unroll
                for (uint32_t h = 0; h < kLaneDelRow; h += 4) {
                    uint4 q = make_uint4(kTomb, kTomb, kTomb, kTomb);
                    if (h < d.len) q = *reinterpret_cast<const uint4 *>(src + h);
                    e[h] = h < d.len ? q.x : kTomb;
                    e[h + 1] = h + 1 < d.len ? q.y : kTomb;
                    e[h + 2] = h + 2 < d.len ? q.z : kTomb;
                    e[h + 3] = h + 3 < d.len ? q.w : kTomb;
                }
                scanned += d.len;
                if (view.cached(d.off)) scanned_cached += d.len;
                seg_touch(seg_hot, d.off, d.len);
                // Each request takes the first live occurrence; a repeated
                // one the next.
                uint32_t gone = 0;
#pragma unroll
                for (uint32_t j = 0; j < kLaneKeys; ++j) {
                    bool open = j < nk;
#pragma unroll
                    for (uint32_t k = 0; k < kLaneDelRow; ++k)
                        if (open && e[k] == v[j] && v[j] != kTomb) {
                            e[k] = kTomb;
                            open = false;
                            ++gone;
                        }
                }
                if (gone) {
                    uint32_t *wp = view.wptr(d.off);
                    uint32_t w = 0;
#pragma unroll
                    for (uint32_t k = 0; k < kLaneDelRow; ++k)
                        if (e[k] != kTomb) {
                            if (w != k) wp[w] = e[k];
                            ++w;
                        }
                    desc[u] = RowDesc{d.off, w, rd_meta(rd_cls(d), 0)};
                    removed += gone;
                    ++changed;
                }
            }
        }
        // Rows that grew past kWarpRowMax since the index was built: chunks for
        // the whole grid, or, with repeated requests, a block.
        uint32_t scans = __ballot_sync(kFull, scan);
        while (scans) {
            const uint32_t l = __ffs(scans) - 1;
            scans &= scans - 1;
            const uint32_t lg = __shfl_sync(kFull, g, l), ls = __shfl_sync(kFull, gs, l);
            const uint32_t le = ls + __shfl_sync(kFull, nk, l);
            const uint32_t chunks = (__shfl_sync(kFull, row_len, l) + kDelChunk - 1) / kDelChunk;
            const bool rep = warp_has_repeats(keys, ls, le);
            uint32_t at = 0;
            if (lane_id() == 0) {
                if (rep) {
                    dl.big[atomicAdd(dl.big_count, 1u)] = lg;
                } else {
                    at = atomicAdd(dl.chunk_count, chunks);
                    dl.first[lg] = at;
                    dl.scan[atomicAdd(dl.scan_count, 1u)] = lg;
                }
            }
            if (rep) continue;
            at = __shfl_sync(kFull, at, 0);
            for (uint32_t i = lane_id(); i < chunks; i += 32u) dl.chunk_map[at + i] = lg;
            for (uint32_t i = ls + lane_id(); i < le; i += 32u) dl.firstpos[i] = kInf;
        }
        warp_enqueue(wide, g, dl.wide, dl.wide_count, ng, st);
        warp_enqueue(huge, g, dl.huge, dl.huge_count, ng, st);
        warp_enqueue(compact, u, cl.rows, cl.count, cl.cap, st);
        if (compact_big) cl.rows[cl.cap - 1u - atomicAdd(cl.big_count, 1u)] = u;
    }
    if (stats) {
        warp_count(&stats[kCntRemoved], removed);
        warp_count(&stats[kCntChanged], changed);
    }
    warp_count(&scan_stats[kCntDelScanned], scanned);
    warp_count(&scan_stats[kCntDelScannedCached], scanned_cached);
}

// The index entries of an ordered group (repeated requests on an indexed row)
// recounted from the row; thread `t` of `stride`.
__device__ __forceinline__ void idx_recount_group(const AdjView &view, const RowDesc &d, uint32_t u,
                                                  const unsigned long long *keys, uint32_t gs, uint32_t ge,
                                                  uint32_t t, uint32_t stride, const PosIndex &ix) {
    for (uint32_t j = gs + t; j < ge; j += stride) {
        if (j > gs && keys[j] == keys[j - 1]) continue;  // one pass per distinct key
        const uint32_t v = key_low(keys[j]);
        const unsigned long long s = idx_find(ix, (static_cast<unsigned long long>(u) << 32) | v);
        if (s == ~0ull) continue;
        uint32_t first = kInf, live = 0;
        for (uint32_t q = 0; q < d.len; ++q)
            if (*view.at(d.off + q) == v) {
                if (first == kInf) first = q;
                ++live;
            }
        ix.val[s] = make_uint2(first, live);
    }
}

// Out of line: inlined, the scan would take registers from all of del_wide.
__device__ __noinline__ void del_wide_scan(AdjView view, const RowDesc *desc, const unsigned long long *keys,
                                           Groups gr, DelLists dl, uint32_t *sk, uint32_t *filt,
                                           unsigned long long *stats, uint32_t *seg_hot) {
    del_scan_chunks(view, desc, keys, gr, [&](uint32_t g) { return dl.first[g]; }, dl.chunk_map, *dl.chunk_count,
                    dl.firstpos, sk, filt, stats, seg_hot);
}

__global__ void __launch_bounds__(kMutWarps * 32, 3)
    del_wide(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr, PosIndex ix, DelLists dl,
             CompactList cl, uint32_t *matched, uint32_t *seg_hot, unsigned long long *stats,
             unsigned long long *scan_stats, Status *st) {
    __shared__ uint32_t skeys[kMutWarps][kSmemKeys];
    __shared__ uint32_t sfilt[kMutWarps][kDelFilterWords];
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (*dl.chunk_count)
        del_wide_scan(view, desc, keys, gr, dl, skeys[threadIdx.x >> 5], sfilt[threadIdx.x >> 5], scan_stats, seg_hot);
    uint32_t removed = 0, changed = 0, scanned = 0, scanned_cached = 0;  // lane 0 counts
    const uint32_t nw = *dl.wide_count;
    for (uint32_t i = wid; i < nw; i += warps) {
        const uint32_t g = dl.wide[i];
        const uint32_t gs = gr.start[g], ge = gr.end[g];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        const bool indexed = idx_row(ix, u);
        uint32_t tombs = 0;
        if (indexed && !warp_has_repeats(keys, gs, ge)) {
            for (uint32_t j = gs + lane; j < ge; j += 32u)
                tombs += del_index_key(view, d, u, key_low(keys[j]), ix, st);
            tombs = __reduce_add_sync(kFull, tombs);
        } else if (d.len > kWarpRowMax) {
            if (lane == 0) dl.big[atomicAdd(dl.big_count, 1u)] = g;
            continue;
        } else if (d.len) {
            if (ge - gs <= 32u) {
                tombs = warp_tomb_regs(view, d, keys, gs, ge - gs);
            } else {
                for (uint32_t j = gs + lane; j < ge; j += 32u) matched[j] = 0u;
                __syncwarp();
                tombs = warp_tomb_global(view, d, u, keys, gs, ge, matched);
            }
            __syncwarp();
            if (lane == 0) {
                scanned += d.len;
                if (view.cached(d.off)) scanned_cached += d.len;
                seg_touch(seg_hot, d.off, d.len);
            }
            if (indexed) {
                idx_recount_group(view, d, u, keys, gs, ge, lane, 32u, ix);
                __syncwarp();
            }
        }
        if (!tombs) continue;
        const uint32_t t = rd_tombs(d) + tombs;
        const bool compact = 4ull * t >= d.len || t >= kMaxTombs / 2;
        if (compact && d.len <= kWarpMove) {
            __syncwarp();
            const uint32_t w = warp_move_live(view, ix, u, d.off, d.len, d.off, st);
            if (lane == 0) desc[u] = RowDesc{d.off, w, rd_meta(rd_cls(d), 0)};
        } else if (lane == 0) {
            desc[u].meta = rd_meta(rd_cls(d), t);
            if (compact) cl.rows[cl.cap - 1u - atomicAdd(cl.big_count, 1u)] = u;
        }
        if (lane == 0) {
            removed += tombs;
            ++changed;
        }
    }
    // Hub groups: chunk c of their concatenated 32-key chunks goes to warp c
    // mod warps; every warp walks the (short) list in the same order.  A
    // group with repeated requests goes to the block path whole.
    const uint32_t nh = *dl.huge_count;
    uint64_t prefix = 0;
    for (uint32_t h = 0; h < nh; ++h) {
        const uint32_t g = dl.huge[h];
        const uint32_t gs = gr.start[g], ge = gr.end[g];
        if (warp_has_repeats(keys, gs, ge)) {
            if (wid == 0 && lane == 0) dl.big[atomicAdd(dl.big_count, 1u)] = g;
            continue;
        }
        const uint32_t nk = ge - gs;
        const uint64_t chunks = (nk + 31u) / 32u;
        uint64_t c = prefix + (wid + warps - static_cast<uint32_t>(prefix % warps)) % warps;
        if (c < prefix + chunks) {
            const uint32_t u = key_src(keys[gs]);
            const RowDesc d = desc[u];  // only `meta` changes meanwhile
            uint32_t tombs = 0;
            for (; c < prefix + chunks; c += warps) {
                const uint32_t j = static_cast<uint32_t>(c - prefix) * 32u + lane;
                if (j < nk) tombs += del_index_key(view, d, u, key_low(keys[gs + j]), ix, st);
            }
            tombs = __reduce_add_sync(kFull, tombs);
            if (lane == 0 && tombs) {
                atomicAdd(&desc[u].meta, tombs << 6);
                removed += tombs;
            }
        }
        prefix += chunks;
    }
    if (stats) {
        warp_count(&stats[kCntRemoved], removed);
        warp_count(&stats[kCntChanged], changed);
    }
    warp_count(&scan_stats[kCntDelScanned], scanned);
    warp_count(&scan_stats[kCntDelScannedCached], scanned_cached);
}

// Rows left by the two kernels before: ordered groups on rows above
// kWarpRowMax, hub groups' rows that are due for compaction, and the queued
// compactions.
__global__ void __launch_bounds__(kTpbMut)
    del_rest(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr, PosIndex ix, DelLists dl,
             CompactList cl, uint32_t *matched, uint32_t *seg_hot, unsigned long long *stats,
             unsigned long long *scan_stats, Status *st) {
    __shared__ OrderedSmem om;
    __shared__ MoveSmem sm;
    const uint32_t tid = threadIdx.x;
    const uint32_t nb = *dl.big_count;
    for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const uint32_t gs = gr.start[dl.big[b]], ge = gr.end[dl.big[b]];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        if (ge - gs > kBigKeys)
            for (uint32_t j = gs + tid; j < ge; j += kTpbMut) matched[j] = 0u;
        __syncthreads();
        const uint32_t done = block_tomb_ordered(view, d, u, keys, gs, ge, matched, om);
        __syncthreads();
        if (idx_row(ix, u)) {
            idx_recount_group(view, d, u, keys, gs, ge, tid, kTpbMut, ix);
            __syncthreads();
        }
        const uint32_t t = rd_tombs(d) + done;
        uint32_t len = d.len, tombs = t;
        if (done && (4ull * t >= d.len || t >= kMaxTombs / 2)) {
            len = block_move_live(view, ix, u, d.off, d.len, d.off, sm, st);
            tombs = 0;
        }
        if (tid == 0 && done) {
            desc[u] = RowDesc{d.off, len, rd_meta(rd_cls(d), tombs)};
            if (stats) {
                atomicAdd(&stats[kCntRemoved], static_cast<unsigned long long>(done));
                atomicAdd(&stats[kCntChanged], 1ull);
            }
        }
        if (tid == 0) {
            seg_touch(seg_hot, d.off, d.len);
            atomicAdd(&scan_stats[kCntDelScanned], static_cast<unsigned long long>(d.len));
            if (view.cached(d.off)) atomicAdd(&scan_stats[kCntDelScannedCached], static_cast<unsigned long long>(d.len));
        }
        __syncthreads();
    }
    const uint32_t ns = *dl.scan_count;
    for (uint32_t b = blockIdx.x; b < ns; b += gridDim.x) {
        const uint32_t gs = gr.start[dl.scan[b]], ge = gr.end[dl.scan[b]];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        if (tid == 0) om.left = 0;
        __syncthreads();
        uint32_t mine = 0;
        for (uint32_t j = gs + tid; j < ge; j += kTpbMut) {
            const uint32_t p = dl.firstpos[j];
            if (p == kInf) continue;  // a missing delete
            write_slot(view, d.off + p, kTomb);
            ++mine;
        }
        mine = __reduce_add_sync(kFull, mine);
        if (lane_id() == 0 && mine) atomicAdd(&om.left, mine);
        __syncthreads();
        const uint32_t done = om.left;
        const uint32_t t = rd_tombs(d) + done;
        uint32_t len = d.len, tombs = t;
        if (done && (4ull * t >= d.len || t >= kMaxTombs / 2)) {
            len = block_move_live(view, ix, u, d.off, d.len, d.off, sm, st);
            tombs = 0;
        }
        if (tid == 0 && done) {
            desc[u] = RowDesc{d.off, len, rd_meta(rd_cls(d), tombs)};
            if (stats) {
                atomicAdd(&stats[kCntRemoved], static_cast<unsigned long long>(done));
                atomicAdd(&stats[kCntChanged], 1ull);
            }
        }
        __syncthreads();
    }
    const uint32_t nh = *dl.huge_count;
    for (uint32_t h = blockIdx.x; h < nh; h += gridDim.x) {
        const uint32_t gs = gr.start[dl.huge[h]], ge = gr.end[dl.huge[h]];
        bool rep = false;  // then it was in the list above
        for (uint32_t i = gs + tid; i + 1 < ge; i += kTpbMut) rep |= keys[i] == keys[i + 1];
        if (__syncthreads_or(rep)) continue;
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        const uint32_t t = rd_tombs(d);
        const uint32_t before = matched[gs];
        __syncthreads();
        if (t == before) continue;
        if (4ull * t >= d.len || t >= kMaxTombs / 2) {
            const uint32_t w = block_move_live(view, ix, u, d.off, d.len, d.off, sm, st);
            if (tid == 0) desc[u] = RowDesc{d.off, w, rd_meta(rd_cls(d), 0)};
        }
        if (tid == 0 && stats) atomicAdd(&stats[kCntChanged], 1ull);
        __syncthreads();
    }
    compact_listed(view, desc, cl, ix, sm, st);
}

// ---------------------------------------------------------------- addition

// Addition plan.  A row whose block has room appends in place (kKeyNone).  A
// row whose used slots would overflow its block while its live entries and
// the additions fit (kKeyInPlace) drops its tombstones where it is.  A row
// that outgrows its block gets a class (sized for the live entries plus the
// additions) and a rank in that class; it moves as it is, tombstones and
// all, when that fits the new block, which leaves every position, and so the
// position index, as it was.  (Giving the second kind a fresh block of its
// own class, as before, lost a block per overflow for good: 3.2 slots per
// inserted edge on the s22 SSSP stream at a steady size.)
constexpr unsigned long long kKeyOverflow = ~0ull - 1ull;  // degree overflow, reported by the apply kernel
constexpr unsigned long long kKeyInPlace = ~0ull - 2ull;

// Serve this batch's demand of one class.
__device__ __forceinline__ void alloc_class(ArenaAlloc *al, uint32_t c, Status *st) {
    const uint32_t need = al->demand[c];
    al->demand[c] = 0;
    al->avail[c] = 0;
    if (need == 0) return;
    if (c <= kSegShift) {
        const unsigned long long cur = al->cur_next[c], end = al->cur_end[c];
        const unsigned long long room = (end - cur) >> c;
        al->base_cur[c] = cur;
        if (need <= room) {
            al->avail[c] = need;
            al->cur_next[c] = cur + (static_cast<unsigned long long>(need) << c);
            return;
        }
        al->avail[c] = static_cast<uint32_t>(room);
        const unsigned long long rest = need - room;
        const unsigned long long per_seg = 1ull << (kSegShift - c);
        const unsigned long long nseg = (rest + per_seg - 1) / per_seg;
        const unsigned long long s0 = atomicAdd(&al->seg_bump, nseg);
        if (s0 + nseg > al->seg_total) {
            set_error(st, kErrArena, c);
            return;
        }
        al->base_new[c] = s0 << kSegShift;
        al->cur_next[c] = al->base_new[c] + (rest << c);
        al->cur_end[c] = (s0 + nseg) << kSegShift;
    } else {
        const unsigned long long nseg = static_cast<unsigned long long>(need) << (c - kSegShift);
        const unsigned long long s0 = atomicAdd(&al->seg_bump, nseg);
        if (s0 + nseg > al->seg_total) {
            set_error(st, kErrArena, c);
            return;
        }
        al->base_new[c] = s0 << kSegShift;
    }
}

// The last block to finish hands out the blocks (one thread per class) and
// gives the new segments cache slots: two launches less in the chain.
__global__ void plan_add(const RowDesc *desc, const unsigned long long *keys, Groups gr, unsigned long long *plan,
                         ArenaAlloc *al, bool assign, SegTable seg, uint32_t *blocks_done, Status *st) {
    const uint32_t ng = *gr.count;
    const uint32_t rounded = (ng + 31u) & ~31u;
    const uint32_t lane = lane_id();
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < rounded; g += gridDim.x * blockDim.x) {
        unsigned long long p = kKeyNone;
        bool move = false;
        uint32_t cls = 0;
        if (g < ng) {
            const uint32_t gs = gr.start[g];
            const uint32_t ge = gr.end[g];
            const RowDesc d = desc[key_src(keys[gs])];
            const unsigned long long used = static_cast<unsigned long long>(d.len) + (ge - gs);
            const unsigned long long live = static_cast<unsigned long long>(rd_live(d)) + (ge - gs);
            if (live > 0xFFFFFFFFull) {
                p = kKeyOverflow;
            } else if (rd_cls(d) == 0 || live > (1ull << rd_cls(d))) {
                cls = class_for(static_cast<uint32_t>(live));
                move = true;
            } else if (used > (1ull << rd_cls(d))) {
                p = kKeyInPlace;
            }
        }
        // Ranks within a class, one atomic per class present in the warp
        // (tens of thousands of moving rows share a handful of classes).
        const uint32_t movers = __ballot_sync(kFull, move);
        if (move) {
            const uint32_t peers = __match_any_sync(movers, cls);
            const uint32_t leader = __ffs(peers) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&al->demand[cls], static_cast<uint32_t>(__popc(peers)));
            base = __shfl_sync(peers, base, leader);
            p = (static_cast<unsigned long long>(cls) << 32) | (base + __popc(peers & lanemask_lt()));
        }
        if (g < ng) plan[g] = p;
    }
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (uint32_t c = threadIdx.x; c < kNumClasses; c += blockDim.x) alloc_class(al, c, st);
    __syncthreads();
    if (threadIdx.x == 0) {
        *blocks_done = 0;
        if (assign) seg_assign_new(seg, *reinterpret_cast<volatile unsigned long long *>(&al->seg_bump), st);
    }
}

// Addition phase.  mutate_add gives each lane a group of its own when the
// lane can serve it alone (at most kLaneAdds appends, and a moving row of at
// most kLaneRow slots, read into registers with independent loads: rows in
// host memory cost one round trip, not one per entry), so the common
// one-request groups run 32 to a warp.  The other groups are listed for
// mutate_add_wide, which serves them one warp per group over the whole grid
// (a block per row of more than kWarpRowMax slots that must move, or than
// kWarpMove that must drop its tombstones).  Serving them inside the warp that found them left the
// busiest warps a serial queue of up to 32 row copies while most of the grid
// had no group at all.  `vals` is add_v for the forward arena and add_u for
// the reverse arena.  A moving row keeps its tombstones where the new block
// holds them (moves_whole); the short rows that a lane moves drop theirs.
constexpr uint32_t kLaneAdds = 8;
constexpr uint32_t kLaneRow = 8;

// Groups for whole warps and for whole blocks.
struct AddLists {
    uint32_t *warp;
    uint32_t *warp_count;
    uint32_t *block;
    uint32_t *block_count;
};

// A moving row keeps its tombstones when they fit the new block.
__device__ __forceinline__ bool moves_whole(unsigned long long p, const RowDesc &d, uint32_t a) {
    return p != kKeyInPlace && static_cast<unsigned long long>(d.len) + a <= (1ull << static_cast<uint32_t>(p >> 32));
}

__global__ void __launch_bounds__(256, 4)
    mutate_add(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr,
                           const unsigned long long *plan, const ArenaAlloc *al, const uint32_t *vals,
                           AddLists ls, unsigned long long *stats, PosIndex ix, Status *st) {
    if (ld_volatile(&st->err) & kErrArena) return;
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t ng = *gr.count;
    uint32_t changed = 0, moved = 0, moved_entries = 0;  // per lane
    for (uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u; base < ng; base += warps * 32u) {
        const uint32_t g = base + lane;
        bool coop = false, block = false;
        if (g < ng) {
            const unsigned long long p = plan[g];
            const uint32_t gs = gr.start[g];
            const uint32_t a = gr.end[g] - gs;
            const uint32_t u = key_src(keys[gs]);
            const RowDesc d = desc[u];
            const bool indexed = idx_row(ix, u);
            if (p == kKeyOverflow) {
                set_error(st, kErrInternal, g);
            } else if (p != kKeyNone && d.len > (moves_whole(p, d, a) ? kWarpRowMax : kWarpMove)) {
                block = true;
            } else if (a > kLaneAdds) {
                coop = true;
            } else {
                // The appended values first, with independent loads (the
                // stores below could alias them as far as the compiler knows).
                uint32_t add[kLaneAdds];
#pragma unroll
                for (uint32_t j = 0; j < kLaneAdds; ++j) add[j] = j < a ? vals[key_low(keys[gs + j])] : 0u;
                if (p == kKeyNone) {
                    // A block of at most one segment: one slot lookup for the
                    // row's end, then plain stores.
                    if (rd_cls(d) <= kSegShift) {
                        uint32_t *wp = view.wptr(d.off + d.len);
#pragma unroll
                        for (uint32_t j = 0; j < kLaneAdds; ++j)
                            if (j < a) wp[j] = add[j];
                    } else {
                        for (uint32_t j = 0; j < a; ++j) write_slot(view, d.off + d.len + j, add[j]);
                    }
                    if (indexed) idx_add_n<kLaneAdds>(ix, u, add, d.len, a, st);
                    desc[u] = RowDesc{d.off, d.len + a, d.meta};
                    changed += 1;
                } else if (d.len > kLaneRow || indexed) {
                    coop = true;
                } else {
                    // In place, or to a larger block.
                    const bool moves = p != kKeyInPlace;
                    const uint32_t cls = moves ? static_cast<uint32_t>(p >> 32) : rd_cls(d);
                    const unsigned long long off = moves ? alloc_offset(al, cls, static_cast<uint32_t>(p)) : d.off;
                    // Old block (<= kLaneRow slots) and new block (<= 16 slots)
                    // each lie in one segment: one slot lookup apiece.
                    uint32_t row[kLaneRow];
                    const uint32_t *src = d.len ? view.at(d.off) : nullptr;
#pragma unroll
                    for (uint32_t k = 0; k < kLaneRow; ++k) row[k] = k < d.len ? src[k] : kTomb;
                    uint32_t *wp = view.wptr(off);
                    uint32_t w = 0;
#pragma unroll
                    for (uint32_t k = 0; k < kLaneRow; ++k)
                        if (row[k] != kTomb) wp[w++] = row[k];
#pragma unroll
                    for (uint32_t j = 0; j < kLaneAdds; ++j)
                        if (j < a) wp[w + j] = add[j];
                    desc[u] = RowDesc{off, w + a, rd_meta(cls, 0)};
                    moved += moves ? 1u : 0u;
                    moved_entries += moves ? w : 0u;
                    changed += 1;
                }
            }
        }
        warp_enqueue(coop, g, ls.warp, ls.warp_count, ng, st);
        warp_enqueue(block, g, ls.block, ls.block_count, ng, st);
    }
    if (stats) {
        warp_count(&stats[kCntChanged], changed);
        warp_count(&stats[kCntRelocated], moved);
        warp_count(&stats[kCntMovedEntries], moved_entries);
    }
}


// The groups mutate_add listed: a block per long row, then a warp per group.
__global__ void __launch_bounds__(kTpbMut, 2)
    mutate_add_wide(AdjView view, RowDesc *desc, const unsigned long long *keys, Groups gr,
                    const unsigned long long *plan, const ArenaAlloc *al, const uint32_t *vals, AddLists ls,
                    unsigned long long *stats, PosIndex ix, Status *st) {
    __shared__ MoveSmem sm;
    if (ld_volatile(&st->err) & kErrArena) return;
    const uint32_t nb = *ls.block_count;
    for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const uint32_t g = ls.block[b];
        const unsigned long long p = plan[g];
        const uint32_t gs = gr.start[g];
        const uint32_t ge = gr.end[g];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        const uint32_t a = ge - gs;
        const bool moves = p != kKeyInPlace;
        const uint32_t cls = moves ? static_cast<uint32_t>(p >> 32) : rd_cls(d);
        const bool whole = moves_whole(p, d, a);
        const unsigned long long off = moves ? alloc_offset(al, cls, static_cast<uint32_t>(p)) : d.off;
        uint32_t w = d.len;
        if (!whole) {
            w = block_move_live(view, ix, u, d.off, d.len, off, sm, st);
        } else {
            // 16 entries per thread and step, resolved per 16 bytes (a block
            // above one segment may lie in HBM and in host memory).
            for (uint32_t b0 = 0; b0 < d.len; b0 += 16u * kTpbMut) {
                uint4 q[4];
#pragma unroll
                for (uint32_t h = 0; h < 4; ++h) {
                    const uint32_t k = b0 + 4u * (h * kTpbMut + threadIdx.x);
                    if (k < d.len) q[h] = *reinterpret_cast<const uint4 *>(view.at(d.off + k));
                }
#pragma unroll
                for (uint32_t h = 0; h < 4; ++h) {
                    const uint32_t k = b0 + 4u * (h * kTpbMut + threadIdx.x);
                    if (k < d.len) *reinterpret_cast<uint4 *>(view.wptr(off + k)) = q[h];
                }
            }
        }
        __syncthreads();  // moved before the appends behind them (and before their index entries)
        const bool indexed = idx_row(ix, u);
        for (uint32_t j = threadIdx.x; j < a; j += kTpbMut) {
            const uint32_t v = vals[key_low(keys[gs + j])];
            write_slot(view, off + w + j, v);
            if (indexed) idx_add(ix, u, v, w + j, st);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            desc[u] = RowDesc{off, w + a, rd_meta(cls, whole ? rd_tombs(d) : 0u)};
            if (stats) {
                atomicAdd(&stats[kCntChanged], 1ull);
                atomicAdd(&stats[kCntRelocated], moves ? 1ull : 0ull);
                atomicAdd(&stats[kCntMovedEntries], moves ? static_cast<unsigned long long>(w) : 0ull);
            }
        }
    }
    const uint32_t lane = lane_id();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nc = *ls.warp_count;
    uint32_t changed = 0, moved = 0, moved_entries = 0;  // lane 0 counts
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nc; i += warps) {
        const uint32_t gb = ls.warp[i];
        const unsigned long long p = plan[gb];
        const uint32_t gs = gr.start[gb];
        const uint32_t ge = gr.end[gb];
        const uint32_t u = key_src(keys[gs]);
        const RowDesc d = desc[u];
        const uint32_t a = ge - gs;
        if (p == kKeyNone) {
            const bool indexed = idx_row(ix, u);
            for (uint32_t j = lane; j < a; j += 32u) {
                const uint32_t v = vals[key_low(keys[gs + j])];
                write_slot(view, d.off + d.len + j, v);
                if (indexed) idx_add(ix, u, v, d.len + j, st);
            }
            if (lane == 0) desc[u] = RowDesc{d.off, d.len + a, d.meta};
        } else {
            const bool moves = p != kKeyInPlace;
            const uint32_t cls = moves ? static_cast<uint32_t>(p >> 32) : rd_cls(d);
            const bool whole = moves_whole(p, d, a);
            const unsigned long long off = moves ? alloc_offset(al, cls, static_cast<uint32_t>(p)) : d.off;
            uint32_t w = d.len;
            if (!whole) {
                w = warp_move_live(view, ix, u, d.off, d.len, off, st);
            } else if (d.len) {
                // Old and new block each lie in one segment and start on a
                // 16-byte boundary: 512 entries per step, four independent
                // 16-byte loads per lane before any store (a zero-copy row
                // costs one host round trip per step).
                const uint32_t *src = view.at(d.off);
                uint32_t *dst = view.wptr(off);
                for (uint32_t b0 = 0; b0 < d.len; b0 += 512u) {
                    uint4 q[4];
#pragma unroll
                    for (uint32_t h = 0; h < 4; ++h) {
                        const uint32_t k = b0 + 128u * h + 4u * lane;
                        if (k < d.len) q[h] = *reinterpret_cast<const uint4 *>(src + k);
                    }
#pragma unroll
                    for (uint32_t h = 0; h < 4; ++h) {
                        const uint32_t k = b0 + 128u * h + 4u * lane;
                        if (k < d.len) *reinterpret_cast<uint4 *>(dst + k) = q[h];
                    }
                }
                __syncwarp();  // the last 16 bytes may reach past the row's end, where the appends go
            }
            const bool indexed = idx_row(ix, u);
            for (uint32_t j = lane; j < a; j += 32u) {
                const uint32_t v = vals[key_low(keys[gs + j])];
                write_slot(view, off + w + j, v);  // many additions may span segments
                if (indexed) idx_add(ix, u, v, w + j, st);
            }
            if (lane == 0) {
                desc[u] = RowDesc{off, w + a, rd_meta(cls, whole ? rd_tombs(d) : 0u)};
                moved += moves ? 1u : 0u;
                moved_entries += moves ? w : 0u;
            }
        }
        if (lane == 0) changed += 1;
    }
    if (stats) {
        warp_count(&stats[kCntChanged], changed);
        warp_count(&stats[kCntRelocated], moved);
        warp_count(&stats[kCntMovedEntries], moved_entries);
    }
}

}  // namespace cig
