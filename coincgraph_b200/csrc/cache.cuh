// cache.cuh - device-side segment table of the HBM edge cache.
//
// The forward arena is cut into 64 KiB segments; `seg_slot` maps each to a
// slot of the HBM cache pool or to -1 (served zero-copy from pinned host
// memory).  This table is owned and changed by the GPU alone, once per batch
// (after the insertion phase), so a batch never waits on the host for a
// residency decision:
//   - hotness: every row read or rewritten adds its length to `hot` of its
//     segment; the service folds it into a decayed `score` (score/2 + hot);
//   - new segments handed out by the block allocator take a free slot at
//     once (their rows were just written, so they are hot), and the service
//     keeps `reserve` slots free for them by evicting the coldest resident
//     segments (a histogram of log2(score) picks the threshold);
//   - host segments whose score passed admit_score are copied in, at most
//     kMaxAdmit per batch, into slots freed from cold segments;
//   - an evicted segment is written back first if it is dirty.
// The reference keeps per-vertex hotness in a 4-batch uint8 window, sorts
// vertices by it and re-packs the cached rows when the admitted set changes
// (include/framework/variants/driver.cuh:53-247, 691-770; framework.cuh:
// 599-798); residency here is per segment, so admission is a slot copy and
// the arena layout never changes.
#pragma once

#include "common.cuh"

namespace cig {

constexpr uint32_t kAdmitScore = 8192;   // default: ~half a segment of entries read recently
constexpr uint32_t kColdScore = 1u << 30;  // default cap: segments scoring this much are never evicted
constexpr int kScoreBuckets = 33;          // bucket of a score: 32 - clz(score)
constexpr uint32_t kMaxAdmit = 64;       // admissions per batch (4 MiB over the host link)
constexpr uint32_t kMaxEvict = 1024;     // evictions per batch
constexpr uint32_t kNewScore = 16384;    // score of a freshly allocated segment

enum SegCtl : int {
    kCtlFreeTop = 0,    // entries on the free-slot stack
    kCtlBumpSeen = 1,   // allocator bump pointer when slots were last handed out
    kCtlNewLast = 2,    // segments created since the last service
    kCtlVictims = 3,    // cold resident segments found this service
    kCtlAdmits = 4,     // hot host segments found this service
    kCtlExtraTaken = 5, // victims taken from the threshold bucket
    kCtlHist = 16,      // kScoreBuckets counters of resident scores
    kCtlCount = 16 + kScoreBuckets
};

struct SegTable {
    int32_t *seg_slot;    // per segment: slot or -1
    int32_t *slot_seg;    // per slot: owning segment or -1
    uint8_t *seg_dirty;   // per segment: HBM copy newer than the host copy
    uint32_t *score;      // per segment
    uint32_t *hot;        // per segment, since the last service
    uint32_t *free_slots; // stack
    uint32_t *victims;    // this service's evictions (slots)
    uint32_t *admits;     // this service's admissions (segments)
    uint32_t *ctl;        // SegCtl
    uint32_t nslots;
    uint32_t nsegs;
    uint32_t admit_score;  // host segments at or above are admitted
    uint32_t cold_score;   // resident segments below may be evicted
};

__device__ __forceinline__ void seg_touch(uint32_t *hot, uint64_t off, uint32_t len) {
    if (hot && len) atomicAdd(hot + (off >> kSegShift), len);
}

// Slots for the segments the allocator created since the last call (`bump`:
// its bump pointer).  One thread; a handful of segments per batch.
__device__ __forceinline__ void seg_assign_new(const SegTable &t, unsigned long long seg_bump, Status *st) {
    const uint32_t bump = static_cast<uint32_t>(min(seg_bump, static_cast<unsigned long long>(t.nsegs)));
    const uint32_t seen = t.ctl[kCtlBumpSeen];
    uint32_t top = t.ctl[kCtlFreeTop];
    for (uint32_t s = seen; s < bump; ++s) {
        t.score[s] = kNewScore;
        if (t.seg_slot[s] >= 0 || top == 0) continue;
        const uint32_t slot = t.free_slots[--top];
        t.seg_slot[s] = static_cast<int32_t>(slot);
        t.slot_seg[slot] = static_cast<int32_t>(s);
        t.seg_dirty[s] = 0;
        atomicAdd(&st->counters[kCntSegLoaded], 1ull);
    }
    t.ctl[kCtlFreeTop] = top;
    t.ctl[kCtlNewLast] += bump > seen ? bump - seen : 0u;
    t.ctl[kCtlBumpSeen] = max(seen, bump);
}

// Clear the per-batch counters, before the batch's first allocation; one
// thread per word (at least kCtlCount threads).
__device__ __forceinline__ void seg_ctl_clear(uint32_t *ctl) {
    const uint32_t i = threadIdx.x;
    if (i < kCtlCount && i != kCtlFreeTop && i != kCtlBumpSeen) ctl[i] = 0u;
}

// Start of a phase: advance the batch epoch (the "invalidated in this batch"
// marker of aff_stamp, kept on the device so that a captured batch graph
// needs no new arguments; null: keep it), clear the counters of `counters` (64
// words) whose bit is set in `mask` and the segment table's per-batch ones
// (null: no table), in place of one memset each.  One block of at least 64
// threads.
__device__ __forceinline__ void begin_phase(uint32_t *epoch, uint32_t *counters, unsigned long long mask,
                                            uint32_t *seg_ctl) {
    if (epoch && threadIdx.x == 0) *epoch += 1u;
    if (threadIdx.x < 64u && ((mask >> threadIdx.x) & 1u)) counters[threadIdx.x] = 0u;
    if (seg_ctl) seg_ctl_clear(seg_ctl);
}

__device__ __forceinline__ uint32_t score_bucket(uint32_t sc) { return 32u - __clz(sc); }

// One block copies one 64 KiB segment: each thread has eight 16-byte loads
// in flight before it stores them, so a copy from host memory (about 2 us
// away) takes two round trips instead of sixteen.
__device__ __forceinline__ void copy_segment(uint4 *dst, const uint4 *src) {
    constexpr uint32_t kVec = kSegEdges / 4, kDepth = 8;
    for (uint32_t i0 = 0; i0 < kVec; i0 += kDepth * blockDim.x) {
        uint4 r[kDepth];
#pragma unroll
        for (uint32_t j = 0; j < kDepth; ++j) {
            const uint32_t i = i0 + j * blockDim.x + threadIdx.x;
            r[j] = i < kVec ? src[i] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (uint32_t j = 0; j < kDepth; ++j) {
            const uint32_t i = i0 + j * blockDim.x + threadIdx.x;
            if (i < kVec) dst[i] = r[j];
        }
    }
}

// The service of one batch (cooperative launch), in four steps with a grid
// barrier between them; a batch with nothing to evict or admit ends after the
// first.  (Five kernels and two memsets before: 16 to 25 us of launches for
// what is mostly one pass over the scores.)  The counters of seg_ctl_clear
// are zero at launch, kCtlNewLast counts this batch's new segments.
//   1. decay the scores, histogram the resident ones that may go (below
//      cold_score), list hot host segments as admission candidates;
//   2. choose the victims: enough to keep `reserve` slots free for new
//      segments (twice the last batch's count, 16..1024) plus the admissions,
//      the coldest first: whole buckets below a threshold, then part of it;
//   3. a block per victim: write back if dirty, unmap, free the slot;
//   4. a block per candidate while free slots above the reserve last: copy
//      the host segment into a slot and map it.
__global__ void __launch_bounds__(256) seg_service(SegTable t, uint32_t bump, uint32_t *cache, uint32_t *host,
                                                   Status *st) {
    __shared__ uint32_t hist[kScoreBuckets];
    __shared__ uint32_t s_top, s_reserve, s_need, s_thr, s_extra;
    __shared__ int32_t slot_s;
    // Every block makes the plan below for itself, so its inputs are read
    // before the first barrier: behind it a block with nothing to evict goes
    // straight to the admissions, which take from kCtlFreeTop, and a later
    // reader would plan an eviction and wait at a barrier the others skip.
    if (threadIdx.x == 0) {
        s_top = ld_volatile(t.ctl + kCtlFreeTop);
        s_reserve = min(1024u, max(16u, 2u * ld_volatile(t.ctl + kCtlNewLast)));
    }
    const uint32_t gtid = blockIdx.x * blockDim.x + threadIdx.x, gthreads = gridDim.x * blockDim.x;
    for (uint32_t b = threadIdx.x; b < kScoreBuckets; b += blockDim.x) hist[b] = 0;
    __syncthreads();
    for (uint32_t s = gtid; s < bump; s += gthreads) {
        const uint32_t h = t.hot[s];
        if (h) t.hot[s] = 0;
        const uint32_t sc = (t.score[s] >> 1) + min(h, 1u << 24);
        t.score[s] = sc;
        if (t.seg_slot[s] >= 0) {
            if (sc < t.cold_score) atomicAdd(hist + score_bucket(sc), 1u);
        } else if (sc >= t.admit_score) {
            const uint32_t i = atomicAdd(t.ctl + kCtlAdmits, 1u);
            if (i < kMaxAdmit) t.admits[i] = s;
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kScoreBuckets; b += blockDim.x)
        if (hist[b]) atomicAdd(t.ctl + kCtlHist + b, hist[b]);
    if (!grid_barrier(st)) return;
    const uint32_t na = min(ld_volatile(t.ctl + kCtlAdmits), kMaxAdmit);
    if (threadIdx.x == 0) {  // every block comes to the same plan
        const uint32_t want = s_reserve + na;
        const uint32_t top = s_top;
        uint32_t need = min(want > top ? want - top : 0u, kMaxEvict);
        uint32_t below = 0, b = 0;
        if (need)
            for (; b < static_cast<uint32_t>(kScoreBuckets); ++b) {
                const uint32_t c = ld_volatile(t.ctl + kCtlHist + b);
                if (below + c >= need) break;
                below += c;
            }
        if (b == static_cast<uint32_t>(kScoreBuckets)) need = below;  // fewer evictable segments than wanted
        s_need = need;
        s_thr = b;
        s_extra = need - below;
    }
    __syncthreads();
    const uint32_t need = s_need, reserve = s_reserve;
    if (!need && !na) return;
    if (need) {
        for (uint32_t s = gtid; s < bump; s += gthreads) {
            const int32_t slot = t.seg_slot[s];
            if (slot < 0) continue;
            const uint32_t sc = t.score[s];
            if (sc >= t.cold_score) continue;
            const uint32_t b = score_bucket(sc);
            bool take = b < s_thr;
            if (!take && b == s_thr && s_extra) take = atomicAdd(t.ctl + kCtlExtraTaken, 1u) < s_extra;
            if (take) {
                const uint32_t i = atomicAdd(t.ctl + kCtlVictims, 1u);
                if (i < need) t.victims[i] = static_cast<uint32_t>(slot);
            }
        }
        if (!grid_barrier(st)) return;
        const uint32_t nv = min(need, ld_volatile(t.ctl + kCtlVictims));
        for (uint32_t v = blockIdx.x; v < nv; v += gridDim.x) {
            const uint32_t slot = t.victims[v];
            const int32_t seg = t.slot_seg[slot];
            if (seg < 0) continue;
            if (t.seg_dirty[seg])
                copy_segment(reinterpret_cast<uint4 *>(host + (static_cast<uint64_t>(seg) << kSegShift)),
                             reinterpret_cast<const uint4 *>(cache + (static_cast<uint64_t>(slot) << kSegShift)));
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence_system();
                t.seg_dirty[seg] = 0;
                t.seg_slot[seg] = -1;
                t.slot_seg[slot] = -1;
                const uint32_t pos = atomicAdd(t.ctl + kCtlFreeTop, 1u);
                if (pos < t.nslots)
                    t.free_slots[pos] = slot;
                else
                    set_error(st, kErrInternal, pos);
                atomicAdd(&st->counters[kCntSegEvicted], 1ull);
            }
            __syncthreads();
        }
        if (!grid_barrier(st)) return;
    }
    for (uint32_t a = blockIdx.x; a < na; a += gridDim.x) {
        const uint32_t seg = t.admits[a];
        if (threadIdx.x == 0 && t.seg_slot[seg] < 0) {
            slot_s = -1;
            // Take a slot only while more than `reserve` remain.
            uint32_t top = ld_volatile(t.ctl + kCtlFreeTop);
            while (top > reserve) {
                const uint32_t prev = atomicCAS(t.ctl + kCtlFreeTop, top, top - 1);
                if (prev == top) {
                    slot_s = static_cast<int32_t>(t.free_slots[top - 1]);
                    break;
                }
                top = prev;
            }
        }
        if (threadIdx.x == 0 && t.seg_slot[seg] >= 0) slot_s = -1;
        __syncthreads();
        const int32_t slot = slot_s;
        if (slot >= 0) {
            copy_segment(reinterpret_cast<uint4 *>(cache + (static_cast<uint64_t>(slot) << kSegShift)),
                         reinterpret_cast<const uint4 *>(host + (static_cast<uint64_t>(seg) << kSegShift)));
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                t.seg_dirty[seg] = 0;
                t.slot_seg[slot] = static_cast<int32_t>(seg);
                t.seg_slot[seg] = slot;
                atomicAdd(&st->counters[kCntSegLoaded], 1ull);
            }
        }
        __syncthreads();
    }
}

}  // namespace cig
