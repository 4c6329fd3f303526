// Counting without moving: the histogram of every (scale, context) pair where each sees a narrow range of symbols, as
// the contexts of a quantised weight do -- a few dozen neighbouring BF16 patterns each, a few thousand where values go
// through zero.  Patterns of either sign are a range of their own (a half segment).
//
//   range    smallest and largest symbol of every half segment
//   count    a counter per symbol of every range; the counters of one scale, some ten thousand, in shared memory, a
//            stretch of units of that scale per CTA, then added to the scale's counters in global memory
//   items    counters -> items, ascending: half segments of positive patterns precede those of negative ones
//
// Nothing is scattered: the general form (histogram.cuh) writes every symbol to its segment, two bytes at a place of
// their own, and reads it back.  Taken where the counters are no more than elements and those of a scale fit shared
// memory; the rest, and rows that do not come in fours, go the general way.
// Bound: shared-memory atomics, one per element, and one read of the tensor per pass.
// Measured, us, 14336 x 4096 FP8 per channel | 4096 x 4096 INT4 by group: ranges 71 | 30, counts 73 | 48, items 31 | 50.  With
// pieces of four elements, divisions to find them, ranges of two words and stretches in one round and a bit: 103 | 39, 98 |
// 58; with a warp per segment however long: 76 | 96.  The general form: 770 | 540 in all.
#pragma once

#include <cooperative_groups.h>

#include "histogram.cuh"

namespace mps {
namespace hist {

constexpr int kDenseThreads = 512;                  // (1024 where a scale's counters leave room for one CTA per SM)
constexpr int kDenseCounters = 56 * 1024;           // most counters of a scale: what one CTA's shared memory holds (up to 26 K two share an SM)
// Fewer elements per scale than this: not tried, the counters of a scale are then as many as its elements.  Whole builds, us,
// counters | the general form, INT4 by scale, by elements per scale: 1044: 947 | 850, 3518: 1192 | 1091, 6512: 1214 | 1113,
// 12157: 903 | 1233, 39756: 1290 | 1627.  (FP8 weights have a tenth of the counters and meet below 2 K: 612: 918 | 845,
// 1351: 847 | 751, 2674: 598 | 765, 6553: 530 | 650.)
constexpr long long kDenseMinPerScale = 8192;

// A CTA takes a stretch of the unit list, of one scale and at most `upc` units (a scale of a few units is a stretch too:
// stretches of equal length over several scales leave the CTAs at the ends of the distribution, with dozens of scales
// each, as stragglers).  Its threads walk the pieces (V neighbouring elements, eight where rows and pointers allow) of it.
struct DenseGeom {
    Geom g;
    const uint32_t* first;           // first unit of every stretch, [0, *count)
    const uint32_t* count;
    uint32_t upc;
    uint32_t row, unit;              // pieces of a unit's row, of a unit
    uint32_t by_row, by_unit;        // ceil(2^32 / those): a stretch has fewer than 2^32 / unit pieces (dense_magic)
    int units_shift;                 // nbu1 == 1 << units_shift, or -1
};
// x / d == umulhi(x, dense_magic(d)) where x * d < 2^32 (d > 1; a 1 is left to the caller)
inline uint32_t dense_magic(uint32_t d) { return d > 1u ? (uint32_t)(((1ull << 32) + d - 1u) / d) : 0u; }

// f(context, symbol) of pieces [first, last) of units j0 and on, UN pieces of a thread in flight
template <int V, int UN, class F>
__device__ __forceinline__ void for_pieces(const DenseGeom& d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx,
                                           const uint32_t* __restrict__ unit_sorted, long long j0, uint32_t first, uint32_t last, F&& f) {
    static_assert(V == 4 || V == 8, "a piece is one or two words of context bytes");
    for (uint32_t q0 = first + threadIdx.x; q0 < last; q0 += UN * blockDim.x) {
        uint32_t cw[UN][V / 4], sw[UN][V / 2];
        bool in[UN];
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            const uint32_t q = q0 + i * blockDim.x;
            in[i] = q < last;
            long long at = 0;
            if (in[i]) {
                const uint32_t j = d.unit == 1u ? q : __umulhi(q, d.by_unit), w = q - j * d.unit;
                const uint32_t u = unit_sorted[j0 + j];
                const uint32_t bi = d.units_shift >= 0 ? u >> d.units_shift : u / (uint32_t)d.g.nbu1, bj = u - bi * (uint32_t)d.g.nbu1;
                // (uniform shortcut: one row per unit)
                const uint32_t r = d.g.ub0 == 1 ? 0u : (d.row == 1u ? w : __umulhi(w, d.by_row)), c = w - r * d.row;
                const uint32_t row = bi * (uint32_t)d.g.ub0 + r, col = bj * (uint32_t)d.g.ub1 + V * c;   // (fewer than 2^31 elements)
                in[i] = row < (uint32_t)d.g.n && col < (uint32_t)d.g.m;     // (m and ub1 are multiples of V)
                at = (long long)row * d.g.m + col;
            }
            if constexpr (V == 8) {
                const uint2 c = in[i] ? *reinterpret_cast<const uint2*>(ctx + at) : make_uint2(0u, 0u);
                const uint4 x = in[i] ? *reinterpret_cast<const uint4*>(sym + at) : make_uint4(0u, 0u, 0u, 0u);
                cw[i][0] = c.x; cw[i][1] = c.y;
                sw[i][0] = x.x; sw[i][1] = x.y; sw[i][2] = x.z; sw[i][3] = x.w;
            } else {
                cw[i][0] = in[i] ? *reinterpret_cast<const uint32_t*>(ctx + at) : 0u;
                const uint2 x = in[i] ? *reinterpret_cast<const uint2*>(sym + at) : make_uint2(0u, 0u);
                sw[i][0] = x.x; sw[i][1] = x.y;
            }
        }
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            if (!in[i]) continue;
#pragma unroll
            for (int v = 0; v < V; ++v)
                f((cw[i][v >> 2] >> (8 * (v & 3))) & d.g.ctx_mask, (v & 1) ? sw[i][v >> 1] >> 16 : sw[i][v >> 1] & 0xFFFFu);
        }
    }
}

// First unit of every stretch, `most` of them, by `ctas` CTAs; `base`: the stretches before those of every scale value.  The other
// CTAs look at lists that a caller handed in: beside the searches that costs a build nothing, in a launch of its own 5 us.
__global__ void dense_stretch_fill_kernel(Geom g, const uint16_t* __restrict__ scales, UnitLists lists, const uint32_t* __restrict__ base,
                                          uint32_t upc, uint32_t most, uint32_t ctas, uint32_t* __restrict__ first) {
    if (blockIdx.x >= ctas) { check_unit_lists(g, scales, lists, blockIdx.x - ctas, gridDim.x - ctas); return; }
    const uint32_t* const unit_ofs = lists.ofs;
    const uint32_t all = base[kScaleValues] < most ? base[kScaleValues] : most;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < all; s += ctas * blockDim.x) {
        uint32_t lo = 0, hi = kScaleValues;     // base[lo] <= s < base[hi]
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (base[mid] <= s) lo = mid; else hi = mid;
        }
        first[s] = unit_ofs[lo] + (s - base[lo]) * upc;
    }
}

// Calls f(rank, first unit, end) for the CTA's stretch, if it has one.  (uniform)
template <class F>
__device__ __forceinline__ void for_stretch(const DenseGeom& d, const uint16_t* __restrict__ scales, const UnitLists& lists, F&& f) {
    if (*lists.bad || blockIdx.x >= *d.count) return;
    const uint32_t j = d.first[blockIdx.x];
    if (j >= lists.units) return;       // (of a scale that no unit has: the totals give such lists away)
    const uint32_t v = unit_scale(d.g, scales, lists.sorted[j]);
    const uint32_t past = lists.ofs[v + 1];          // the list is ordered by scale
    f(lists.rank[v], (long long)j, (long long)(j + d.upc < past ? j + d.upc : past));
}

// lo / hi of half segment h: [rank * nctx * 2 + context * 2 + sign], preset to 0xFFFFFFFF and 0.  A range is kept as one word,
// smallest symbol | (largest - smallest) << 16, so that an element costs one look, a subtraction and a comparison; the few
// that widen a range do so in two words beside it and renew it (a word that is behind costs others an atomic too many).
template <int V>
__global__ void __launch_bounds__(kDenseThreads)
dense_range_kernel(DenseGeom d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx, const uint16_t* __restrict__ scales,
                   UnitLists lists, uint32_t* __restrict__ lo, uint32_t* __restrict__ hi) {
    const uint32_t* __restrict__ const unit_sorted = lists.sorted;
    constexpr uint32_t kEmpty = 0xFFFFu;      // (a range of the one symbol that is no BF16 number's)
    __shared__ uint32_t s_range[512], s_lo[512], s_hi[512];
    const uint32_t halves = (uint32_t)d.g.nctx * 2u;
    for_stretch(d, scales, lists, [&](uint32_t rk, long long j0, long long j1) {
        for (uint32_t h = threadIdx.x; h < halves; h += kDenseThreads) { s_range[h] = kEmpty; s_lo[h] = 0xFFFFFFFFu; s_hi[h] = 0u; }
        __syncthreads();
        auto widen = [&](uint32_t c, uint32_t v) {
            const uint32_t h = c * 2u + (v >> 15);
            uint32_t r;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(&s_range[h])));
            if (v - (r & 0xFFFFu) > (r >> 16) || v == kEmpty) {
                const uint32_t lo_now = min(atomicMin(&s_lo[h], v), v), hi_now = max(atomicMax(&s_hi[h], v), v);
                *reinterpret_cast<volatile uint32_t*>(&s_range[h]) = lo_now | ((hi_now - lo_now) << 16);
            }
        };
        // a first piece per thread by itself: against empty ranges every element is an exchange, against those of some
        // thousand elements few are
        const uint32_t total = (uint32_t)(j1 - j0) * d.unit, few = total < kDenseThreads ? total : kDenseThreads;
        for_pieces<V, 1>(d, sym, ctx, unit_sorted, j0, 0u, few, widen);
        __syncthreads();
        for_pieces<V, 4>(d, sym, ctx, unit_sorted, j0, few, total, widen);
        __syncthreads();
        for (uint32_t h = threadIdx.x; h < halves; h += kDenseThreads) {
            if (s_lo[h] <= s_hi[h]) {
                atomicMin(&lo[(size_t)rk * halves + h], s_lo[h]);
                atomicMax(&hi[(size_t)rk * halves + h], s_hi[h]);
            }
        }
        __syncthreads();
    });
}

// ranges before the first symbol
__global__ void dense_preset_kernel(uint32_t* __restrict__ lo, uint32_t* __restrict__ hi, long long nhalf) {
    for (long long h = (long long)blockIdx.x * blockDim.x + threadIdx.x; h < nhalf; h += (long long)gridDim.x * blockDim.x) {
        lo[h] = 0xFFFFFFFFu;
        hi[h] = 0u;
    }
}

// counters of every half segment (one entry more, for the total after the scan) and which segments there are
__global__ void dense_sizes_kernel(const uint32_t* __restrict__ lo, const uint32_t* __restrict__ hi, long long nseg,
                                   unsigned long long* __restrict__ size, uint32_t* __restrict__ present) {
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s <= nseg; s += (long long)gridDim.x * blockDim.x) {
        uint32_t any = 0u;
        for (int g = 0; g < 2; ++g) {
            const long long h = 2 * s + g;
            if (s == nseg) { if (g == 0) size[h] = 0ull; continue; }
            const uint32_t n = lo[h] <= hi[h] ? hi[h] - lo[h] + 1u : 0u;
            size[h] = n;
            any |= n;
        }
        present[s] = any ? 1u : 0u;
    }
}

// most counters of a scale
__global__ void dense_largest_kernel(const unsigned long long* __restrict__ ofs, long long num_scales, int halves, uint32_t* __restrict__ largest) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < num_scales; r += (long long)gridDim.x * blockDim.x)
        atomicMax(largest, (uint32_t)(ofs[(r + 1) * halves] - ofs[r * halves]));
}

struct DenseTotals { unsigned long long counters; uint32_t contexts, most; int lists_bad; };   // most: counters of a scale

__global__ void dense_totals_kernel(const unsigned long long* __restrict__ ofs, const uint32_t* __restrict__ ctx_id, const uint32_t* __restrict__ largest,
                                    long long nseg, UnitLists lists, DenseTotals* __restrict__ totals) {
    totals->lists_bad = lists_verdict(lists);
    totals->counters = ofs[2 * nseg];
    totals->contexts = ctx_id[nseg];
    totals->most = *largest;
}

// Sizes, their running sums and the totals of up to kOffsetsMost segments in one launch: a cluster of eight CTAs, a thread per
// eight segments.  (One kernel for the sizes, two device-wide scans and one more for the largest: 28 us with the gaps.)
constexpr int kOffsetsCtas = 8;
constexpr long long kOffsetsMost = kOffsetsCtas * 1024LL * 8;
__global__ void __cluster_dims__(kOffsetsCtas, 1, 1) __launch_bounds__(1024)
dense_offsets_kernel(const uint32_t* __restrict__ lo, const uint32_t* __restrict__ hi, int nseg, int nctx, unsigned long long* __restrict__ ofs,
                     uint32_t* __restrict__ ctx_id, UnitLists lists, DenseTotals* __restrict__ totals) {
    __shared__ unsigned long long s_sum[32];
    __shared__ uint32_t s_present[32], s_most[32];
    __shared__ DenseTotals s_all;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, me = (int)cluster.block_rank();
    const int g0 = (me * 1024 + tid) * 8;
    const int verdict = me == 0 && tid == 0 ? lists_verdict(lists) : 0;
    uint32_t size[16], present = 0;
    uint32_t sum32 = 0;        // (sixteen ranges of at most 32768 symbols)
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        size[i] = 0u;
        if (g0 + (i >> 1) < nseg) {
            const uint32_t a = lo[2 * g0 + i], b = hi[2 * g0 + i];
            size[i] = a <= b ? b - a + 1u : 0u;
        }
        sum32 += size[i];
        if (i & 1) present += (size[i] | size[i - 1]) ? 1u : 0u;
    }
    // a scale's segments are those of 32 (256 contexts) or 2 (16 contexts) neighbouring threads
    uint32_t scale = sum32;
    for (int o = 1; o < nctx / 8; o <<= 1) scale += __shfl_xor_sync(0xFFFFFFFFu, scale, o);
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, scale);
    unsigned long long at = sum32;
    uint32_t id = present;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, at, o);
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, id, o);
        if (lane >= o) { at += x; id += y; }
    }
    if (lane == 31) { s_sum[w] = at; s_present[w] = id; s_most[w] = most; }
    __syncthreads();
    at -= sum32; id -= present;
    DenseTotals all = {0ull, 0u, 0u, 0};
    for (int i = 0; i < 32; ++i) {
        if (i < w) { at += s_sum[i]; id += s_present[i]; }
        all.counters += s_sum[i]; all.contexts += s_present[i];
        all.most = all.most > s_most[i] ? all.most : s_most[i];
    }
    if (tid == 0) s_all = all;
    cluster.sync();
    DenseTotals total = {0ull, 0u, 0u, 0};
    for (int i = 0; i < kOffsetsCtas; ++i) {
        const DenseTotals q = *cluster.map_shared_rank(&s_all, i);
        if (i < me) { at += q.counters; id += q.contexts; }
        total.counters += q.counters; total.contexts += q.contexts;
        total.most = total.most > q.most ? total.most : q.most;
    }
    cluster.sync();      // (shared memory of the others is read no more)
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int s = g0 + (i >> 1);
        if (s < nseg) {
            ofs[2 * g0 + i] = at;
            if (!(i & 1)) { ctx_id[s] = id; id += (size[i] | size[i + 1]) ? 1u : 0u; }
        }
        at += size[i];
    }
    if (me == 0 && tid == 0) {
        ofs[2LL * nseg] = total.counters;
        ctx_id[nseg] = total.contexts;
        total.lists_bad = verdict;
        *totals = total;
    }
}

template <int V>
__global__ void __launch_bounds__(1024)
dense_count_kernel(DenseGeom d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx, const uint16_t* __restrict__ scales,
                   UnitLists lists, const uint32_t* __restrict__ lo, const unsigned long long* __restrict__ ofs, uint32_t* __restrict__ counters) {
    extern __shared__ uint32_t s_count[];
    __shared__ uint32_t s_base[512];     // counter of symbol 0 of the half segment (modulo 2^32)
    const uint32_t halves = (uint32_t)d.g.nctx * 2u;
    const uint32_t* __restrict__ const unit_sorted = lists.sorted;
    for_stretch(d, scales, lists, [&](uint32_t rk, long long j0, long long j1) {
        const unsigned long long first = ofs[(size_t)rk * halves];
        const uint32_t n = (uint32_t)(ofs[(size_t)(rk + 1u) * halves] - first);
        for (uint32_t h = threadIdx.x; h < halves; h += blockDim.x)
            s_base[h] = (uint32_t)(ofs[(size_t)rk * halves + h] - first) - lo[(size_t)rk * halves + h];
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) s_count[i] = 0u;
        __syncthreads();
        for_pieces<V, 4>(d, sym, ctx, unit_sorted, j0, 0u, (uint32_t)(j1 - j0) * d.unit,
                         [&](uint32_t c, uint32_t v) { atomicAdd(&s_count[s_base[c * 2u + (v >> 15)] + v], 1u); });
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
            if (s_count[i]) atomicAdd(&counters[first + i], s_count[i]);
        __syncthreads();
    });
}

// Counters of a segment from which on all warps of a CTA share it: a context through zero has thousands, and one warp walking
// them while all others are done took most of these two kernels' time (14336 x 4096 FP8: 31 and 45 us).
constexpr uint32_t kDenseShared = 1024;
constexpr int kDenseWarps = 8;

// Distinct symbols of every segment; a warp per segment, eight per CTA.  (distinct[nseg] is set to 0)
__global__ void __launch_bounds__(kDenseWarps * 32)
dense_distinct_kernel(const unsigned long long* __restrict__ ofs, const uint32_t* __restrict__ counters, long long nseg,
                      uint32_t* __restrict__ distinct) {
    __shared__ uint32_t s_sum;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long s0 = (long long)blockIdx.x * kDenseWarps; s0 <= nseg; s0 += (long long)gridDim.x * kDenseWarps) {
        const long long s = s0 + w;
        uint32_t n = 0, size = 0;
        if (s < nseg) {
            const unsigned long long a = ofs[2 * s];
            size = (uint32_t)(ofs[2 * s + 2] - a);
            if (size < kDenseShared) {
#pragma unroll 8
                for (uint32_t i = lane; i < size; i += 32) n += counters[a + i] ? 1u : 0u;
                n = __reduce_add_sync(0xFFFFFFFFu, n);
            }
        }
        if (lane == 0 && s <= nseg && size < kDenseShared) distinct[s] = n;
        if (!__syncthreads_or(size >= kDenseShared)) continue;
        for (long long t = s0; t < s0 + kDenseWarps && t < nseg; ++t) {
            const unsigned long long a = ofs[2 * t];
            const uint32_t all = (uint32_t)(ofs[2 * t + 2] - a);
            if (all < kDenseShared) continue;       // (uniform)
            if (threadIdx.x == 0) s_sum = 0u;
            __syncthreads();
            uint32_t m = 0;
#pragma unroll 8
            for (uint32_t i = threadIdx.x; i < all; i += kDenseWarps * 32) m += counters[a + i] ? 1u : 0u;
            m = __reduce_add_sync(0xFFFFFFFFu, m);
            if (lane == 0) atomicAdd(&s_sum, m);
            __syncthreads();
            if (threadIdx.x == 0) distinct[t] = s_sum;
            __syncthreads();
        }
    }
}

// The items of counters [a + i0, a + i1) of a half segment whose symbols begin at `first`; from place `at` on.  A warp.
__device__ __forceinline__ uint32_t dense_write_items(const uint32_t* __restrict__ counters, unsigned long long a, uint32_t i0, uint32_t i1,
                                                      uint32_t first, uint32_t key, uint32_t at, unsigned long long* __restrict__ items,
                                                      int* __restrict__ counts) {
    const int lane = threadIdx.x & 31;
    constexpr uint32_t UN = 8;       // several loads in flight
    for (; i0 < i1; i0 += 32u * UN) {
        uint32_t c[UN];
#pragma unroll
        for (uint32_t q = 0; q < UN; ++q) {
            const uint32_t i = i0 + 32u * q + lane;
            c[q] = i < i1 ? counters[a + i] : 0u;
        }
#pragma unroll
        for (uint32_t q = 0; q < UN; ++q) {
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, c[q] != 0u);
            if (c[q]) {
                const uint32_t p = at + __popc(mask & ((1u << lane) - 1u));
                items[p] = ((unsigned long long)key << 16) | (first + i0 + 32u * q + lane);
                counts[p] = (int)c[q];
            }
            at += __popc(mask);
        }
    }
    return at;
}

// Counters -> items and counts, in segment order; a warp per segment, eight per CTA.
__global__ void __launch_bounds__(kDenseWarps * 32)
dense_items_kernel(const unsigned long long* __restrict__ ofs, const uint32_t* __restrict__ lo,
                   const uint32_t* __restrict__ counters, const uint32_t* __restrict__ item_ofs,
                   const uint32_t* __restrict__ ctx_id, long long nseg, int nctx, const uint16_t* __restrict__ scale_of_rank,
                   unsigned long long* __restrict__ items, int* __restrict__ counts, int* __restrict__ ctx_ofs,
                   uint32_t* __restrict__ ctx_key) {
    __shared__ uint32_t s_count[kDenseWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (long long s0 = (long long)blockIdx.x * kDenseWarps; s0 < nseg; s0 += (long long)gridDim.x * kDenseWarps) {
        const long long s = s0 + w;
        bool large = false;
        if (s < nseg) {
            uint32_t at = item_ofs[s];
            if (item_ofs[s + 1] != at) {
                const uint32_t key = ((uint32_t)scale_of_rank[s / nctx] << 16) | (uint32_t)(s % nctx), g = ctx_id[s];
                if (lane == 0) { ctx_ofs[g] = (int)at; ctx_key[g] = key; }
                const unsigned long long a = ofs[2 * s], b = ofs[2 * s + 1], c = ofs[2 * s + 2];
                large = c - a >= kDenseShared;
                if (!large) {
                    at = dense_write_items(counters, a, 0u, (uint32_t)(b - a), lo[2 * s], key, at, items, counts);
                    dense_write_items(counters, b, 0u, (uint32_t)(c - b), lo[2 * s + 1], key, at, items, counts);
                }
            }
        }
        if (!__syncthreads_or(large)) continue;
        for (long long t = s0; t < s0 + kDenseWarps && t < nseg; ++t) {
            const unsigned long long a = ofs[2 * t], b = ofs[2 * t + 1], c = ofs[2 * t + 2];
            uint32_t at = item_ofs[t];
            if (c - a < kDenseShared || item_ofs[t + 1] == at) continue;    // (uniform)
            const uint32_t key = ((uint32_t)scale_of_rank[t / nctx] << 16) | (uint32_t)(t % nctx);
            // a stretch of the counters per warp: how many are not zero, then their places
            const uint32_t all = (uint32_t)(c - a), per = ((all + kDenseWarps - 1) / kDenseWarps + 31u) & ~31u;
            const uint32_t i0 = min(w * per, all), i1 = min(i0 + per, all), split = (uint32_t)(b - a);
            uint32_t n = 0;
#pragma unroll 8
            for (uint32_t i = i0 + lane; i < i1; i += 32) n += counters[a + i] ? 1u : 0u;
            n = __reduce_add_sync(0xFFFFFFFFu, n);
            __syncthreads();
            if (lane == 0) s_count[w] = n;
            __syncthreads();
            for (int q = 0; q < w; ++q) at += s_count[q];
            if (i0 < split) at = dense_write_items(counters, a, i0, min(i1, split), lo[2 * t], key, at, items, counts);
            if (i1 > split) dense_write_items(counters, b, max(i0, split) - split, i1 - split, lo[2 * t + 1], key, at, items, counts);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctx_ofs[ctx_id[nseg]] = (int)item_ofs[nseg];
}

}  // namespace hist
}  // namespace mps
