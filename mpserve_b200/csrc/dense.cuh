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
// Measured: finding ranges, counting and writing items of a 14336 x 4096 FP8 weight per channel 0.28 ms (the general form
// 0.77), of a 4096 x 4096 INT4 weight by group 0.19 (0.54).
#pragma once

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
// each, as stragglers).  Its threads walk the quads (four neighbouring elements) of the stretch.
struct DenseGeom {
    Geom g;
    const uint32_t* first;           // first unit of every stretch, [0, *count)
    const uint32_t* count;
    uint32_t upc;
    uint32_t quads_row, quads_unit;  // quads of a unit's row, of a unit
};

// f(context, symbol) of quads [first, last) of units j0 and on, UN quads of a thread in flight
template <int UN, class F>
__device__ __forceinline__ void for_quads(const DenseGeom& d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx,
                                          const uint32_t* __restrict__ unit_sorted, long long j0, uint32_t first, uint32_t last, F&& f) {
    for (uint32_t q0 = first + threadIdx.x; q0 < last; q0 += UN * blockDim.x) {
        uint32_t cw[UN];
        uint2 sw[UN];
        bool in[UN];
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            const uint32_t q = q0 + i * blockDim.x;
            in[i] = q < last;
            long long at = 0;
            if (in[i]) {
                const uint32_t j = q / d.quads_unit, w = q - j * d.quads_unit;
                const uint32_t u = unit_sorted[j0 + j];
                // (uniform shortcuts: a unit per row, one row per unit)
                const uint32_t bi = d.g.nbu1 == 1 ? u : u / (uint32_t)d.g.nbu1, bj = u - bi * (uint32_t)d.g.nbu1;
                const uint32_t r = d.g.ub0 == 1 ? 0u : w / d.quads_row, c4 = w - r * d.quads_row;
                const long long row = (long long)bi * d.g.ub0 + r, col = (long long)bj * d.g.ub1 + 4u * c4;
                in[i] = row < d.g.n && col < d.g.m;     // (both are multiples of four)
                at = row * d.g.m + col;
            }
            cw[i] = in[i] ? *reinterpret_cast<const uint32_t*>(ctx + at) : 0u;
            sw[i] = in[i] ? *reinterpret_cast<const uint2*>(sym + at) : make_uint2(0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < UN; ++i) {
            if (!in[i]) continue;
            const uint32_t m = d.g.ctx_mask;
            f(cw[i] & m, sw[i].x & 0xFFFFu);
            f((cw[i] >> 8) & m, sw[i].x >> 16);
            f((cw[i] >> 16) & m, sw[i].y & 0xFFFFu);
            f((cw[i] >> 24) & m, sw[i].y >> 16);
        }
    }
}

// stretches of every scale value; one entry more, for the total after the scan
__global__ void dense_stretches_kernel(const uint32_t* __restrict__ per_scale, uint32_t upc, uint32_t* __restrict__ count) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v <= kScaleValues) count[v] = v < kScaleValues ? (per_scale[v] + upc - 1u) / upc : 0u;
}

__global__ void dense_stretch_fill_kernel(const uint32_t* __restrict__ base, const uint32_t* __restrict__ unit_ofs, uint32_t upc,
                                          uint32_t* __restrict__ first) {
    const int v = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (v >= kScaleValues) return;
    const uint32_t b = base[v], n = base[v + 1] - b;
    for (uint32_t j = lane; j < n; j += 32u) first[b + j] = unit_ofs[v] + j * upc;
}

// Calls f(rank, first unit, end) for the CTA's stretch, if it has one.  (uniform)
template <class F>
__device__ __forceinline__ void for_stretch(const DenseGeom& d, const uint16_t* __restrict__ scales, const uint32_t* __restrict__ rank,
                                            const uint32_t* __restrict__ unit_ofs, const uint32_t* __restrict__ unit_sorted, F&& f) {
    if (blockIdx.x >= *d.count) return;
    const uint32_t j = d.first[blockIdx.x];
    const uint32_t v = unit_scale(d.g, scales, unit_sorted[j]);
    const uint32_t past = unit_ofs[v + 1];          // the list is ordered by scale
    f(rank[v], (long long)j, (long long)(j + d.upc < past ? j + d.upc : past));
}

// lo / hi of half segment h: [rank * nctx * 2 + context * 2 + sign], preset to 0xFFFFFFFF and 0
__global__ void __launch_bounds__(kDenseThreads)
dense_range_kernel(DenseGeom d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx, const uint16_t* __restrict__ scales,
                   const uint32_t* __restrict__ rank, const uint32_t* __restrict__ unit_ofs, const uint32_t* __restrict__ unit_sorted,
                   uint32_t* __restrict__ lo, uint32_t* __restrict__ hi) {
    __shared__ uint2 s_range[512];       // smallest, largest symbol
    const uint32_t halves = (uint32_t)d.g.nctx * 2u;
    for_stretch(d, scales, rank, unit_ofs, unit_sorted, [&](uint32_t rk, long long j0, long long j1) {
        for (uint32_t h = threadIdx.x; h < halves; h += kDenseThreads) s_range[h] = make_uint2(0xFFFFFFFFu, 0u);
        __syncthreads();
        auto widen = [&](uint32_t c, uint32_t v) {
            const uint32_t h = c * 2u + (v >> 15);
            // (a stale range only costs an atomic too many)
            uint2 r;
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"((uint32_t)__cvta_generic_to_shared(&s_range[h])));
            if (v < r.x) atomicMin(&s_range[h].x, v);
            if (v > r.y) atomicMax(&s_range[h].y, v);
        };
        // a first quad per thread by itself: against empty ranges every element is an atomic, against those of two
        // thousand elements few are
        const uint32_t total = (uint32_t)(j1 - j0) * d.quads_unit, few = total < kDenseThreads ? total : kDenseThreads;
        for_quads<1>(d, sym, ctx, unit_sorted, j0, 0u, few, widen);
        __syncthreads();
        for_quads<4>(d, sym, ctx, unit_sorted, j0, few, total, widen);
        __syncthreads();
        for (uint32_t h = threadIdx.x; h < halves; h += kDenseThreads) {
            const uint2 r = s_range[h];
            if (r.x <= r.y) {
                atomicMin(&lo[(size_t)rk * halves + h], r.x);
                atomicMax(&hi[(size_t)rk * halves + h], r.y);
            }
        }
        __syncthreads();
    });
}

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

__global__ void __launch_bounds__(1024)
dense_count_kernel(DenseGeom d, const uint16_t* __restrict__ sym, const uint8_t* __restrict__ ctx, const uint16_t* __restrict__ scales,
                   const uint32_t* __restrict__ rank, const uint32_t* __restrict__ unit_ofs, const uint32_t* __restrict__ unit_sorted,
                   const uint32_t* __restrict__ lo, const unsigned long long* __restrict__ ofs, uint32_t* __restrict__ counters) {
    extern __shared__ uint32_t s_count[];
    __shared__ uint32_t s_base[512];     // counter of symbol 0 of the half segment (modulo 2^32)
    const uint32_t halves = (uint32_t)d.g.nctx * 2u;
    for_stretch(d, scales, rank, unit_ofs, unit_sorted, [&](uint32_t rk, long long j0, long long j1) {
        const unsigned long long first = ofs[(size_t)rk * halves];
        const uint32_t n = (uint32_t)(ofs[(size_t)(rk + 1u) * halves] - first);
        for (uint32_t h = threadIdx.x; h < halves; h += blockDim.x)
            s_base[h] = (uint32_t)(ofs[(size_t)rk * halves + h] - first) - lo[(size_t)rk * halves + h];
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) s_count[i] = 0u;
        __syncthreads();
        for_quads<4>(d, sym, ctx, unit_sorted, j0, 0u, (uint32_t)(j1 - j0) * d.quads_unit,
                     [&](uint32_t c, uint32_t v) { atomicAdd(&s_count[s_base[c * 2u + (v >> 15)] + v], 1u); });
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
            if (s_count[i]) atomicAdd(&counters[first + i], s_count[i]);
        __syncthreads();
    });
}

// Distinct symbols of every segment; a warp per segment.  (distinct[nseg] is set to 0)
__global__ void dense_distinct_kernel(const unsigned long long* __restrict__ ofs, const uint32_t* __restrict__ counters, long long nseg,
                                      uint32_t* __restrict__ distinct) {
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s <= nseg; s += warps) {
        uint32_t n = 0;
        if (s < nseg) {
            const unsigned long long a = ofs[2 * s], b = ofs[2 * s + 2];
            #pragma unroll 8
            for (unsigned long long i = a + lane; i < b; i += 32) n += counters[i] ? 1u : 0u;
            n = __reduce_add_sync(0xFFFFFFFFu, n);
        }
        if (lane == 0) distinct[s] = n;
    }
}

// Counters -> items and counts, in segment order; a warp per segment.
__global__ void dense_items_kernel(const unsigned long long* __restrict__ ofs, const uint32_t* __restrict__ lo,
                                   const uint32_t* __restrict__ counters, const uint32_t* __restrict__ item_ofs,
                                   const uint32_t* __restrict__ ctx_id, long long nseg, int nctx, const uint16_t* __restrict__ scale_of_rank,
                                   unsigned long long* __restrict__ items, int* __restrict__ counts, int* __restrict__ ctx_ofs,
                                   uint32_t* __restrict__ ctx_key) {
    const int lane = threadIdx.x & 31;
    const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long s = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nseg; s += warps) {
        uint32_t at = item_ofs[s];
        if (item_ofs[s + 1] == at) continue;
        const uint32_t key = ((uint32_t)scale_of_rank[s / nctx] << 16) | (uint32_t)(s % nctx), g = ctx_id[s];
        if (lane == 0) { ctx_ofs[g] = (int)at; ctx_key[g] = key; }
        for (int half = 0; half < 2; ++half) {
            const long long h = 2 * s + half;
            const unsigned long long a = ofs[h];
            const uint32_t n = (uint32_t)(ofs[h + 1] - a), first = lo[h];
            constexpr uint32_t UN = 8;       // (a context through zero has thousands of counters: several loads in flight)
            for (uint32_t i0 = 0; i0 < n; i0 += 32u * UN) {
                uint32_t c[UN];
#pragma unroll
                for (uint32_t q = 0; q < UN; ++q) {
                    const uint32_t i = i0 + 32u * q + lane;
                    c[q] = i < n ? counters[a + i] : 0u;
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
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctx_ofs[ctx_id[nseg]] = (int)item_ofs[nseg];
}

}  // namespace hist
}  // namespace mps
