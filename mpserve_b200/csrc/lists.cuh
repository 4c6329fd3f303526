// Bucket lists made on the GPU: the groups of a tensor (rows, or pieces of rows that have a scale of their own) in the
// order (scale, row, column), cut into buckets of at most `cap` groups of one scale -- the ragged layout
// (build_huffman.cu:1353-1392), and the rectangular one of scalar and per-row scales (:611-660).
//
// Bound: launches; a stable sort of 16-bit keys over some 10^5 groups and five passes over as many numbers.
// Made by numpy on the host, the lists took 4.7 of the 6.3 ms that the build of a 4096 x 4096 INT4 weight (131072 groups) then
// took, and 0.2 of the 1.9 ms of a 14336 x 4096 FP8 weight with a scale per row.
#pragma once

#include <cooperative_groups.h>
#include <cub/device/device_radix_sort.cuh>

#include "mps_common.cuh"

namespace mps {
namespace lists {

constexpr int kScaleValues = 65536;

struct Geom {
    long long groups, per_row;      // groups of the tensor, of a row
    long long sb0, nb1;             // two-dimensional scales: rows of a scale block, blocks of a row
    int scale_mode;                 // 0 scalar, 1 per row, 2 per block
};

__global__ void keys_kernel(Geom g, const uint16_t* __restrict__ scales, uint16_t* __restrict__ key, uint32_t* __restrict__ group) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < g.groups; i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / g.per_row, c = i - row * g.per_row;
        key[i] = g.scale_mode == 0 ? scales[0] : (g.scale_mode == 1 ? scales[row] : scales[(row / g.sb0) * g.nb1 + c]);
        group[i] = (uint32_t)i;
    }
}

// first and one past the last group of every scale value (both 0 where it does not occur)
__global__ void runs_kernel(const uint16_t* __restrict__ key, long long groups, uint32_t* __restrict__ first, uint32_t* __restrict__ end) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t v = key[i];
        if (i == 0 || key[i - 1] != v) first[v] = (uint32_t)i;
        if (i == groups - 1 || key[i + 1] != v) end[v] = (uint32_t)i + 1u;
    }
}

// Running sums over the 65536 scale values, by one cluster of eight CTAs, a thread per eight values: of the groups (units of
// work) that have the value, of the values that occur, and of the parts of at most `per_part` groups that a value's are cut
// into.  One entry more in each, the total.  `end` null: `first` holds how many groups a value has.  Outputs that are null
// are left out.  (Three flag or count kernels and as many device-wide scans took 45 us with the gaps between them, this 5.)
constexpr int kScanCtas = 8;
struct ScanTotals { uint32_t parts, scales; };
__global__ void __cluster_dims__(kScanCtas, 1, 1) __launch_bounds__(1024)
scale_scan_kernel(const uint32_t* __restrict__ first, const uint32_t* __restrict__ end, uint32_t per_part, uint32_t* __restrict__ part_base,
                  uint32_t* __restrict__ unit_ofs, uint32_t* __restrict__ unit_cur, uint32_t* __restrict__ rank,
                  uint16_t* __restrict__ scale_of_rank, ScanTotals* __restrict__ totals) {
    static_assert(kScanCtas * 1024 * 8 == kScaleValues, "a thread per eight values");
    __shared__ uint3 s_warp[32];
    __shared__ uint3 s_all;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, me = (int)cluster.block_rank();
    const int v0 = (me * 1024 + tid) * 8;
    uint32_t n[8], parts[8];
    uint3 mine = make_uint3(0u, 0u, 0u);     // groups, values, parts
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        n[i] = end ? end[v0 + i] - first[v0 + i] : first[v0 + i];
        parts[i] = n[i] / per_part + (n[i] % per_part ? 1u : 0u);
        mine.x += n[i]; mine.y += n[i] ? 1u : 0u; mine.z += parts[i];
    }
    uint3 at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, at.x, o), y = __shfl_up_sync(0xFFFFFFFFu, at.y, o), z = __shfl_up_sync(0xFFFFFFFFu, at.z, o);
        if (lane >= o) { at.x += x; at.y += y; at.z += z; }
    }
    if (lane == 31) s_warp[w] = at;
    __syncthreads();
    uint3 all = make_uint3(0u, 0u, 0u);
    at.x -= mine.x; at.y -= mine.y; at.z -= mine.z;
    for (int i = 0; i < 32; ++i) {
        const uint3 q = s_warp[i];
        if (i < w) { at.x += q.x; at.y += q.y; at.z += q.z; }
        all.x += q.x; all.y += q.y; all.z += q.z;
    }
    if (tid == 0) s_all = all;
    cluster.sync();
    uint3 total = make_uint3(0u, 0u, 0u);
    for (int i = 0; i < kScanCtas; ++i) {
        const uint3 q = *cluster.map_shared_rank(&s_all, i);
        if (i < me) { at.x += q.x; at.y += q.y; at.z += q.z; }
        total.x += q.x; total.y += q.y; total.z += q.z;
    }
    cluster.sync();      // (shared memory of the others is read no more)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (part_base) part_base[v0 + i] = at.z;
        if (unit_ofs) unit_ofs[v0 + i] = at.x;
        if (unit_cur) unit_cur[v0 + i] = at.x;
        if (rank) rank[v0 + i] = at.y;
        if (scale_of_rank && n[i]) scale_of_rank[at.y] = (uint16_t)(v0 + i);
        at.x += n[i]; at.y += n[i] ? 1u : 0u; at.z += parts[i];
    }
    if (me == 0 && tid == 0) {
        if (part_base) part_base[kScaleValues] = total.z;
        if (unit_ofs) unit_ofs[kScaleValues] = total.x;
        if (rank) rank[kScaleValues] = total.y;
        totals->parts = total.z;
        totals->scales = total.y;
    }
}

// a warp per scale value: the buckets of its groups
__global__ void buckets_kernel(const uint32_t* __restrict__ first, const uint32_t* __restrict__ end, const uint32_t* __restrict__ base,
                               uint32_t cap, long long groups, uint16_t* __restrict__ bucket_scale, int32_t* __restrict__ bucket_ofs) {
    const int v = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (v >= kScaleValues) return;
    const uint32_t b0 = base[v], n = base[v + 1] - b0;
    for (uint32_t j = lane; j < n; j += 32u) {
        bucket_scale[b0 + j] = (uint16_t)v;
        bucket_ofs[b0 + j] = (int32_t)(first[v] + j * cap);
    }
    if (v == 0 && lane == 0) bucket_ofs[base[kScaleValues]] = (int32_t)groups;
}

__global__ void members_kernel(const uint32_t* __restrict__ sorted, long long groups, uint32_t per_row, uint32_t group_size,
                               int32_t* __restrict__ rows, int32_t* __restrict__ cols) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t g = sorted[i], r = g / per_row;
        rows[i] = (int32_t)r;
        if (cols) cols[i] = (int32_t)((g - r * per_row) * group_size);
    }
}

struct Arrays {     // device workspace
    uint16_t *key, *key_sorted;
    uint32_t *group, *sorted, *first, *end, *base;
    ScanTotals* totals;
    uint8_t* cub;
    size_t cub_bytes, bytes;
};

static inline size_t up(size_t x) { return (x + 255) / 256 * 256; }

static size_t sort_bytes(long long groups) {
    size_t sort = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort, (const uint16_t*)nullptr, (uint16_t*)nullptr, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int)groups, 0, 16);
    return sort;
}

static Arrays carve(uint8_t* ws, long long groups) {
    Arrays a;
    size_t off = 0;
    auto take = [&](size_t bytes) { uint8_t* p = ws + off; off += up(bytes); return p; };
    a.sorted = reinterpret_cast<uint32_t*>(take(groups * 4));
    a.first = reinterpret_cast<uint32_t*>(take(kScaleValues * 4));       // (first and end: one run of memory, zeroed together)
    a.end = reinterpret_cast<uint32_t*>(take(kScaleValues * 4));
    a.base = reinterpret_cast<uint32_t*>(take((kScaleValues + 1) * 4));
    a.totals = reinterpret_cast<ScanTotals*>(take(sizeof(ScanTotals)));
    a.group = reinterpret_cast<uint32_t*>(take(groups * 4));
    a.key = reinterpret_cast<uint16_t*>(take(groups * 2));
    a.key_sorted = reinterpret_cast<uint16_t*>(take(groups * 2));
    a.cub_bytes = sort_bytes(groups);
    a.cub = take(a.cub_bytes);
    a.bytes = off;
    return a;
}

static int grid_of(long long n) {
    long long b = (n + 255) / 256;
    if (b > 148LL * 8) b = 148LL * 8;
    return b < 1 ? 1 : (int)b;
}

}  // namespace lists
}  // namespace mps
