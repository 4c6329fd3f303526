// Bucket lists made on the GPU: the groups of a tensor (rows, or pieces of rows that have a scale of their own) in the
// order (scale, row, column), cut into buckets of at most `cap` groups of one scale -- the ragged layout
// (build_huffman.cu:1353-1392), and the rectangular one of scalar and per-row scales (:611-660).
//
// Bound: launches; a stable sort of 16-bit keys over some 10^5 groups and five passes over as many numbers.
// Made by numpy on the host, the lists took 4.7 of the 6.3 ms that the build of a 4096 x 4096 INT4 weight (131072 groups) then
// took, and 0.2 of the 1.9 ms of a 14336 x 4096 FP8 weight with a scale per row.
#pragma once

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

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

// buckets of every scale value; one entry more, for the total after the scan
__global__ void counts_kernel(const uint32_t* __restrict__ first, const uint32_t* __restrict__ end, uint32_t cap, uint32_t* __restrict__ buckets) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < kScaleValues) {
        const uint32_t n = end[v] - first[v];
        buckets[v] = n / cap + (n % cap ? 1u : 0u);
    } else if (v == kScaleValues) {
        buckets[v] = 0u;
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
    uint8_t* cub;
    size_t cub_bytes, bytes;
};

static inline size_t up(size_t x) { return (x + 255) / 256 * 256; }

static size_t sort_bytes(long long groups) {
    size_t sort = 0, scan = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort, (const uint16_t*)nullptr, (uint16_t*)nullptr, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int)groups, 0, 16);
    cub::DeviceScan::ExclusiveSum(nullptr, scan, (const uint32_t*)nullptr, (uint32_t*)nullptr, kScaleValues + 1);
    return sort > scan ? sort : scan;
}

static Arrays carve(uint8_t* ws, long long groups) {
    Arrays a;
    size_t off = 0;
    auto take = [&](size_t bytes) { uint8_t* p = ws + off; off += up(bytes); return p; };
    a.sorted = reinterpret_cast<uint32_t*>(take(groups * 4));
    a.first = reinterpret_cast<uint32_t*>(take(kScaleValues * 4));       // (first and end: one run of memory, zeroed together)
    a.end = reinterpret_cast<uint32_t*>(take(kScaleValues * 4));
    a.base = reinterpret_cast<uint32_t*>(take((kScaleValues + 1) * 4));
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
