// The order in which a plan's launches take its work items: at their end longest first, made once, when the plan is.
//
// A launch is over when its last SM is, and items differ a hundredfold: a bucket is the rows of a weight that share a
// scale, up to 128 of them.  In the order of the descriptors an SM may take one of the longest when the others have
// nothing left.  Taken longest first, what is left for the end are items of a few steps.  (Plans of up to ten times their
// longest item per SM are sorted all through, kSortedLoad.)  Which items are long stands in device memory (the row
// offsets), so the order is made there; it is a permutation of the items whatever the sidecars hold at that time, and
// only how even the load is depends on it.
//
// Neighbours of equal length keep their order, so that buckets of one scale, whose tables are the same and are staged
// once, stay together; up to kMaxGrab of them make a batch that one CTA takes at once, fewer as the work that is left
// gets less.  Measured, us, in the order of the descriptors | longest first, the next item taken late in both (kTakeLead in
// decode_bucket.cu): nine layers of a tensor-parallel rank's share of a 70B model 1063 | 905 (batches by number of items,
// whatever their length, let one SM run 200 us after the others), an 8B layer 215 | 208.  Made in some 100 us.
#include <cub/cub.cuh>

#include "stream_common.cuh"

namespace mps {

// What an item costs besides its steps, in steps: tables, first chunks, hand-over.
constexpr uint32_t kItemSteps = 40;
constexpr uint32_t kMostSteps = (1u << 24) - 1;
constexpr int kOrderThreads = 1024;
// Only the last items are sorted, this many times the longest one's cost for every SM; what comes before keeps the order of the
// descriptors.  Short items in a row leave preparing the next one no time, and a launch that is sorted all through ends in a run
// of them that grows with it.  us, by number | sorted all through | the end sorted: 8B, 32 layers, 29 times the longest per SM, 5805 |
// 5840 | 5782, 24 layers 4396 | 4387 | 4347; 70B, a tensor-parallel rank of 8, 40 layers 3889 | 3935 | 3870, 20 layers 2001 | 1976 | 1952.
constexpr uint32_t kSortedLoad = 10;

static __device__ __forceinline__ int tensor_of(const int64_t* __restrict__ prefix, int count, long long item) {
    int lo = 0, hi = count;   // largest ti with prefix[ti] <= item
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

struct Totals { unsigned long long all; uint32_t longest; };

// Cost of every item and a hash of its bucket's context -> table map: a warp per item.
__global__ void __launch_bounds__(256)
item_cost_kernel(const mps_bucket_tensor* __restrict__ tensors, const int64_t* __restrict__ prefix, int count, int items, uint32_t span,
                 uint32_t* __restrict__ cost_of, uint32_t* __restrict__ id, uint32_t* __restrict__ maps, Totals* __restrict__ totals) {
    const int item = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (item >= items) return;
    const int ti = tensor_of(prefix, count, item);
    const mps_bucket_tensor& T = tensors[ti];
    const uint32_t chunks = ((uint32_t)T.k + span - 1) / span;
    const long long local = item - prefix[ti], b = local / chunks, t_begin = (local - b * chunks) * span;
    const int contexts = T.mode == 0 ? 256 : 16;
    uint32_t h = 0;
    for (int c = lane; c < contexts; c += 32) h += (uint32_t)T.bucket_table[b * contexts + c] * (2u * (uint32_t)c + 0x9E3779B1u);
    h = __reduce_add_sync(0xFFFFFFFFu, h);
    if (lane) return;
    const long long rows = (long long)T.bucket_row_offsets[b + 1] - T.bucket_row_offsets[b];
    const long long width = T.mode == 2 ? T.group_size : T.bucket_col_len[b];
    uint32_t cost = 0;   // (an item that is not valid is skipped by the decoder)
    if (rows > 0 && width > 0) {
        const unsigned long long elements = (unsigned long long)rows * (unsigned long long)width;
        const unsigned long long steps = elements > (unsigned long long)t_begin ? (elements - t_begin + T.k - 1) / T.k : 0ull;
        cost = (uint32_t)(steps < kMostSteps - kItemSteps ? steps : kMostSteps - kItemSteps) + kItemSteps;
    }
    cost_of[item] = cost;
    id[item] = (uint32_t)item;
    maps[item] = h;
    atomicAdd(&totals->all, (unsigned long long)cost);
    atomicMax(&totals->longest, cost);
}

// What the items are sorted by; one CTA.  Those of the launch's end by their cost, the others first and by number.
__global__ void __launch_bounds__(kOrderThreads)
order_key_kernel(const uint32_t* __restrict__ cost_of, int items, const Totals* __restrict__ totals, uint32_t ctas, uint32_t* __restrict__ key) {
    using SumU64 = cub::BlockScan<unsigned long long, kOrderThreads>;
    __shared__ typename SumU64::TempStorage tmp;
    const unsigned long long all = totals->all, sorted = (unsigned long long)kSortedLoad * ctas * totals->longest;
    unsigned long long done = 0;
    for (int base = 0; base < items; base += kOrderThreads) {
        const int i = base + (int)threadIdx.x;
        const uint32_t cost = i < items ? cost_of[i] : 0u;
        unsigned long long sum, round;
        SumU64(tmp).ExclusiveSum((unsigned long long)cost, sum, round);
        __syncthreads();
        if (i < items) key[i] = all - (done + sum) > sorted ? kMostSteps : cost;
        done += round;
    }
}

// How many items of a cost a batch holds at most, a power of two: so many that it is no more than a share of the work that is
// left, its first item included.
__device__ __forceinline__ uint32_t most_of(unsigned long long left, uint32_t cost, uint32_t ctas) {
    uint32_t most = kMaxGrab;
    while (most > 1u && (unsigned long long)most * kGrabSlack * ctas * (cost ? cost : 1u) > left) most >>= 1;
    return most;
}

// Entries in sorted order and the starts of the batches; one CTA.
__global__ void __launch_bounds__(kOrderThreads)
write_order_kernel(const mps_bucket_tensor* __restrict__ tensors, const int64_t* __restrict__ prefix, int count, int items, uint32_t span,
                   const uint32_t* __restrict__ cost_of, const uint32_t* __restrict__ id, const uint32_t* __restrict__ maps,
                   const Totals* __restrict__ totals, uint32_t ctas, uint32_t* __restrict__ batch_start, uint4* __restrict__ entry) {
    using SumU64 = cub::BlockScan<unsigned long long, kOrderThreads>;
    using ScanU32 = cub::BlockScan<uint32_t, kOrderThreads>;
    __shared__ union { typename SumU64::TempStorage sum; typename ScanU32::TempStorage scan; } tmp;
    const unsigned long long all = totals->all;
    unsigned long long done = 0;        // cost of the items before this round's
    uint32_t run_start = 0, batches = 0;
    for (int base = 0; base < items; base += kOrderThreads) {
        const int i = base + (int)threadIdx.x;
        const bool in = i < items;
        uint32_t cost = 0, cost_before = 0, item = 0, map = 0;
        int ti = -1, before = -1;
        uint32_t map_before = 0;
        if (in) {
            item = id[i]; cost = cost_of[item]; map = maps[item];
            ti = tensor_of(prefix, count, item);
            const uint32_t chunks = ((uint32_t)tensors[ti].k + span - 1) / span;
            const long long local = item - prefix[ti], b = local / chunks;
            entry[i] = make_uint4((uint32_t)ti, (uint32_t)b, (uint32_t)(local - b * chunks) * span, 0u);
            if (i > 0) {
                const uint32_t other = id[i - 1];
                cost_before = cost_of[other];
                before = tensor_of(prefix, count, other);
                map_before = maps[other];
            }
        }
        unsigned long long sum, round;
        SumU64(tmp.sum).ExclusiveSum((unsigned long long)cost, sum, round);
        __syncthreads();
        // first item of the run of equal tables and equal `most` that this one is in: the most falls where the work that is
        // left does and rises where items get shorter, and an item of the one does not lead a batch of the other
        const unsigned long long left = all - (done + sum);
        const uint32_t most = most_of(left, cost, ctas);
        uint32_t start = (in && (ti != before || map != map_before || most != most_of(left + cost_before, cost_before, ctas))) ? (uint32_t)i : 0u;
        uint32_t start_max;
        ScanU32(tmp.scan).InclusiveScan(start, start, cub::Max(), start_max);
        start = start > run_start ? start : run_start;
        run_start = run_start > start_max ? run_start : start_max;
        __syncthreads();
        // every multiple of it, counted from the run's first item, starts a batch
        uint32_t lead = in && ((uint32_t)i - start) % most == 0u ? 1u : 0u, pos, leads;
        ScanU32(tmp.scan).ExclusiveSum(lead, pos, leads);
        __syncthreads();
        if (lead) batch_start[batches + pos] = (uint32_t)i;
        batches += leads;
        done += round;
    }
    for (int i = (int)batches + (int)threadIdx.x; i <= items; i += kOrderThreads) batch_start[i] = (uint32_t)items;
}

struct OrderScratch {
    uint32_t *cost, *key, *key_sorted, *id, *id_sorted, *maps;
    Totals* totals;
    void* cub;
    size_t cub_bytes, bytes;
};

static cudaError_t order_scratch(void* base, long long items, OrderScratch* s) {
    const size_t words = ((size_t)items * 4 + 255) & ~(size_t)255;
    uint8_t* p = static_cast<uint8_t*>(base);
    auto take = [&](size_t bytes) { uint8_t* q = p; p += bytes; return q; };
    s->totals = reinterpret_cast<Totals*>(take(256));
    s->cost = reinterpret_cast<uint32_t*>(take(words));
    s->key = reinterpret_cast<uint32_t*>(take(words));
    s->key_sorted = reinterpret_cast<uint32_t*>(take(words));
    s->id = reinterpret_cast<uint32_t*>(take(words));
    s->id_sorted = reinterpret_cast<uint32_t*>(take(words));
    s->maps = reinterpret_cast<uint32_t*>(take(words));
    s->cub = p;
    s->cub_bytes = 0;
    const cudaError_t e = cub::DeviceRadixSort::SortPairsDescending(nullptr, s->cub_bytes, s->key, s->key_sorted, s->id, s->id_sorted,
                                                                    (int)items, 0, 24, (cudaStream_t)0);
    s->bytes = (size_t)(p - static_cast<uint8_t*>(base)) + s->cub_bytes;
    return e;
}

}  // namespace mps

using namespace mps;

extern "C" {

size_t mps_bucket_batch_order_bytes(int64_t total_items) {
    return total_items <= 0 || total_items > MPS_ORDER_MAX_ITEMS ? 0 : order_batch_bytes(total_items) + (size_t)total_items * sizeof(uint4);
}

size_t mps_bucket_batch_order_scratch_bytes(int64_t total_items) {
    if (total_items <= 0 || total_items > MPS_ORDER_MAX_ITEMS) return 0;
    OrderScratch s;
    return order_scratch(nullptr, total_items, &s) == cudaSuccess ? s.bytes : 0;
}

int mps_bucket_batch_order(const mps_bucket_tensor* tensors_dev, const int64_t* item_prefix_dev, int count, int64_t total_items,
                           int32_t threads, int32_t chains, void* order_dev, size_t order_bytes, void* scratch, size_t scratch_bytes,
                           void* stream) {
    if (!tensors_dev || !item_prefix_dev || count <= 0 || threads <= 0 || chains <= 0 || !order_dev || !scratch ||
        ((reinterpret_cast<uintptr_t>(order_dev) & 15u) | (reinterpret_cast<uintptr_t>(scratch) & 255u)) != 0) {
        set_error("mps_bucket_batch_order: bad arguments");
        return MPS_ERR_INVALID;
    }
    if (total_items <= 0 || total_items > MPS_ORDER_MAX_ITEMS) { set_error("mps_bucket_batch_order: too few or too many work items"); return MPS_ERR_INVALID; }
    OrderScratch s;
    MPS_CUDA_TRY(order_scratch(scratch, total_items, &s));
    if (order_bytes < mps_bucket_batch_order_bytes(total_items) || scratch_bytes < s.bytes) {
        set_error("mps_bucket_batch_order: buffer too small");
        return MPS_ERR_WORKSPACE;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t span = (uint32_t)threads * (uint32_t)chains;
    const int items = (int)total_items;
    MPS_CUDA_TRY(cudaMemsetAsync(s.totals, 0, sizeof(*s.totals), st));
    item_cost_kernel<<<(unsigned)((items + 7) / 8), 256, 0, st>>>(tensors_dev, item_prefix_dev, count, items, span, s.cost, s.id, s.maps, s.totals);
    order_key_kernel<<<1, kOrderThreads, 0, st>>>(s.cost, items, s.totals, (uint32_t)sm_count(), s.key);
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cub::DeviceRadixSort::SortPairsDescending(s.cub, s.cub_bytes, s.key, s.key_sorted, s.id, s.id_sorted, items, 0, 24, st));
    write_order_kernel<<<1, kOrderThreads, 0, st>>>(tensors_dev, item_prefix_dev, count, items, span, s.cost, s.id_sorted, s.maps, s.totals,
                                                    (uint32_t)sm_count(), static_cast<uint32_t*>(order_dev),
                                                    reinterpret_cast<uint4*>(static_cast<uint8_t*>(order_dev) + order_batch_bytes(items)));
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

}  // extern "C"
