// Pieces shared by the persistent decode kernels: launch arguments, the work item a scout warp
// prepares, and thin wrappers over the sm_100a instructions they are built from (mbarrier,
// cp.async, cp.async.bulk without tensor map or multicast, named barriers, cache-hinted prefetch).
#pragma once

#include "mps_common.cuh"

namespace mps {

struct BatchArgs {
    mps_bucket_tensor single;            // used when tensors == nullptr
    const mps_bucket_tensor* tensors;    // device array, or nullptr
    const int64_t* item_prefix;          // device [count+1], or nullptr (single tensor)
    const uint32_t* batch_start;         // device [total_items + 1]: batches of items in `order`, or nullptr (items by number)
    const uint4* order;                  // device [total_items]: tensor, bucket, first sub-stream
    int count;
    int total_items;
    int stall_block_plus1;               // self-test only: the producer leaves block (this - 1) of steps out; 0: never
    uint32_t spin_limit;                 // polls before a wait gives up; 0: kSpinLimit
};

// ------------------------------------------------------------------------------------------------
// Work item prepared one item ahead by the scout warp, so that the decoding warps start every item
// with its geometry and row bases already in shared memory and its tables already on their way
// into L2 instead of walking a chain of dependent global loads.
// ------------------------------------------------------------------------------------------------
struct Prepared {
    int valid;  // 0: the queue is empty
    int ok;     // geometry usable, else the item is skipped
    int ti, mode;
    uint32_t k, k_eff, t_begin, ebits;
    long long b, total, wb;
    int32_t row_a, nrows, col_start, col_len;   // (int32 in the sidecar)
    int rows_ok, rows_vec, rows_al16;
    uint32_t bit_lo;  // low six bits of the bucket's bit base (0 in every sidecar the reference encoder writes)
    // tables: must they be staged (another context -> table map than the item decoded before), and are they
    // one run of consecutive table ids in context order (the reference encoder numbers tables by (scale, context))
    int16_t restage, tab_dense;
    int32_t tab_first;   // table id of the first context that has one
    uint32_t tab_count;  // contexts that have one
};

struct BitOrigin {        // bitstream of the item seen from a 16-byte aligned origin
    const uint8_t* base;  // 16-byte aligned
    uint32_t last_ofs;    // largest 16-byte aligned offset whose chunk lies wholly inside the bitstream
    uint32_t tail_ofs;    // offset of a final 8-byte half chunk (bitstream ends mid-chunk), else 0xFFFFFFFF
    uint32_t bit_delta;   // bits between the origin and the bucket's first bit
};

// Geometry of one work item on the streaming path (uniform across the CTA).
struct StreamItem {
    const uint8_t* ctx_bytes;
    uint16_t* out;
    const uint32_t* startbit;
    const uint32_t* rowbase;
    BitOrigin bo;
    uint32_t t_begin, k_eff, col_len;
    uint32_t nsteps;       // steps of this item, a ragged last one included
    uint32_t nfull;        // steps in which every sub-stream of the bucket has an element
    uint32_t last_active;  // local sub-streams that have an element in the ragged last step (0: there is none)
    uint32_t flat_bytes;   // != 0: the bucket's whole bitstream, this many bytes from bo.base, is copied into shared memory
    uint32_t nrows;        // rows (groups) of the bucket
};

constexpr uint32_t kSpinLimit = 1u << 22;  // bounded waits: give up, flag, return
constexpr int kMaxGrab = 8;          // most work items one CTA takes from the queue at once
constexpr int kGrabSlack = 4;        // a grab is at most 1/(kGrabSlack * CTAs) of what is left

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2::evict_last [%0];" ::"l"(p)); }

// barrier 1 (decoding threads only) with an OR reduction
__device__ __forceinline__ int group_or(int pred, int nthreads) {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"(pred), "r"(nthreads) : "memory");
    return r;
}
__device__ __forceinline__ void group_sync(int nthreads) { asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory"); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Returns false when the barrier did not complete within `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = kSpinLimit) {
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t lds_ordered(uint32_t addr) {  // ordered with the async copies
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// The buckets of a lone tensor, longest first: a launch of more items than CTAs is over when its last SM is, so what is
// left for its end must be short (a plan's items are ordered when it is made, plan_order.cu).  All NW warps of a CTA call
// this at its start, every CTA with the same result: a stable counting sort by length in classes of an eighth of an octave,
// `order[i]` the i-th bucket.  `hist`: NW * 128 words of scratch.  It takes 1.7 us.  What is gained: orders_itself.
constexpr int kOrderMost = 1792;    // buckets: shared memory has no room for more (28672 x 8192, 2240: 522 us by number)
template <int NW>
__device__ __forceinline__ void order_by_length(const mps_bucket_tensor& T, uint32_t* hist, uint16_t* order) {
    constexpr int kRounds = (kOrderMost + NW * 32 - 1) / (NW * 32);     // of 32 buckets per warp
    const int B = (int)T.num_buckets, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = ((B + NW - 1) / NW + 31) & ~31, begin = warp * per;
    uint32_t cls[kRounds];
#pragma unroll
    for (int j = 0; j < kRounds; ++j) {
        const int b = begin + 32 * j + lane;
        cls[j] = 128u;      // none
        if (32 * j < per && b < B) {
            const float rows = (float)(T.bucket_row_offsets[b + 1] - T.bucket_row_offsets[b]);
            const float width = (float)(T.mode == 2 ? T.group_size : T.bucket_col_len[b]);
            const float steps = rows * width / (float)T.k + 1.f;
            const int c = (int)(__float_as_uint(steps > 1.f ? steps : 1.f) >> 20) - (127 << 3);
            cls[j] = c < 127 ? 127u - (uint32_t)c : 0u;     // (ascending: longest first)
        }
    }
    for (int i = threadIdx.x; i < NW * 128; i += NW * 32) hist[i] = 0u;
    __syncthreads();
    uint32_t* mine = hist + warp * 128;
    uint32_t same[kRounds];        // lanes of the round with the same class
#pragma unroll
    for (int j = 0; j < kRounds; ++j) {
        same[j] = 0u;
        if (32 * j < per) {             // (uniform)
            same[j] = __match_any_sync(0xFFFFFFFFu, cls[j]);
            if (cls[j] < 128u && lane == __ffs((int)same[j]) - 1) mine[cls[j]] += (uint32_t)__popc(same[j]);
            __syncwarp();
        }
    }
    __syncthreads();
    // starts of every (class, warp): a warp per 32 classes, each adding up what the classes before its own hold
    if (warp < 4) {
        uint32_t carry = 0, count[NW], sum = 0;
        for (int c = lane; c < 32 * warp; c += 32)
#pragma unroll
            for (int w = 0; w < NW; ++w) carry += hist[w * 128 + c];
        carry = __reduce_add_sync(0xFFFFFFFFu, carry);
#pragma unroll
        for (int w = 0; w < NW; ++w) { count[w] = hist[w * 128 + 32 * warp + lane]; sum += count[w]; }
        uint32_t at = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, at, o);
            if (lane >= o) at += v;
        }
        at += carry - sum;
#pragma unroll
        for (int w = 0; w < NW; ++w) { const uint32_t c = count[w]; count[w] = at; at += c; }
        asm volatile("bar.sync 1, 128;" ::: "memory");      // (the sums above have been read)
#pragma unroll
        for (int w = 0; w < NW; ++w) hist[w * 128 + 32 * warp + lane] = count[w];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRounds; ++j) {
        if (32 * j < per) {
            if (cls[j] < 128u) {
                const uint32_t at = mine[cls[j]] + (uint32_t)__popc(same[j] & ((1u << lane) - 1u));
                order[at] = (uint16_t)(begin + 32 * j + lane);
            }
            __syncwarp();
            if (cls[j] < 128u && lane == __ffs((int)same[j]) - 1) mine[cls[j]] += (uint32_t)__popc(same[j]);
            __syncwarp();
        }
    }
    __syncthreads();
}
// Builders list buckets by scale, and the scales of a weight are many in the middle of their range and few at its ends: in
// the order of their numbers the long buckets begin in the first wave and the short ones are left for the last.  Longest first pays
// where buckets are so many that the middle is not reached at once, and short of a launch's time, as the parts of at most a
// thousand groups that by-scale sidecars are cut into; two long ones that share an SM slow each other.  Measured, us, by number |
// longest first: by scale, k = 256, 512 x 4096 (324 buckets) 20.3 | 22.9, 2048 38 | 42, 4096 (460) 61.0 | 62.8, 5000 79 | 67,
// 8192 (615) 98 | 93, 14336 (825) 160 | 146; parts of a bucket (k = 1024) 2048 50.6 | 53.2, 14336 178.5 | 182; FP8 buckets of
// up to 128 rows, heavy tails, 4096 x 3000 53 | 61, 8192 x 3000 90 | 105, 14336 x 1024 50 | 58.
constexpr long long kOrderLoad = 256;      // steps for every place of the GPU
inline bool orders_itself(const BatchArgs& args, int grid, int span) {
    const mps_bucket_tensor& T = args.single;
    return args.tensors == nullptr && T.mode == 2 && T.k <= span && T.num_buckets > grid && T.num_buckets <= kOrderMost &&
           T.n * T.m >= kOrderLoad * grid * T.k;
}

// CH context bytes of one step, as the decoding thread loads them from the ring
template <int CH> struct Ctx;
template <> struct Ctx<1> {
    using T = uint32_t;
    static __device__ __forceinline__ T ld(const uint8_t* p) { return ld_stream_u8(p); }
    static __device__ __forceinline__ uint32_t byte(T v, int) { return v; }
};
template <> struct Ctx<2> {
    using T = uint32_t;
    static __device__ __forceinline__ T ld(const uint8_t* p) { return ld_stream_u16(p); }
    static __device__ __forceinline__ uint32_t byte(T v, int c) { return __byte_perm(v, 0u, 0x4440u | (uint32_t)c); }
};
template <> struct Ctx<4> {
    using T = uint32_t;
    static __device__ __forceinline__ T ld(const uint8_t* p) { return ld_stream_u32(p); }
    static __device__ __forceinline__ uint32_t byte(T v, int c) { return __byte_perm(v, 0u, 0x4440u | (uint32_t)c); }
};
template <> struct Ctx<8> {
    using T = uint2;
    static __device__ __forceinline__ T ld(const uint8_t* p) { return ld_stream_u64(p); }
    static __device__ __forceinline__ uint32_t byte(T v, int c) { return __byte_perm((c < 4) ? v.x : v.y, 0u, 0x4440u | (uint32_t)(c & 3)); }
};

template <int CH>
__device__ __forceinline__ typename Ctx<CH>::T lds_ctx(uint32_t addr) {
    if constexpr (CH == 8) {
        uint2 v;
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
        return v;
    } else {
        uint32_t v;
        if constexpr (CH == 4) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
        else if constexpr (CH == 2) asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
        else asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
        return v;
    }
}

// Where the items lie in the memory of an order (plan_order.cu): after the starts of the batches.
inline size_t order_batch_bytes(long long items) { return ((size_t)(items + 1) * 4 + 15) & ~(size_t)15; }

// SM count of the current device (148 on B200), remembered per device.
inline int sm_count() {
    static int cached[64] = {0};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
        cached[dev] = n;
    }
    return cached[dev];
}

}  // namespace mps
