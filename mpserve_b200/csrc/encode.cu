// GPU builder of the Huffman sidecar: replaces the single-threaded CPU encoder of the reference
// (kernel/build_huffman.cu) with device passes that produce byte-identical artifacts.
//
//   analyze    the histogram of every context (build_huffman.cu:392-412), contexts in ascending key
//              order: a counter per symbol of every context's range where those are few (dense.cuh), else a
//              two-level count, by scale and then by context (histogram.cuh); no sort over the elements
//   codebooks  per context: order by (count, symbol), ESC reduction when there are more symbols than
//              table slots (:479-535), length-limited code lengths (package-merge, :46-118), canonical
//              codes in item order (:171-203), lookup-table fill and 4-bit length packing (:205-239);
//              a warp or a CTA per context (codebook.cuh)
//   layout     the code of every element, stored in bucket order, bits of every sub-stream, prefix sums per
//              bucket, 64-bit aligned bucket bases (:811-879); a CTA per range of neighbouring sub-streams
//   emit       the stored codes assembled MSB-first in shared memory and written out word by word (:881-911)
//              (layout.cuh; the shared-table layout, below, goes element by element with atomics)
//
// Device-wide scans, and the sorts of the shared-table layout and of the bucket lists, use CUB from the CUDA
// toolkit; everything else is written here.  Bucket lists come from the scale tensor: sorted ones from lists.cuh, those of
// rectangular scale blocks, which need no sort, from the caller (mpserve_b200/encoder.py).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <string.h>

#include "codebook.cuh"
#include "dense.cuh"
#include "histogram.cuh"
#include "layout.cuh"
#include "lists.cuh"
#include "mps_common.cuh"

namespace mps {

// ------------------------------------------------------------------------------------------------
// build state: where things live inside the caller's workspace (host-side POD, opaque to callers)
// ------------------------------------------------------------------------------------------------
struct BuildState {
    int64_t numel, n, m;
    int64_t N;                 // distinct (context, symbol) pairs
    int64_t G;                 // contexts
    int32_t L, variant;
    int32_t group_size, pad_;  // elements per group of the ragged layout
    uint8_t* ws;               // device workspace base
    size_t ws_bytes;
    // offsets (bytes) into ws
    size_t o_items;            // uint64 [N]  scale<<32 | ctx<<16 | sym, ascending
    size_t o_counts;           // int32  [N]
    size_t o_ctx_ofs;          // int32  [G+1] first item of each context
    size_t o_ctx_key;          // uint32 [G]   scale<<16 | ctx
    size_t o_enc;              // uint32 [N]   len<<16 | code of each item, 0 = not coded (ESC'd)
    size_t o_esc;              // uint32 [G]   len<<16 | code of the context's ESC code (0: none)
    size_t o_escsym;           // uint16 [G]
    size_t o_scratch;          // start of the reusable scratch area
    size_t scratch_bytes;
    int32_t* d_flag;           // device error flags (first words of ws): of the layout, of the codebooks, of the lists; at +64 bytes its Totals
    // shared-table layout only (carved from the scratch area by the shared-table calls)
    int64_t num_scales, num_chunks;
    size_t o_sh_keep;          // start of what the layout call leaves for the emit call
    size_t o_sh_end;           // end of it
    // rectangular buckets: what the layout call leaves in the scratch area for the emit call
    size_t o_rect_codes;       // uint16 or uint32 [numel] code of every element, in bucket order (layout.cuh)
    size_t o_rect_ebase;       // uint64 [B+1]   first element of every bucket in that order
    size_t o_rect_part;        // uint32         bits in front of every team's stretch
    int64_t rect_buckets;      // B of the layout call (0: nothing in the scratch area for an emit call)
    int32_t rect_k;            // k of the layout call
    int8_t rect_ragged, rect_vec, pad2_[2];   // ragged buckets; rows and sub-streams come in fours
};
static_assert(sizeof(BuildState) <= 256, "mps_build_state is 256 bytes");

static inline size_t align_up(size_t x, size_t a = 256) { return (x + a - 1) / a * a; }

// SM count of the current device (148 on B200)
static int sm_count_host() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    return n;
}

static int grid_for(long long n, int threads = 256) {
    long long b = (n + threads - 1) / threads;
    if (b > 148LL * 32) b = 148LL * 32;
    if (b < 1) b = 1;
    return (int)b;
}

// ------------------------------------------------------------------------------------------------
// bucket tables, layout, emit (rectangular buckets: FP8 and AWQ bucket builders)
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int find_u32(const uint32_t* __restrict__ a, int n, uint32_t key) {
    int lo = 0, hi = n - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const uint32_t v = a[mid];
        if (v == key) return mid;
        if (v < key) lo = mid + 1; else hi = mid - 1;
    }
    return -1;
}

// context -> table id of every bucket (build_huffman.cu:737-746)
__global__ void bucket_table_kernel(const uint32_t* __restrict__ ctx_key, int G, const uint16_t* __restrict__ bucket_scale,
                                    long long B, int nctx, int32_t* __restrict__ out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < B * nctx; i += (long long)gridDim.x * blockDim.x) {
        const long long b = i / nctx;
        const uint32_t c = (uint32_t)(i - b * nctx);
        out[i] = find_u32(ctx_key, G, ((uint32_t)bucket_scale[b] << 16) | c);
    }
}

// first-appearance list of a bucket's tables and context -> position in it (build_huffman.cu:748-783).
// One warp per bucket walks the 256 contexts 32 at a time: every lane first looks its table id up in
// the list built so far (kept in shared memory), the lanes that bring a new id are grouped by value
// with a warp match, and the lowest lane of each group appends the id at the position its rank
// among those leaders gives, which is the order a sequential scan would have appended them in.
constexpr int kUniqueWarps = 4;
__global__ void __launch_bounds__(kUniqueWarps * 32)
bucket_unique_kernel(const int32_t* __restrict__ bt, long long B, int32_t* __restrict__ U, int32_t* __restrict__ uniq,
                     int16_t* __restrict__ uidx) {
    __shared__ int32_t s_list[kUniqueWarps][256];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t* list = s_list[w];
    for (long long b = (long long)blockIdx.x * kUniqueWarps + w; b < B; b += (long long)gridDim.x * kUniqueWarps) {
        int32_t gids[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) gids[j] = bt[b * 256 + 32 * j + lane];
        // Ids that ascend with the context, as those of one scale do, are all new where they stand: no list to look
        // through (which took 43 us for the 174 buckets of a 14336 x 4096 weight).
        int32_t u = 0, last = -1;
        bool ascend = true;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t has = __ballot_sync(0xFFFFFFFFu, gids[j] >= 0), below = has & ((1u << lane) - 1u);
            const int32_t before = __shfl_sync(0xFFFFFFFFu, gids[j], below ? 31 - __clz((int)below) : 0);
            if (gids[j] >= 0 && gids[j] <= (below ? before : last)) ascend = false;
            const int32_t top = __shfl_sync(0xFFFFFFFFu, gids[j], has ? 31 - __clz((int)has) : 0);
            if (has) last = top;
        }
        if (__all_sync(0xFFFFFFFFu, ascend)) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t has = __ballot_sync(0xFFFFFFFFu, gids[j] >= 0);
                const int32_t pos = u + __popc(has & ((1u << lane) - 1u));
                if (gids[j] >= 0) uniq[b * 256 + pos] = gids[j];
                uidx[b * 256 + 32 * j + lane] = (int16_t)(gids[j] >= 0 ? pos : -1);
                u += __popc(has);
            }
            for (int j = u + lane; j < 256; j += 32) uniq[b * 256 + j] = -1;
            if (lane == 0) U[b] = u;
            continue;
        }
#pragma unroll
        for (int c0 = 0; c0 < 256; c0 += 32) {
            const int32_t gid = gids[c0 >> 5];
            const bool valid = gid >= 0;
            int32_t pos = -1;
            if (valid)
                for (int32_t j = 0; j < u; ++j)
                    if (list[j] == gid) { pos = j; break; }
            const bool fresh = valid && pos < 0;
            // lanes without a new id get a key no other lane has (-1 - lane is below every table id)
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, fresh ? gid : -1 - lane);
            const int first = __ffs(same) - 1;
            const bool leader = fresh && first == lane;
            const uint32_t leaders = __ballot_sync(0xFFFFFFFFu, leader);
            int32_t mine = u + __popc(leaders & ((1u << lane) - 1u));
            if (leader) list[mine] = gid;
            mine = __shfl_sync(0xFFFFFFFFu, mine, first);
            if (fresh) pos = mine;
            uidx[b * 256 + c0 + lane] = (int16_t)pos;
            u += __popc(leaders);
            __syncwarp();
        }
        for (int j = lane; j < 256; j += 32) uniq[b * 256 + j] = (j < u) ? list[j] : -1;
        if (lane == 0) U[b] = u;
        __syncwarp();
    }
}

__global__ void table_keys_kernel(const uint32_t* __restrict__ ctx_key, long long G, uint16_t* __restrict__ tscale,
                                  uint16_t* __restrict__ tctx) {
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < G; g += (long long)gridDim.x * blockDim.x) {
        tscale[g] = (uint16_t)(ctx_key[g] >> 16);
        tctx[g] = (uint16_t)(ctx_key[g] & 0xFFFF);
    }
}

// ------------------------------------------------------------------------------------------------
// shared-table layout (build_huffman.cu:2157-2633): one stream per (scale id, context), present or
// not; one bitstream per scale holding its elements in flat order; chunks of at most 255 consecutive
// elements of one stream
// ------------------------------------------------------------------------------------------------
__global__ void shared_rows_kernel(const uint32_t* __restrict__ ctx_key, long long G, const int32_t* __restrict__ sid_lut,
                                   int* __restrict__ row_of, int* __restrict__ stream_ctx) {
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < G; g += (long long)gridDim.x * blockDim.x) {
        const uint32_t key = ctx_key[g];
        const int sid = sid_lut[key >> 16];
        const int row = sid * 16 + (int)(key & 0xFu);
        row_of[g] = row;
        stream_ctx[row] = (int)g;
    }
}

// per element: its stream, its code (len << 16 | code, bit 31: 16 raw bits follow) and its bit count
__global__ void shared_elem_kernel(const uint16_t* __restrict__ sym, const uint8_t* __restrict__ q,
                                   const uint16_t* __restrict__ scales, int scale_mode, long long m, long long nb1,
                                   long long sb0, long long sb1, const int32_t* __restrict__ sid_lut,
                                   const int* __restrict__ stream_ctx, CodeBook cb, long long numel,
                                   int* __restrict__ stream, uint32_t* __restrict__ lc, int* __restrict__ nbits,
                                   int* __restrict__ run_head, int* __restrict__ err) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (long long)gridDim.x * blockDim.x) {
        auto stream_at = [&](long long e) -> int {
            uint16_t sc;
            if (scale_mode == 0) sc = scales[0];
            else {
                const long long r = e / m, c = e - r * m;
                sc = (scale_mode == 1) ? scales[r] : scales[(r / sb0) * nb1 + (c / sb1)];
            }
            return sid_lut[sc] * 16 + (int)(q[e] & 0xFu);
        };
        const int st = stream_at(i);
        stream[i] = st;
        run_head[i] = (i == 0 || stream_at(i - 1) != st) ? (int)i : 0;
        const int gid = stream_ctx[st];
        uint32_t code = 0; int len = 0; bool raw = false;
        const int nb = (gid >= 0) ? element_code(cb, gid, sym[i], code, len, raw) : -1;
        if (nb < 0) { atomicExch(err, 3); lc[i] = 0; nbits[i] = 0; continue; }
        lc[i] = ((uint32_t)len << 16) | code | (raw ? 0x80000000u : 0u);
        nbits[i] = nb;
    }
}

__global__ void shared_chunk_heads_kernel(const int* __restrict__ run_start, long long numel, int* __restrict__ chead) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (long long)gridDim.x * blockDim.x)
        chead[i] = ((i - run_start[i]) % 255 == 0) ? 1 : 0;
}

__global__ void shared_sid_keys_kernel(const int* __restrict__ stream, long long numel, int* __restrict__ key, int* __restrict__ val) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (long long)gridDim.x * blockDim.x)
        { key[i] = stream[i] >> 4; val[i] = (int)i; }
}

__global__ void gather_bits_kernel(const int* __restrict__ src, const int* __restrict__ idx, long long N,
                                   unsigned long long* __restrict__ dst) {   // 64-bit: the running sum passes 2^31 bits
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (unsigned long long)src[idx[i]];
}

// in scale-sorted order: where every scale's run starts and how many bits it holds
__global__ void shared_segments_kernel(const int* __restrict__ sid_sorted, const unsigned long long* __restrict__ nb_sorted,
                                       const unsigned long long* __restrict__ cum, long long numel,
                                       unsigned long long* __restrict__ seg_base, unsigned long long* __restrict__ seg_bits_end) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < numel; j += (long long)gridDim.x * blockDim.x) {
        const int sid = sid_sorted[j];
        if (j == 0 || sid_sorted[j - 1] != sid) seg_base[sid] = cum[j] - nb_sorted[j];
        if (j == numel - 1 || sid_sorted[j + 1] != sid) seg_bits_end[sid] = cum[j];
    }
}

__global__ void shared_relpos_kernel(const int* __restrict__ sid_sorted, const int* __restrict__ idx_sorted,
                                     const unsigned long long* __restrict__ nb_sorted, const unsigned long long* __restrict__ cum,
                                     const unsigned long long* __restrict__ seg_base, long long numel,
                                     uint32_t* __restrict__ rel) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < numel; j += (long long)gridDim.x * blockDim.x) {
        rel[idx_sorted[j]] = (uint32_t)(cum[j] - nb_sorted[j] - seg_base[sid_sorted[j]]);
    }
}

// scale_bit_base: every scale's bitstream starts on a 64-bit boundary (:2543-2560); res[0] = total bits
__global__ void shared_bases_kernel(const unsigned long long* __restrict__ seg_base, const unsigned long long* __restrict__ seg_end,
                                    long long S, long long* __restrict__ scale_bit_base, long long* __restrict__ res) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    long long total = 0;
    for (long long s = 0; s < S; ++s) {
        total = (total + 63) & ~63LL;
        scale_bit_base[s] = total;
        total += (long long)(seg_end[s] - seg_base[s]);
    }
    total = (total + 63) & ~63LL;
    scale_bit_base[S] = total;
    res[0] = total;
}

__global__ void shared_chunk_pos_kernel(const int* __restrict__ chead, const int* __restrict__ cidx, long long numel,
                                        long long C, int* __restrict__ cpos) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (long long)gridDim.x * blockDim.x) {
        if (chead[i]) cpos[cidx[i]] = (int)i;
        if (i == 0) cpos[C] = (int)numel;
    }
}

__global__ void shared_chunk_fill_kernel(const int* __restrict__ cpos, long long C, const int* __restrict__ stream,
                                         const uint32_t* __restrict__ rel, uint32_t* __restrict__ c_start,
                                         uint32_t* __restrict__ c_base, uint32_t* __restrict__ c_meta,
                                         int32_t* __restrict__ c_sid, int* __restrict__ c_stream) {
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < C; c += (long long)gridDim.x * blockDim.x) {
        const int i = cpos[c];
        const int st = stream[i];
        c_base[c] = (uint32_t)i;
        c_start[c] = rel[i];
        c_sid[c] = st >> 4;
        c_meta[c] = ((uint32_t)(cpos[c + 1] - i) << 8) | (uint32_t)(st & 15);
        c_stream[c] = st;
    }
}

__global__ void shared_emit_kernel(const uint16_t* __restrict__ sym, const int* __restrict__ stream,
                                   const uint32_t* __restrict__ lc, const uint32_t* __restrict__ rel,
                                   const long long* __restrict__ scale_bit_base, long long numel,
                                   unsigned long long* __restrict__ bitstream) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t v = lc[i];
        const int len = (int)((v >> 16) & 0x7FFFu);
        const bool raw = (v >> 31) != 0;
        unsigned long long bits = v & 0xFFFFu;
        int nb = len;
        if (raw) { bits = (bits << 16) | sym[i]; nb += 16; }
        if (nb <= 0) continue;
        const long long pos = scale_bit_base[stream[i] >> 4] + (long long)rel[i];
        const long long w = pos >> 6;
        const int o = (int)(pos & 63);
        if (o + nb <= 64) atomicOr(&bitstream[w], bits << (64 - o - nb));
        else {
            const int second = o + nb - 64;
            atomicOr(&bitstream[w], bits >> second);
            atomicOr(&bitstream[w + 1], bits << (64 - second));
        }
    }
}

__global__ void shared_stream_ofs_kernel(const int* __restrict__ keys_sorted, long long C, long long num_streams,
                                         long long* __restrict__ ofs) {
    for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s <= num_streams; s += (long long)gridDim.x * blockDim.x) {
        long long lo = 0, hi = C;  // first chunk whose stream is >= s
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (keys_sorted[mid] < s) lo = mid + 1; else hi = mid;
        }
        ofs[s] = lo;
    }
}

__global__ void iota_i32_kernel(int32_t* __restrict__ p, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        p[i] = (int32_t)i;
}

}  // namespace mps

// ------------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------------
using namespace mps;

namespace {

// device-wide primitives' temporary storage: the radix sort may want a full extra key buffer
static size_t cub_temp_bytes(int64_t numel) { return (64ull << 20) + (size_t)numel * 9; }
constexpr size_t kCodebookScratch = 160ull << 20;  // contexts whose codebooks do not fit shared memory: a slice per CTA

struct Carver {
    uint8_t* base; size_t off, cap;
    template <typename T> T* take(size_t count) {
        off = align_up(off);
        T* p = reinterpret_cast<T*>(base + off);
        off += count * sizeof(T);
        return p;
    }
    bool ok() const { return off <= cap; }
};

inline BuildState* state_of(mps_build_state* s) { return reinterpret_cast<BuildState*>(s); }

// Codebooks of every context (codebook.cuh), with scratch from workspace offset `off` on.
int run_codebooks(BuildState& S, size_t off, const int* row_of, uint16_t* out_syms, uint8_t* out_lens, cudaStream_t st) {
    Carver C{S.ws, off, S.ws_bytes};
    cbk::Args a;
    a.items = reinterpret_cast<unsigned long long*>(S.ws + S.o_items);
    a.counts = reinterpret_cast<int*>(S.ws + S.o_counts);
    a.ctx_ofs = reinterpret_cast<int*>(S.ws + S.o_ctx_ofs);
    a.G = (int)S.G; a.L = S.L; a.variant = S.variant;
    a.wide = (unsigned long long)S.numel * (unsigned)S.L >= 0xFFFFFFFFull;
    a.row_of = row_of;
    a.out_syms = out_syms; a.out_lens = out_lens;
    a.pairs = (reinterpret_cast<uintptr_t>(out_syms) & 3u) == 0 && (S.variant != V_AWQ_SHARED || (reinterpret_cast<uintptr_t>(out_lens) & 1u) == 0);
    a.enc = reinterpret_cast<uint32_t*>(S.ws + S.o_enc);
    a.esc = reinterpret_cast<uint32_t*>(S.ws + S.o_esc);
    a.escsym = reinterpret_cast<uint16_t*>(S.ws + S.o_escsym);
    a.err = S.d_flag + 1;
    a.big = C.take<int>((size_t)S.G);
    a.big_count = C.take<unsigned int>(2);
    a.queue = a.big_count + 1;
    const int sms = sm_count_host();
    const cbk::CtaShape shape = cbk::cta_shape(S.L, a.wide, sms, kCodebookScratch);
    auto* scratch = C.take<uint8_t>(shape.in_shared ? 0 : shape.stride * shape.grid);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    MPS_CUDA_TRY(cudaMemsetAsync(a.big_count, 0, 2 * sizeof(unsigned int), st));
    return cbk::launch(a, shape, sms, scratch, st);
}

// Can the counters be tried?  Rows, units and pointers must come in fours, units be pieces that share out well, and
// scales have elements enough that a scale's counters are worth their zeroing.
bool dense_possible(const hist::Geom& g, int64_t numel, uint32_t num_scales, const uint16_t* sym, const uint8_t* ctx) {
    return num_scales > 0 && g.m % 4 == 0 && g.ub1 % 4 == 0 && g.ub0 * g.ub1 <= 65536 && (reinterpret_cast<uintptr_t>(sym) & 7u) == 0 &&
           (reinterpret_cast<uintptr_t>(ctx) & 3u) == 0 && numel / num_scales >= hist::kDenseMinPerScale;
}

// How the units of a scale are cut into stretches (dense.cuh): units per stretch at most, the stretches before every scale's.
struct Stretches { long long units; uint32_t upc; uint32_t* base; };

// A CTA's stretch: every CTA slot of the GPU gets one, or three under 256 contexts, so that a last round of a few stretches
// costs less.  How many counters a scale has, which every one of its stretches zeroes and adds up, is not known yet: an FP8
// weight's few thousand do not matter, 50 K, as many as a CTA can hold, cost more than a stretch's elements.  Builds, us, one
// stretch per slot | three: FP8 14336 x 4096 with one scale 775 | 777, with heavy tails 841 | 802, per channel with heavy tails 1095
// | 1040, 28672 x 8192 1580 | 1564; with 51 K counters 14336 x 4096 3585 | 3640, 60 such scales 4830 | 4925.
uint32_t units_per_stretch(const hist::Geom& g, int64_t numel) {
    const long long slots = (g.nctx == 256 ? 12LL : 4LL) * sm_count_host();
    long long per_cta = (numel + slots - 1) / slots;
    if (per_cta < 32768) per_cta = 32768;
    if (per_cta > 131072) per_cta = 131072;
    const long long upc = per_cta / (g.ub0 * g.ub1);
    return upc > 1 ? (uint32_t)upc : 1u;
}

int bad_lists() {
    set_error("mps_build_analyze_listed: the lists are not those of these scales");
    return MPS_ERR_INVALID;
}

// The histogram with a counter per symbol of every range (dense.cuh); *done stays false where the ranges are too wide.
// `C` is a copy: scratch taken here is free again afterwards.  `counters`: numel of them.
int dense_histogram(BuildState& S, Carver C, const hist::Geom& g, const uint16_t* sym, const uint8_t* ctx, const uint16_t* scales,
                    uint32_t num_scales, const Stretches& sr, const hist::UnitLists& lists,
                    const uint16_t* scale_of_rank, uint32_t* counters, void* cub_tmp, size_t cub_bytes, cudaStream_t st,
                    bool* done) {
    const long long nseg = (long long)num_scales * g.nctx, nhalf = 2 * nseg;
    auto* lo = C.take<uint32_t>(nhalf);
    auto* hi = C.take<uint32_t>(nhalf);
    auto* ofs = C.take<unsigned long long>(nhalf + 1);
    auto* ctx_id = C.take<uint32_t>(nseg + 1);
    auto* distinct = C.take<uint32_t>(nseg + 1);
    auto* largest = C.take<uint32_t>(1);
    auto* totals = C.take<hist::DenseTotals>(1);
    if (!C.ok() || nhalf + 1 > 0x7FFFFFFFLL) return MPS_OK;
    hist::DenseGeom d;
    d.g = g;
    const bool eights = g.m % 8 == 0 && g.ub1 % 8 == 0 && (reinterpret_cast<uintptr_t>(sym) & 15u) == 0 && (reinterpret_cast<uintptr_t>(ctx) & 7u) == 0;
    d.row = (uint32_t)(g.ub1 / (eights ? 8 : 4));
    d.unit = d.row * (uint32_t)g.ub0;
    d.by_row = hist::dense_magic(d.row);
    d.by_unit = hist::dense_magic(d.unit);
    d.units_shift = -1;
    for (int i = 0; i < 31; ++i) if (g.nbu1 == (1LL << i)) d.units_shift = i;
    d.upc = sr.upc;
    const long long ctas = sr.units / d.upc + num_scales;      // at most
    auto* stretch_first = C.take<uint32_t>(ctas);
    if (!C.ok()) return MPS_OK;
    d.first = stretch_first;
    d.count = sr.base + hist::kScaleValues;
    const int fill_ctas = grid_for(ctas);
    hist::dense_stretch_fill_kernel<<<fill_ctas + (lists.said ? grid_for(sr.units) : 0), 256, 0, st>>>(g, scales, lists, sr.base, d.upc, (uint32_t)ctas,
                                                                                                     (uint32_t)fill_ctas, stretch_first);
    hist::dense_preset_kernel<<<grid_for(nhalf), 256, 0, st>>>(lo, hi, nhalf);
    auto* const range_kernel = eights ? hist::dense_range_kernel<8> : hist::dense_range_kernel<4>;
    range_kernel<<<(unsigned)ctas, hist::kDenseThreads, 0, st>>>(d, sym, ctx, scales, lists, lo, hi);
    size_t need = cub_bytes;
    if (nseg <= hist::kOffsetsMost) {
        hist::dense_offsets_kernel<<<hist::kOffsetsCtas, 1024, 0, st>>>(lo, hi, (int)nseg, g.nctx, ofs, ctx_id, lists, totals);
    } else {
        hist::dense_sizes_kernel<<<grid_for(nseg + 1), 256, 0, st>>>(lo, hi, nseg, ofs, ctx_id);
        MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, ofs, ofs, (int)(nhalf + 1), st));
        need = cub_bytes;
        MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, ctx_id, ctx_id, (int)(nseg + 1), st));
        MPS_CUDA_TRY(cudaMemsetAsync(largest, 0, sizeof(uint32_t), st));
        hist::dense_largest_kernel<<<grid_for(num_scales), 256, 0, st>>>(ofs, num_scales, 2 * g.nctx, largest);
        hist::dense_totals_kernel<<<1, 1, 0, st>>>(ofs, ctx_id, largest, nseg, lists, totals);
    }
    hist::DenseTotals t;
    MPS_CUDA_TRY(cudaMemcpyAsync(&t, totals, sizeof(t), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (t.lists_bad) return bad_lists();
    const unsigned long long total = t.counters;
    const uint32_t most = t.most, contexts = t.contexts;
    if (total > (unsigned long long)S.numel || most > (uint32_t)hist::kDenseCounters) return MPS_OK;
    static bool attr_set[64] = {false};
    int dev = 0;
    MPS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        MPS_CUDA_TRY(cudaFuncSetAttribute(hist::dense_count_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, hist::kDenseCounters * 4));
        MPS_CUDA_TRY(cudaFuncSetAttribute(hist::dense_count_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, hist::kDenseCounters * 4));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    MPS_CUDA_TRY(cudaMemsetAsync(counters, 0, (size_t)total * sizeof(uint32_t), st));
    auto* const count_kernel = eights ? hist::dense_count_kernel<8> : hist::dense_count_kernel<4>;
    count_kernel<<<(unsigned)ctas, most > 26 * 1024 ? 1024 : hist::kDenseThreads, (size_t)most * 4, st>>>(d, sym, ctx, scales, lists, lo, ofs,
                                                                                                         counters);
    hist::dense_distinct_kernel<<<grid_for((nseg + 1) * 32), 256, 0, st>>>(ofs, counters, nseg, distinct);
    need = cub_bytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, distinct, distinct, (int)(nseg + 1), st));
    hist::dense_items_kernel<<<grid_for(nseg * 32), 256, 0, st>>>(
        ofs, lo, counters, distinct, ctx_id, nseg, g.nctx, scale_of_rank, reinterpret_cast<unsigned long long*>(S.ws + S.o_items),
        reinterpret_cast<int*>(S.ws + S.o_counts), reinterpret_cast<int*>(S.ws + S.o_ctx_ofs), reinterpret_cast<uint32_t*>(S.ws + S.o_ctx_key));
    uint32_t n_items = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&n_items, distinct + nseg, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    S.N = n_items;
    S.G = contexts;
    *done = true;
    return MPS_OK;
}

}  // namespace

extern "C" {

size_t mps_build_workspace_bytes(int64_t numel, int64_t substreams) {
    if (numel < 0) numel = 0;
    if (substreams < numel) substreams = numel;
    // (the last term: six 32-bit arrays over the (scale, context) segments, of which a tensor has at most
    // 256 per distinct scale and no more distinct scales than elements or 16-bit values)
    const size_t max_scales = (size_t)(numel < 65536 ? numel : 65536);
    return 256 + (size_t)numel * 34 + (size_t)numel * 40 + (size_t)substreams * 4 + cub_temp_bytes(numel) + kCodebookScratch +
           (4ull << 20) + (max_scales * 256 + 1) * 24;
}

size_t mps_build_lists_workspace_bytes(int64_t groups) {
    if (groups <= 0 || groups >= (1LL << 31)) return 0;
    return lists::carve(nullptr, groups).bytes;
}

int mps_build_lists_sort(const uint16_t* scales_u16, int32_t scale_mode, int64_t nb1, int64_t sb0, int64_t n, int64_t group_cap,
                         void* workspace, size_t workspace_bytes, void* stream, int64_t* num_buckets_out) {
    int64_t scales = 0;
    return mps_build_lists_sort_counted(scales_u16, scale_mode, nb1, sb0, n, group_cap, workspace, workspace_bytes, stream, num_buckets_out, &scales);
}

int mps_build_lists_sort_counted(const uint16_t* scales_u16, int32_t scale_mode, int64_t nb1, int64_t sb0, int64_t n, int64_t group_cap,
                                 void* workspace, size_t workspace_bytes, void* stream, int64_t* num_buckets_out, int64_t* num_scales_out) {
    if (!scales_u16 || !workspace || !num_buckets_out || !num_scales_out) { set_error("mps_build_lists_sort: null argument"); return MPS_ERR_INVALID; }
    if (scale_mode < 0 || scale_mode > 2 || n <= 0 || group_cap <= 0 || (scale_mode == 2 && (nb1 <= 0 || sb0 <= 0))) {
        set_error("mps_build_lists_sort: bad argument");
        return MPS_ERR_INVALID;
    }
    lists::Geom g;
    g.per_row = scale_mode == 2 ? nb1 : 1;
    if (n >= (1LL << 31) || g.per_row >= (1LL << 31) || n * g.per_row >= (1LL << 31)) { set_error("too many groups"); return MPS_ERR_UNSUPPORTED; }
    g.groups = n * g.per_row; g.sb0 = sb0; g.nb1 = nb1; g.scale_mode = scale_mode;
    if ((reinterpret_cast<uintptr_t>(workspace) & 3u) != 0) { set_error("mps_build_lists_sort: workspace must be 4-byte aligned"); return MPS_ERR_WORKSPACE; }
    const lists::Arrays a = lists::carve(static_cast<uint8_t*>(workspace), g.groups);
    if (workspace_bytes < a.bytes) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t cap = group_cap < 0x7FFFFFFFLL ? (uint32_t)group_cap : 0x7FFFFFFFu;
    lists::keys_kernel<<<lists::grid_of(g.groups), 256, 0, st>>>(g, scales_u16, a.key, a.group);
    size_t bytes = a.cub_bytes;
    MPS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(a.cub, bytes, a.key, a.key_sorted, a.group, a.sorted, (int)g.groups, 0, 16, st));
    MPS_CUDA_TRY(cudaMemsetAsync(a.first, 0, (size_t)((uint8_t*)a.base - (uint8_t*)a.first), st));
    lists::runs_kernel<<<lists::grid_of(g.groups), 256, 0, st>>>(a.key_sorted, g.groups, a.first, a.end);
    lists::scale_scan_kernel<<<lists::kScanCtas, 1024, 0, st>>>(a.first, a.end, cap, a.base, nullptr, nullptr, nullptr, nullptr, a.totals);
    lists::ScanTotals totals;
    MPS_CUDA_TRY(cudaMemcpyAsync(&totals, a.totals, sizeof(totals), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    *num_buckets_out = totals.parts;
    *num_scales_out = totals.scales;
    return MPS_OK;
}

int mps_build_lists_write(int64_t groups, int64_t groups_per_row, int64_t group_size, int64_t group_cap, void* workspace,
                          size_t workspace_bytes, uint16_t* bucket_scale_u16, int32_t* bucket_offsets_i32, int32_t* rows_i32,
                          int32_t* col_start_i32, void* stream) {
    if (!workspace || !bucket_scale_u16 || !bucket_offsets_i32 || !rows_i32 || groups <= 0 || groups >= (1LL << 31) || groups_per_row <= 0 ||
        groups_per_row > groups || group_cap <= 0 || group_size <= 0 || group_size >= (1LL << 31)) {
        set_error("mps_build_lists_write: bad argument");
        return MPS_ERR_INVALID;
    }
    if ((reinterpret_cast<uintptr_t>(workspace) & 3u) != 0) { set_error("mps_build_lists_write: workspace must be 4-byte aligned"); return MPS_ERR_WORKSPACE; }
    const lists::Arrays a = lists::carve(static_cast<uint8_t*>(workspace), groups);
    if (workspace_bytes < a.bytes) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t cap = group_cap < 0x7FFFFFFFLL ? (uint32_t)group_cap : 0x7FFFFFFFu;
    lists::buckets_kernel<<<lists::kScaleValues * 32 / 256, 256, 0, st>>>(a.first, a.end, a.base, cap, groups, bucket_scale_u16, bucket_offsets_i32);
    lists::members_kernel<<<lists::grid_of(groups), 256, 0, st>>>(a.sorted, groups, (uint32_t)groups_per_row, (uint32_t)group_size, rows_i32,
                                                                  col_start_i32);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

int mps_build_analyze(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* ctx_bytes,
                      const uint16_t* scales_u16, int32_t scale_mode, int64_t nb1, int64_t sb0, int64_t sb1, int64_t n,
                      int64_t m, int32_t variant, int64_t max_len, void* workspace, size_t workspace_bytes, void* stream,
                      int64_t* num_tables_out, int64_t* num_items_out) {
    return mps_build_analyze_listed(state, bf16_bits, ctx_bytes, scales_u16, scale_mode, nb1, sb0, sb1, n, m, variant, max_len, workspace,
                                    workspace_bytes, nullptr, 0, 0, stream, num_tables_out, num_items_out);
}

int mps_build_analyze_listed(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* ctx_bytes,
                             const uint16_t* scales_u16, int32_t scale_mode, int64_t nb1, int64_t sb0, int64_t sb1, int64_t n,
                             int64_t m, int32_t variant, int64_t max_len, void* workspace, size_t workspace_bytes, void* lists_workspace,
                             size_t lists_workspace_bytes, int64_t lists_scales, void* stream, int64_t* num_tables_out, int64_t* num_items_out) {
    if (!state || !bf16_bits || !ctx_bytes || !scales_u16 || !workspace || !num_tables_out || !num_items_out) {
        set_error("mps_build_analyze: null argument");
        return MPS_ERR_INVALID;
    }
    if (n <= 0 || m <= 0) { set_error("bf16_params shape must be non-empty"); return MPS_ERR_INVALID; }
    if (variant < V_FP8 || variant > V_AWQ_SHARED) { set_error("unknown builder variant %d", variant); return MPS_ERR_INVALID; }
    if (max_len <= 0 || max_len > 15) { set_error("max_len must be in [1, 15]"); return MPS_ERR_INVALID; }
    if (scale_mode < 0 || scale_mode > 2 || (scale_mode == 2 && (nb1 <= 0 || sb0 <= 0 || sb1 <= 0))) {
        set_error("unsupported scales layout");
        return MPS_ERR_INVALID;
    }
    const int64_t numel = n * m;
    if (numel >= (1LL << 31)) { set_error("tensors of 2^31 elements or more are not supported by the builder"); return MPS_ERR_UNSUPPORTED; }
    if (workspace_bytes < mps_build_workspace_bytes(numel, numel)) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    BuildState& S = *state_of(state);
    memset(&S, 0, sizeof(S));
    S.numel = numel; S.n = n; S.m = m; S.L = (int32_t)max_len; S.variant = variant;
    S.group_size = (int32_t)((scale_mode == 2) ? sb1 : m);
    S.ws = static_cast<uint8_t*>(workspace); S.ws_bytes = workspace_bytes;
    Carver C{S.ws, 256, workspace_bytes};
    S.d_flag = reinterpret_cast<int32_t*>(S.ws);
    auto* items = C.take<unsigned long long>(numel);  S.o_items = (uint8_t*)items - S.ws;
    auto* counts = C.take<int>(numel);                S.o_counts = (uint8_t*)counts - S.ws;
    auto* ctx_ofs = C.take<int>(numel + 1);           S.o_ctx_ofs = (uint8_t*)ctx_ofs - S.ws;
    auto* ctx_key = C.take<uint32_t>(numel);          S.o_ctx_key = (uint8_t*)ctx_key - S.ws;
    auto* enc = C.take<uint32_t>(numel);              S.o_enc = (uint8_t*)enc - S.ws;
    auto* esc = C.take<uint32_t>(numel);              S.o_esc = (uint8_t*)esc - S.ws;
    auto* escsym = C.take<uint16_t>(numel);           S.o_escsym = (uint8_t*)escsym - S.ws;
    C.off = align_up(C.off);
    S.o_scratch = C.off; S.scratch_bytes = workspace_bytes - C.off;
    // ---- scratch of the histogram ------------------------------------------------------------------
    MPS_CUDA_TRY(cudaMemsetAsync(S.d_flag, 0, 256, st));
    hist::Geom g;
    g.n = n; g.m = m; g.scale_mode = scale_mode;
    g.ctx_mask = (variant == V_FP8) ? 0xFFu : 0x0Fu;
    g.nctx = (variant == V_FP8) ? 256 : 16;
    if (scale_mode == 2) {
        if (nb1 * sb1 < m) { set_error("unsupported scales layout"); return MPS_ERR_INVALID; }
        g.ub0 = sb0; g.ub1 = sb1; g.nbu1 = nb1; g.nbu0 = (n + sb0 - 1) / sb0;
    } else {  // pieces of rows
        g.ub0 = 1; g.ub1 = (m <= 8192) ? m : 4096; g.nbu1 = (m + g.ub1 - 1) / g.ub1; g.nbu0 = n;
    }
    const long long units = g.nbu0 * g.nbu1;
    const size_t kCubTempBytes = cub_temp_bytes(numel);
    void* cub_tmp = C.take<uint8_t>(kCubTempBytes);
    auto* per_scale = C.take<uint32_t>(hist::kScaleValues + 1);   // units of every scale value
    auto* unit_ofs = C.take<uint32_t>(hist::kScaleValues + 1);
    auto* rank = C.take<uint32_t>(hist::kScaleValues + 1);        // flags, then ranks; [65536] = number of distinct scales
    auto* unit_cur = C.take<uint32_t>(hist::kScaleValues);
    auto* scale_of_rank = C.take<uint16_t>(hist::kScaleValues);
    auto* unit_sorted = C.take<uint32_t>(units);
    auto* seg_syms = C.take<uint16_t>(numel);
    auto* st_sym = C.take<uint16_t>(numel);
    auto* st_cnt = C.take<uint32_t>(numel);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    size_t need = 0;

    // scales: rank of every distinct value, units listed by scale -- as the bucket lists have them already where a unit is a
    // group of those
    Stretches sr{units, units_per_stretch(g, numel), C.take<uint32_t>(hist::kScaleValues + 1)};
    auto* scan_totals = C.take<lists::ScanTotals>(1);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    uint32_t num_scales = 0;
    const bool listed = lists_workspace != nullptr && g.nbu0 == n && g.nbu1 == (scale_mode == 2 ? nb1 : 1);
    if (lists_workspace != nullptr && ((reinterpret_cast<uintptr_t>(lists_workspace) & 3u) != 0 || lists_scales <= 0 || lists_scales > units)) {
        set_error("mps_build_analyze: bad lists");
        return MPS_ERR_INVALID;
    }
    if (listed) {
        const lists::Arrays a = lists::carve(static_cast<uint8_t*>(lists_workspace), units);
        if (lists_workspace_bytes < a.bytes) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
        unit_sorted = a.sorted;
        lists::scale_scan_kernel<<<lists::kScanCtas, 1024, 0, st>>>(a.first, a.end, sr.upc, sr.base, unit_ofs, nullptr, rank, scale_of_rank, scan_totals);
        num_scales = (uint32_t)lists_scales;
    } else {
        MPS_CUDA_TRY(cudaMemsetAsync(per_scale, 0, (hist::kScaleValues + 1) * sizeof(uint32_t), st));
        hist::unit_scale_count_kernel<<<grid_for(units), 256, 0, st>>>(g, scales_u16, units, per_scale);
        lists::scale_scan_kernel<<<lists::kScanCtas, 1024, 0, st>>>(per_scale, nullptr, sr.upc, sr.base, unit_ofs, unit_cur, rank, scale_of_rank, scan_totals);
        hist::unit_scatter_kernel<<<grid_for(units), 256, 0, st>>>(g, scales_u16, units, unit_cur, unit_sorted);
        lists::ScanTotals t;
        MPS_CUDA_TRY(cudaMemcpyAsync(&t, scan_totals, sizeof(t), cudaMemcpyDeviceToHost, st));
        MPS_CUDA_TRY(cudaStreamSynchronize(st));
        num_scales = t.scales;
    }
    MPS_CUDA_TRY(cudaGetLastError());
    const long long nseg = (long long)num_scales * g.nctx;
    const hist::UnitLists lists{unit_sorted, unit_ofs, rank, &scan_totals->scales, (uint32_t)units, listed ? num_scales : 0u, S.d_flag + 2};

    // few symbols per context: a counter for each (counted in place, the tensor is read twice and nothing is moved)
    if (dense_possible(g, numel, num_scales, bf16_bits, ctx_bytes)) {
        bool done = false;
        const int rc = dense_histogram(S, C, g, bf16_bits, ctx_bytes, scales_u16, num_scales, sr, lists, scale_of_rank, st_cnt, cub_tmp, kCubTempBytes, st, &done);
        if (rc) return rc;
        if (done) {
            *num_tables_out = S.G;
            *num_items_out = S.N;
            return MPS_OK;
        }
    }
    if (listed) hist::unit_lists_check_kernel<<<grid_for(units), 256, 0, st>>>(g, scales_u16, lists);

    // segments (scale rank, context): sizes, offsets, symbols
    auto* seg_cnt = C.take<uint32_t>(nseg + 1);
    auto* seg_ofs = C.take<uint32_t>(nseg + 1);
    auto* seg_cur = C.take<uint32_t>(nseg + 1);      // write cursors, later distinct symbols per segment, then item offsets
    auto* chunk_ofs = C.take<uint32_t>(nseg + 1);    // chunks per segment, then their prefix
    auto* split_id = C.take<uint32_t>(nseg + 1);     // split flags, then their prefix
    auto* ctx_id = C.take<uint32_t>(nseg + 1);       // non-empty flags, then their prefix: the context index
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    long long upw = hist::kWarpElems / (g.ub0 * g.ub1);
    if (upw < 1) upw = 1;
    const long long walk_warps = (units + upw - 1) / upw;
    const unsigned walk_grid = (unsigned)((walk_warps + hist::kWalkWarps - 1) / hist::kWalkWarps);
    MPS_CUDA_TRY(cudaMemsetAsync(seg_cnt, 0, (nseg + 1) * sizeof(uint32_t), st));
    hist::segment_walk_kernel<false><<<walk_grid, hist::kWalkWarps * 32, 0, st>>>(g, bf16_bits, ctx_bytes, scales_u16, lists, upw, seg_cnt,
                                                                                  nullptr);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, seg_cnt, seg_ofs, (int)(nseg + 1), st));
    MPS_CUDA_TRY(cudaMemcpyAsync(seg_cur, seg_ofs, (nseg + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    hist::segment_walk_kernel<true><<<walk_grid, hist::kWalkWarps * 32, 0, st>>>(g, bf16_bits, ctx_bytes, scales_u16, lists, upw, seg_cur,
                                                                                 seg_syms);
    hist::chunk_plan_kernel<<<grid_for(nseg + 1), 256, 0, st>>>(seg_cnt, nseg, chunk_ofs, split_id, ctx_id);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, chunk_ofs, chunk_ofs, (int)(nseg + 1), st));
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, split_id, split_id, (int)(nseg + 1), st));
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, ctx_id, ctx_id, (int)(nseg + 1), st));
    auto* segment_totals = C.take<hist::SegmentTotals>(1);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    hist::segment_totals_kernel<<<1, 1, 0, st>>>(chunk_ofs, split_id, ctx_id, nseg, lists, segment_totals);
    hist::SegmentTotals totals;
    MPS_CUDA_TRY(cudaMemcpyAsync(&totals, segment_totals, sizeof(totals), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (totals.lists_bad) return bad_lists();
    const long long num_chunks = totals.chunks, num_split = totals.split;
    const int G = (int)totals.contexts;

    // symbols of every segment counted by value
    auto* chunk_seg = C.take<uint32_t>(num_chunks);
    auto* split_seg = C.take<uint32_t>(num_split);
    auto* dense = C.take<uint32_t>((size_t)num_split * 65536u);
    auto* split_range = C.take<uint32_t>((size_t)num_split * 2);     // smallest, largest symbol of every split segment
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    hist::chunk_fill_kernel<<<grid_for(nseg), 256, 0, st>>>(seg_cnt, nseg, chunk_ofs, split_id, chunk_seg, split_seg);
    if (num_split) {
        MPS_CUDA_TRY(cudaMemsetAsync(dense, 0, (size_t)num_split * 65536u * sizeof(uint32_t), st));
        hist::split_range_init_kernel<<<grid_for(num_split), 256, 0, st>>>(split_range, num_split);
    }
    MPS_CUDA_TRY(cudaMemsetAsync(seg_cur, 0, (nseg + 1) * sizeof(uint32_t), st));
    if (num_chunks)
        hist::chunk_count_kernel<<<(unsigned)num_chunks, 256, 0, st>>>(seg_syms, seg_cnt, seg_ofs, chunk_seg, chunk_ofs, split_id, dense,
                                                                       split_range, st_sym, st_cnt, seg_cur);
    if (num_split) hist::split_finish_kernel<<<(unsigned)num_split, 256, 0, st>>>(split_seg, seg_ofs, dense, split_range, st_sym, st_cnt, seg_cur);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, seg_cur, seg_cur, (int)(nseg + 1), st));
    hist::gather_items_kernel<<<grid_for(nseg * 32), 256, 0, st>>>(seg_cnt, seg_ofs, seg_cur, ctx_id, nseg, g.nctx, scale_of_rank, st_sym,
                                                                   st_cnt, items, counts, ctx_ofs, ctx_key);
    uint32_t n_items = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&n_items, seg_cur + nseg, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    const long long N = n_items;
    S.N = N;

    S.G = G;
    *num_tables_out = G;
    *num_items_out = N;
    return MPS_OK;
}

int mps_build_codebooks(mps_build_state* state, uint16_t* decode_syms_u16, uint8_t* decode_lens_u8,
                        uint16_t* table_scale_u16, uint16_t* table_ctx_u16, void* stream) {
    int rc = mps_build_codebooks_async(state, decode_syms_u16, decode_lens_u8, table_scale_u16, table_ctx_u16, stream);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int flag = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&flag, state_of(state)->d_flag + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (flag == 2) { set_error("Internal error: not enough packages"); return (int)cudaErrorUnknown; }
    return MPS_OK;
}

int mps_build_codebooks_async(mps_build_state* state, uint16_t* decode_syms_u16, uint8_t* decode_lens_u8,
                              uint16_t* table_scale_u16, uint16_t* table_ctx_u16, void* stream) {
    if (!state || !decode_syms_u16 || !decode_lens_u8 || !table_scale_u16 || !table_ctx_u16) {
        set_error("mps_build_codebooks: null argument");
        return MPS_ERR_INVALID;
    }
    BuildState& S = *state_of(state);
    if (S.variant == V_AWQ_SHARED) { set_error("shared-table sidecars use mps_build_shared_codebooks"); return MPS_ERR_INVALID; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    S.rect_buckets = 0;   // the scratch area is used here: what a layout call left there is gone
    int rc = run_codebooks(S, S.o_scratch, nullptr, decode_syms_u16, decode_lens_u8, st);
    if (rc) return rc;
    auto* ctx_key = reinterpret_cast<uint32_t*>(S.ws + S.o_ctx_key);
    table_keys_kernel<<<grid_for(S.G), 256, 0, st>>>(ctx_key, S.G, table_scale_u16, table_ctx_u16);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

int mps_build_bucket_table(mps_build_state* state, const uint16_t* bucket_scale_u16, int64_t num_buckets,
                           int32_t* bucket_table_i32, void* stream) {
    if (!state || !bucket_scale_u16 || !bucket_table_i32 || num_buckets < 0) { set_error("mps_build_bucket_table: bad argument"); return MPS_ERR_INVALID; }
    BuildState& S = *state_of(state);
    const int nctx = (S.variant == V_FP8) ? 256 : 16;
    auto* ctx_key = reinterpret_cast<uint32_t*>(S.ws + S.o_ctx_key);
    if (num_buckets == 0) return MPS_OK;
    bucket_table_kernel<<<grid_for(num_buckets * nctx), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        ctx_key, (int)S.G, bucket_scale_u16, num_buckets, nctx, bucket_table_i32);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

int mps_build_bucket_unique(const int32_t* bucket_table_i32, int64_t num_buckets, int32_t* bucket_U_i32,
                            int32_t* bucket_unique_gid_i32, int16_t* bucket_fp8_uidx_i16, void* stream) {
    if (!bucket_table_i32 || !bucket_U_i32 || !bucket_unique_gid_i32 || !bucket_fp8_uidx_i16 || num_buckets < 0) {
        set_error("mps_build_bucket_unique: bad argument");
        return MPS_ERR_INVALID;
    }
    if (num_buckets == 0) return MPS_OK;
    bucket_unique_kernel<<<grid_for((num_buckets + kUniqueWarps - 1) / kUniqueWarps, 1), kUniqueWarps * 32, 0,
                           static_cast<cudaStream_t>(stream)>>>(
        bucket_table_i32, num_buckets, bucket_U_i32, bucket_unique_gid_i32, bucket_fp8_uidx_i16);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

static int rect_common(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* ctx_bytes,
                       const int32_t* bucket_table_i32, const int32_t* bucket_col_start_i32,
                       const int32_t* bucket_col_len_i32, const int32_t* bucket_row_offsets_i32,
                       const int32_t* row_indices_i32, int64_t num_buckets, int32_t k, RectGeom* g, CodeBook* cb) {
    if (!state || !bf16_bits || !ctx_bytes || !bucket_table_i32 || !bucket_col_start_i32 ||
        !bucket_row_offsets_i32 || !row_indices_i32 || num_buckets < 0 || k <= 0 || k > MPS_MAX_SUBSTREAMS) {
        set_error("sidecar layout: bad argument");
        return MPS_ERR_INVALID;
    }
    BuildState& S = *state_of(state);
    // ragged (by-scale) layout: bucket_col_len is null, bucket_col_start lists the column start of every
    // group, the row list holds the groups' rows and every group has S.group_size elements
    const bool ragged = (bucket_col_len_i32 == nullptr);
    if (ragged && S.group_size <= 0) { set_error("sidecar layout: group size not set"); return MPS_ERR_INVALID; }
    g->sym = bf16_bits; g->ctx = ctx_bytes; g->bucket_table = bucket_table_i32;
    g->col_start = ragged ? nullptr : bucket_col_start_i32; g->group_col = ragged ? bucket_col_start_i32 : nullptr;
    g->group_size = S.group_size;
    g->col_len = bucket_col_len_i32; g->row_ofs = bucket_row_offsets_i32; g->rows = row_indices_i32;
    g->B = num_buckets; g->m = S.m; g->k = k; g->nctx = (S.variant == V_FP8) ? 256 : 16;
    g->ctx_mask = (S.variant == V_FP8) ? 0xFFu : 0x0Fu;
    cb->items = reinterpret_cast<unsigned long long*>(S.ws + S.o_items);
    cb->ctx_ofs = reinterpret_cast<int*>(S.ws + S.o_ctx_ofs);
    cb->enc = reinterpret_cast<uint32_t*>(S.ws + S.o_enc);
    cb->esc = reinterpret_cast<uint32_t*>(S.ws + S.o_esc);
    cb->escsym = reinterpret_cast<uint16_t*>(S.ws + S.o_escsym);
    return MPS_OK;
}

// sizes of the layout and emit launches, from what both calls know
static lay::Shape rect_shape(const BuildState& S, const RectGeom& g) {
    const long long largest = g.group_col ? 4 * (S.numel / (g.B > 0 ? g.B : 1)) : 128LL * S.group_size;
    return lay::shape_of(S.numel, g.B, largest, g.k, S.L, S.rect_vec != 0, sm_count_host());
}
static size_t rect_units(const BuildState& S, const RectGeom& g, const lay::Shape& s) {
    return (size_t)g.B * (1 + (size_t)g.k / (lay::kThreads * s.v)) + (size_t)(S.numel / s.unit) + 1;
}
static lay::Args rect_args(const BuildState& S, const RectGeom& g, const CodeBook& cb, const lay::Shape& s) {
    lay::Args a;
    memset(&a, 0, sizeof(a));
    a.g = g; a.cb = cb; a.G = S.G; a.numel = S.numel;
    a.ebase = reinterpret_cast<const unsigned long long*>(S.ws + S.o_rect_ebase);
    a.codes = S.ws + S.o_rect_codes;
    a.part = s.small ? nullptr : reinterpret_cast<uint32_t*>(S.ws + S.o_rect_part);
    a.unit = s.unit; a.map_cap = s.map_cap; a.buf_words = s.buf_words;
    a.err = S.d_flag;
    return a;
}

// Layout with S.rect_vec as it stands: start bits, bucket bases, the stream's bits (`total`) and the error flag.
static int rect_layout_pass(BuildState& S, const RectGeom& g, const CodeBook& cb, uint32_t* startbit, int64_t* bit_base, cudaStream_t st,
                            long long* total, int* flag) {
    const lay::Shape shape = rect_shape(S, g);
    Carver C{S.ws, S.o_scratch, S.ws_bytes};
    // kept for the emit call: codes, bucket offsets into them, what every team starts behind
    auto* codes = C.take<uint8_t>((size_t)S.numel * (shape.wide ? 4 : 2));
    auto* ebase = C.take<unsigned long long>(g.B + 1);
    auto* part = C.take<uint32_t>(shape.small ? 0 : rect_units(S, g, shape) * (lay::kThreads * lay::kMaxV));
    auto* bits = C.take<uint32_t>((size_t)g.B * g.k);
    auto* bucket_bits = C.take<unsigned long long>(g.B + 1);
    if (!C.ok()) { set_error("workspace too small for %lld buckets of %d sub-streams", g.B, g.k); return MPS_ERR_WORKSPACE; }
    S.o_rect_codes = codes - S.ws; S.o_rect_ebase = (uint8_t*)ebase - S.ws; S.o_rect_part = (uint8_t*)part - S.ws;
    MPS_CUDA_TRY(cudaMemsetAsync(S.d_flag, 0, sizeof(int), st));   // (lists that were refused may be followed by better ones)
    if (g.B > 0) {
        lay::element_bases_kernel<<<1, 1024, 0, st>>>(g, S.numel, ebase, S.d_flag);
        lay::Args a = rect_args(S, g, cb, shape);
        a.bits = bits;
        const int rc = lay::launch_codes(a, shape, st);
        if (rc) return rc;
        lay::starts_kernel<<<grid_for((g.B + 7) / 8, 1), 256, 0, st>>>(bits, g.B, g.k, startbit, bucket_bits);
        S.rect_buckets = g.B; S.rect_k = g.k; S.rect_ragged = g.group_col != nullptr;
    }
    auto* const totals = reinterpret_cast<lay::Totals*>(S.ws + 64);
    lay::bit_bases_kernel<<<1, 1024, 0, st>>>(bucket_bits, g.B, S.d_flag, reinterpret_cast<long long*>(bit_base), totals);
    MPS_CUDA_TRY(cudaGetLastError());
    lay::Totals t;
    MPS_CUDA_TRY(cudaMemcpyAsync(&t, totals, sizeof(t), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    *total = t.bits;
    *flag = t.err;
    if (t.codebook_err == 2) { set_error("Internal error: not enough packages"); return (int)cudaErrorUnknown; }
    return MPS_OK;
}

int mps_build_rect_layout(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* ctx_bytes,
                          const int32_t* bucket_table_i32, const int32_t* bucket_col_start_i32,
                          const int32_t* bucket_col_len_i32, const int32_t* bucket_row_offsets_i32,
                          const int32_t* row_indices_i32, int64_t num_buckets, int32_t k,
                          uint32_t* bucket_thread_startbit_u32, int64_t* bucket_bit_base_i64, void* stream,
                          int64_t* total_bits_out) {
    RectGeom g; CodeBook cb;
    int rc = rect_common(state, bf16_bits, ctx_bytes, bucket_table_i32, bucket_col_start_i32, bucket_col_len_i32,
                         bucket_row_offsets_i32, row_indices_i32, num_buckets, k, &g, &cb);
    if (rc) return rc;
    if (!bucket_thread_startbit_u32 || !bucket_bit_base_i64 || !total_bits_out) { set_error("sidecar layout: null output"); return MPS_ERR_INVALID; }
    BuildState& S = *state_of(state);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (num_buckets > 0x7FFFFFFFLL) { set_error("too many buckets"); return MPS_ERR_INVALID; }
    S.rect_buckets = 0;
    S.rect_vec = (S.m % 4 == 0 && S.group_size % 4 == 0 && k % 4 == 0 && (reinterpret_cast<uintptr_t>(ctx_bytes) & 3u) == 0 &&
                  (reinterpret_cast<uintptr_t>(bf16_bits) & 7u) == 0) ? 1 : 0;
    long long total = 0; int flag = 0;
    rc = rect_layout_pass(S, g, cb, bucket_thread_startbit_u32, bucket_bit_base_i64, st, &total, &flag);
    if (rc) return rc;
    if (flag == lay::kNotFours) {   // columns that a caller cut elsewhere: the elements one by one
        S.rect_vec = 0;
        rc = rect_layout_pass(S, g, cb, bucket_thread_startbit_u32, bucket_bit_base_i64, st, &total, &flag);
        if (rc) return rc;
    }
    if (flag == 3) { set_error("symbol not found and no ESC for (scale,ctx) key"); return (int)cudaErrorUnknown; }
    if (flag == 4) { set_error("the buckets hold more elements than the tensor has"); return MPS_ERR_INVALID; }
    *total_bits_out = total;
    return MPS_OK;
}

int mps_build_rect_emit(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* ctx_bytes,
                        const int32_t* bucket_table_i32, const int32_t* bucket_col_start_i32,
                        const int32_t* bucket_col_len_i32, const int32_t* bucket_row_offsets_i32,
                        const int32_t* row_indices_i32, int64_t num_buckets, int32_t k,
                        const uint32_t* bucket_thread_startbit_u32, const int64_t* bucket_bit_base_i64,
                        uint64_t* bitstream_u64, int64_t bitstream_words, void* stream) {
    RectGeom g; CodeBook cb;
    int rc = rect_common(state, bf16_bits, ctx_bytes, bucket_table_i32, bucket_col_start_i32, bucket_col_len_i32,
                         bucket_row_offsets_i32, row_indices_i32, num_buckets, k, &g, &cb);
    if (rc) return rc;
    if (!bucket_thread_startbit_u32 || !bucket_bit_base_i64 || (bitstream_words > 0 && !bitstream_u64)) { set_error("sidecar emit: null argument"); return MPS_ERR_INVALID; }
    BuildState& S = *state_of(state);
    // the codes and team starts that the layout call left are laid out by its buckets and k
    if (num_buckets > 0 && (S.rect_buckets != num_buckets || S.rect_k != k || (S.rect_ragged != 0) != (g.group_col != nullptr))) {
        set_error("sidecar emit: call mps_build_rect_layout for the same buckets and sub-streams first");
        return MPS_ERR_INVALID;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (bitstream_words > 0) MPS_CUDA_TRY(cudaMemsetAsync(bitstream_u64, 0, (size_t)bitstream_words * 8, st));
    if (num_buckets > 0) {
        const lay::Shape shape = rect_shape(S, g);
        lay::Args a = rect_args(S, g, cb, shape);
        a.startbit = bucket_thread_startbit_u32;
        a.bit_base = reinterpret_cast<const long long*>(bucket_bit_base_i64);
        a.stream = reinterpret_cast<unsigned long long*>(bitstream_u64);
        rc = lay::launch_emit(a, shape, st);
        if (rc) return rc;
    }
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

// ---- shared-table layout -----------------------------------------------------------------------

int mps_build_shared_codebooks(mps_build_state* state, const int32_t* sid_lut_i32, int64_t num_scales,
                               int16_t* decode_syms_i16, uint8_t* decode_nbits_u8, void* stream) {
    if (!state || !sid_lut_i32 || !decode_syms_i16 || !decode_nbits_u8 || num_scales <= 0) {
        set_error("mps_build_shared_codebooks: bad argument");
        return MPS_ERR_INVALID;
    }
    BuildState& S = *state_of(state);
    if (S.variant != V_AWQ_SHARED) { set_error("state was not analyzed for the shared-table layout"); return MPS_ERR_INVALID; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t TS = 1ull << S.L;
    const long long num_streams = num_scales * 16;
    S.num_scales = num_scales;
    Carver C{S.ws, S.o_scratch, S.ws_bytes};
    auto* row_of = C.take<int>(S.G);
    auto* stream_ctx = C.take<int>(num_streams);
    S.o_sh_keep = (uint8_t*)row_of - S.ws;
    S.o_sh_end = align_up(C.off);
    MPS_CUDA_TRY(cudaMemsetAsync(decode_syms_i16, 0, (size_t)num_streams * TS * 2, st));
    MPS_CUDA_TRY(cudaMemsetAsync(decode_nbits_u8, 0, (size_t)num_streams * TS, st));
    MPS_CUDA_TRY(cudaMemsetAsync(stream_ctx, 0xFF, (size_t)num_streams * sizeof(int), st));
    shared_rows_kernel<<<grid_for(S.G), 256, 0, st>>>(reinterpret_cast<uint32_t*>(S.ws + S.o_ctx_key), S.G, sid_lut_i32, row_of, stream_ctx);
    int rc = run_codebooks(S, S.o_sh_end, row_of, reinterpret_cast<uint16_t*>(decode_syms_i16), decode_nbits_u8, st);
    if (rc) return rc;
    MPS_CUDA_TRY(cudaGetLastError());
    int flag = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&flag, S.d_flag + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (flag == 2) { set_error("Internal error: not enough packages"); return (int)cudaErrorUnknown; }
    return MPS_OK;
}

namespace {
struct SharedArrays {   // what the layout call leaves in the workspace for the emit call
    int* stream; uint32_t* lc; uint32_t* rel; int* chead; int* cidx;
};
SharedArrays shared_arrays(BuildState& S, Carver& C) {
    SharedArrays a;
    C.off = S.o_sh_end;
    a.stream = C.take<int>(S.numel);
    a.lc = C.take<uint32_t>(S.numel);
    a.rel = C.take<uint32_t>(S.numel);
    a.chead = C.take<int>(S.numel);
    a.cidx = C.take<int>(S.numel);
    return a;
}
}  // namespace

int mps_build_shared_layout(mps_build_state* state, const uint16_t* bf16_bits, const uint8_t* int4_u8,
                            const uint16_t* scales_u16, int32_t scale_mode, int64_t nb1, int64_t sb0, int64_t sb1,
                            const int32_t* sid_lut_i32, int64_t* scale_bit_base_i64, void* stream,
                            int64_t* num_chunks_out, int64_t* total_bits_out) {
    if (!state || !bf16_bits || !int4_u8 || !scales_u16 || !sid_lut_i32 || !scale_bit_base_i64 || !num_chunks_out ||
        !total_bits_out) {
        set_error("mps_build_shared_layout: null argument");
        return MPS_ERR_INVALID;
    }
    BuildState& S = *state_of(state);
    if (S.variant != V_AWQ_SHARED || S.num_scales <= 0) { set_error("call mps_build_shared_codebooks first"); return MPS_ERR_INVALID; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long numel = S.numel, NS = S.num_scales;
    Carver C{S.ws, 0, S.ws_bytes};
    SharedArrays A = shared_arrays(S, C);
    // scratch of this call
    auto* nbits = C.take<int>(numel);
    auto* tmp_a = C.take<int>(numel);      // run heads, then sorted scale ids
    auto* tmp_b = C.take<int>(numel);      // run starts, then sorted element ids
    auto* key = C.take<int>(numel);
    auto* val = C.take<int>(numel);
    auto* nb_sorted = C.take<unsigned long long>(numel);
    auto* cum = C.take<unsigned long long>(numel);
    auto* seg_base = C.take<unsigned long long>(NS);
    auto* seg_end = C.take<unsigned long long>(NS);
    auto* d_res = C.take<long long>(4);
    const size_t kCubTempBytes = cub_temp_bytes(numel);
    void* cub_tmp = C.take<uint8_t>(kCubTempBytes);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    // kept by mps_build_shared_codebooks: row_of [G], then stream_ctx [num_streams]
    auto* stream_ctx = reinterpret_cast<int*>(S.ws + align_up(S.o_sh_keep + (size_t)S.G * sizeof(int)));
    CodeBook cb{reinterpret_cast<unsigned long long*>(S.ws + S.o_items), reinterpret_cast<int*>(S.ws + S.o_ctx_ofs),
                reinterpret_cast<uint32_t*>(S.ws + S.o_enc), reinterpret_cast<uint32_t*>(S.ws + S.o_esc),
                reinterpret_cast<uint16_t*>(S.ws + S.o_escsym)};
    shared_elem_kernel<<<grid_for(numel), 256, 0, st>>>(bf16_bits, int4_u8, scales_u16, scale_mode, S.m, nb1, sb0, sb1,
                                                        sid_lut_i32, stream_ctx, cb, numel, A.stream, A.lc, nbits, tmp_a,
                                                        S.d_flag);
    MPS_CUDA_TRY(cudaGetLastError());
    size_t need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::InclusiveScan(cub_tmp, need, tmp_a, tmp_b, cub::Max(), (int)numel, st));
    shared_chunk_heads_kernel<<<grid_for(numel), 256, 0, st>>>(tmp_b, numel, A.chead);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, need, A.chead, A.cidx, (int)numel, st));
    // every scale's elements in flat order: stable sort by scale id
    shared_sid_keys_kernel<<<grid_for(numel), 256, 0, st>>>(A.stream, numel, key, val);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(cub_tmp, need, key, tmp_a, val, tmp_b, (int)numel, 0, 16, st));
    gather_bits_kernel<<<grid_for(numel), 256, 0, st>>>(nbits, tmp_b, numel, nb_sorted);
    need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceScan::InclusiveSum(cub_tmp, need, nb_sorted, cum, (int)numel, st));
    MPS_CUDA_TRY(cudaMemsetAsync(seg_base, 0, (size_t)NS * 8, st));
    MPS_CUDA_TRY(cudaMemsetAsync(seg_end, 0, (size_t)NS * 8, st));
    shared_segments_kernel<<<grid_for(numel), 256, 0, st>>>(tmp_a, nb_sorted, cum, numel, seg_base, seg_end);
    shared_relpos_kernel<<<grid_for(numel), 256, 0, st>>>(tmp_a, tmp_b, nb_sorted, cum, seg_base, numel, A.rel);
    shared_bases_kernel<<<1, 32, 0, st>>>(seg_base, seg_end, NS, reinterpret_cast<long long*>(scale_bit_base_i64), d_res);
    MPS_CUDA_TRY(cudaGetLastError());
    long long total_bits = 0;
    int last_head = 0, last_idx = 0, flag = 0;
    MPS_CUDA_TRY(cudaMemcpyAsync(&total_bits, d_res, sizeof(long long), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaMemcpyAsync(&last_head, A.chead + (numel - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaMemcpyAsync(&last_idx, A.cidx + (numel - 1), sizeof(int), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaMemcpyAsync(&flag, S.d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (flag == 3) { set_error("symbol not found in enc table for AWQ stream"); return (int)cudaErrorUnknown; }
    S.num_chunks = (long long)last_idx + last_head;
    *num_chunks_out = S.num_chunks;
    *total_bits_out = total_bits;
    return MPS_OK;
}

int mps_build_shared_emit(mps_build_state* state, const uint16_t* bf16_bits, const int64_t* scale_bit_base_i64,
                          uint64_t* bitstream_u64, int64_t bitstream_words, uint32_t* chunk_startbit_rel_u32,
                          uint32_t* chunk_out_base_u32, uint32_t* chunk_meta_u32, int32_t* chunk_scale_id_i32,
                          int32_t* out_idx_i32, int64_t* stream_chunk_ofs_i64, int32_t* stream_chunk_ids_i32, void* stream) {
    if (!state || !bf16_bits || !scale_bit_base_i64 || !bitstream_u64 || !chunk_startbit_rel_u32 || !chunk_out_base_u32 ||
        !chunk_meta_u32 || !chunk_scale_id_i32 || !out_idx_i32 || !stream_chunk_ofs_i64 || !stream_chunk_ids_i32) {
        set_error("mps_build_shared_emit: null argument (state %d, inputs %d%d, bitstream %d, chunks %d%d%d%d, out_idx %d, csr %d%d)",
                  state != nullptr, bf16_bits != nullptr, scale_bit_base_i64 != nullptr, bitstream_u64 != nullptr,
                  chunk_startbit_rel_u32 != nullptr, chunk_out_base_u32 != nullptr, chunk_meta_u32 != nullptr,
                  chunk_scale_id_i32 != nullptr, out_idx_i32 != nullptr, stream_chunk_ofs_i64 != nullptr,
                  stream_chunk_ids_i32 != nullptr);
        return MPS_ERR_INVALID;
    }
    BuildState& S = *state_of(state);
    if (S.variant != V_AWQ_SHARED || S.num_chunks <= 0) { set_error("call mps_build_shared_layout first"); return MPS_ERR_INVALID; }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long numel = S.numel, NC = S.num_chunks, num_streams = S.num_scales * 16;
    Carver C{S.ws, 0, S.ws_bytes};
    SharedArrays A = shared_arrays(S, C);
    auto* cpos = C.take<int>(NC + 1);
    auto* c_stream = C.take<int>(NC);
    auto* c_stream_sorted = C.take<int>(NC);
    auto* c_ids = C.take<int>(NC);
    const size_t kCubTempBytes = cub_temp_bytes(numel);
    void* cub_tmp = C.take<uint8_t>(kCubTempBytes);
    if (!C.ok()) { set_error("workspace too small"); return MPS_ERR_WORKSPACE; }
    shared_chunk_pos_kernel<<<grid_for(numel), 256, 0, st>>>(A.chead, A.cidx, numel, NC, cpos);
    shared_chunk_fill_kernel<<<grid_for(NC), 256, 0, st>>>(cpos, NC, A.stream, A.rel, chunk_startbit_rel_u32, chunk_out_base_u32,
                                                           chunk_meta_u32, chunk_scale_id_i32, c_stream);
    MPS_CUDA_TRY(cudaMemsetAsync(bitstream_u64, 0, (size_t)bitstream_words * 8, st));
    shared_emit_kernel<<<grid_for(numel), 256, 0, st>>>(bf16_bits, A.stream, A.lc, A.rel,
                                                        reinterpret_cast<const long long*>(scale_bit_base_i64), numel,
                                                        reinterpret_cast<unsigned long long*>(bitstream_u64));
    // chunk ids of every stream, ascending (stable sort by stream id) and the CSR offsets
    iota_i32_kernel<<<grid_for(NC), 256, 0, st>>>(c_ids, NC);
    size_t need = kCubTempBytes;
    MPS_CUDA_TRY(cub::DeviceRadixSort::SortPairs(cub_tmp, need, c_stream, c_stream_sorted, c_ids, stream_chunk_ids_i32, (int)NC,
                                                 0, 21, st));
    shared_stream_ofs_kernel<<<grid_for(num_streams + 1), 256, 0, st>>>(c_stream_sorted, NC, num_streams,
                                                                        reinterpret_cast<long long*>(stream_chunk_ofs_i64));
    iota_i32_kernel<<<grid_for(numel), 256, 0, st>>>(out_idx_i32, numel);
    MPS_CUDA_TRY(cudaGetLastError());
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    return MPS_OK;
}


}  // extern "C"
