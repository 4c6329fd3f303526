// AWQ "shared-table" sidecar: chunks of <=255 consecutive elements that share one (scale, qv)
// stream; every stream has a dense 2^L lookup table (int16 symbol + uint8 length, bit 7 = ESC).
//
// On random weights a chunk holds 1.1 elements on average, so the work is a gather, table entries
// read straight from global memory (L2), no shared-memory staging (a 6 KB table per ~200 symbols
// would cost more than it saves).  The table of a chunk is that of the stream that LISTS it, as in the
// reference kernel, not the one its metadata names; every stream counts (the reference launch stops
// at 65535 blocks).
//
// With scratch of a few bytes per chunk (mps_decode_awq_shared_table_ws) that list is inverted first: a
// pass over the positions writes every chunk's stream to `owner`, and the decode then takes the chunks
// in their own order, in which their metadata, code bits, element numbers and outputs are neighbours.
// In the order of the lists the chunks of a stream lie some sixteen apart, so that each of six arrays
// costs a line per chunk; a divergent access is what bounds both forms (the L1 looks up a line a cycle),
// and inverted only the two table lookups and the owner's write are left of eight.
// Measured, 4096 x 4096, 15.3 M chunks, 11 bits: 233 us (250 with the length of every entry looked up), in the order of the lists 442 us.
// Without scratch one thread per position of the index decodes in that order, the stream found by
// binary search in stream_chunk_ofs.
#include <type_traits>

#include "mps_common.cuh"

namespace mps {

__device__ __forceinline__ uint32_t peek_bits_global(const uint64_t* __restrict__ bs, long long nwords, long long bitpos,
                                                     int nbits) {
    const long long w = bitpos >> 6;
    const int o = (int)(bitpos & 63);
    const uint64_t a = (w >= 0 && w < nwords) ? __ldg(bs + w) : 0ull;
    // (the next word only where the bits reach into it)
    const uint64_t b = (o + nbits > 64 && w + 1 >= 0 && w + 1 < nwords) ? __ldg(bs + w + 1) : 0ull;
    const uint64_t hi = o ? ((a << o) | (b >> (64 - o))) : a;
    return (uint32_t)(hi >> (64 - nbits));
}

__global__ void __launch_bounds__(256)
shared_table_decode_kernel(const uint64_t* __restrict__ bs, long long nwords, const int16_t* __restrict__ syms,
                           const uint8_t* __restrict__ nbits, long long table_size, long long num_streams,
                           const long long* __restrict__ scale_bit_base, long long num_scales,
                           const uint32_t* __restrict__ chunk_startbit, const uint32_t* __restrict__ chunk_out_base,
                           const uint32_t* __restrict__ chunk_meta, const int32_t* __restrict__ chunk_scale_id,
                           long long num_chunks, const int32_t* __restrict__ out_idx,
                           const long long* __restrict__ stream_ofs, const int32_t* __restrict__ stream_ids,
                           long long out_len, int L, int16_t* __restrict__ out) {
    const long long npos = stream_ofs[num_streams] < num_chunks ? stream_ofs[num_streams] : num_chunks;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npos; p += (long long)gridDim.x * blockDim.x) {
        // stream s with stream_ofs[s] <= p < stream_ofs[s+1]
        long long lo = 0, hi = num_streams;
        while (hi - lo > 1) {
            const long long mid = (lo + hi) >> 1;
            if (__ldg(stream_ofs + mid) <= p) lo = mid; else hi = mid;
        }
        const long long s = lo;
        const long long chunk = stream_ids[p];
        if (chunk < 0 || chunk >= num_chunks) continue;
        const int sid = chunk_scale_id[chunk];
        if (sid < 0 || sid >= num_scales) continue;
        const uint32_t take = chunk_meta[chunk] >> 8;
        long long bitpos = scale_bit_base[sid] + (long long)chunk_startbit[chunk];
        const long long flat = chunk_out_base[chunk];
        const int16_t* ts = syms + s * table_size;
        const uint8_t* tn = nbits + s * table_size;
        for (uint32_t j = 0; j < take; ++j) {
            const uint32_t t = peek_bits_global(bs, nwords, bitpos, L);
            const uint32_t nb = __ldg(tn + t);
            int16_t sym = __ldg(ts + t);
            bitpos += nb & 0x7Fu;
            if (nb & 0x80u) {
                sym = (int16_t)peek_bits_global(bs, nwords, bitpos, 16);
                bitpos += 16;
            }
            const long long q = flat + j;
            if (q < out_len) {
                const long long dst = out_idx[q];
                if (dst >= 0 && dst < out_len) out[dst] = sym;
            }
        }
    }
}

// ---- with scratch: owner of every chunk, then the chunks in order -----------------------------------

constexpr int kOwnerPositions = 2048;   // positions of the stream index per CTA
constexpr int kSharedJ = 2;             // chunks a thread has in flight

// The last stream in [lo, hi) that starts at or before position p, by the whole warp (32 probes a round).
__device__ __forceinline__ long long stream_of_warp(const long long* __restrict__ ofs, long long lo, long long hi, long long p) {
    const int lane = threadIdx.x & 31;
    while (hi - lo > 1) {
        const long long step = (hi - lo + 31) >> 5;
        const long long i = lo + step * lane;
        const bool before = lane == 0 || (i < hi && __ldg(ofs + i) <= p);
        const int last = 31 - __clz((int)__ballot_sync(0xFFFFFFFFu, before));
        lo += step * last;
        hi = lo + step < hi ? lo + step : hi;
    }
    return lo;
}

// owner[chunk] = stream that lists it; chunks nobody lists keep the all-ones pattern they were filled with.  Its top bit says
// that the stream's table may hold an ESC: a chunk of one symbol, as nine in ten are, needs an entry's length for nothing else,
// and most tables hold none.  Streams are marked without a look where a CTA meets more than kOwnerTables of them or more than
// kOwnerLookBytes of their code lengths.  MARKS false: nothing is marked, and every chunk looks (marks_pay).
// (A look costs the bytes of the tables, what it saves some two thousand lookups.  us, lengths always looked up | a look whatever the
// bytes | up to 64 KB: 512 x 4096, 14 bits 89 | 91 | 85, 15 bits 107 | 118 | 103, 16 bits 124 | 159 | 124, 17 bits 134 | 230 | 134;
// 4096 x 4096, 15 bits 531 | 437 | 429, 16 bits 665 | 582 | 585, 17 bits 753 | 781 | 753.  96 and 128 KB: 14 bits 91 and 92.)
constexpr int kOwnerTables = 8;
constexpr long long kOwnerLookBytes = 65536;
template <typename T> constexpr T kEscMark = (T)((T)1 << (8 * sizeof(T) - 1));
template <typename T, bool MARKS>
__global__ void __launch_bounds__(256)
shared_owner_kernel(const long long* __restrict__ stream_ofs, long long num_streams, const int32_t* __restrict__ stream_ids,
                    long long num_chunks, const uint8_t* __restrict__ nbits, long long table_size, T* __restrict__ owner) {
    __shared__ long long s_range[2];
    __shared__ int s_esc[kOwnerTables];
    const long long npos = stream_ofs[num_streams] < num_chunks ? stream_ofs[num_streams] : num_chunks;
    const long long p0 = (long long)blockIdx.x * kOwnerPositions;
    if (p0 >= npos) return;
    const long long p1 = p0 + kOwnerPositions < npos ? p0 + kOwnerPositions : npos;
    const int warp = threadIdx.x >> 5;
    if (warp < 2) {
        const long long s = stream_of_warp(stream_ofs, 0, num_streams, warp == 0 ? p0 : p1 - 1);
        if ((threadIdx.x & 31) == 0) s_range[warp] = s;
    }
    __syncthreads();
    const long long first = s_range[0], end = s_range[1] + 1;
    const bool look = MARKS && end - first <= kOwnerTables && (end - first) * table_size <= kOwnerLookBytes;
    if (look) {
        if (threadIdx.x < kOwnerTables) s_esc[threadIdx.x] = 0;
        __syncthreads();
        const uint8_t* const tables = nbits + first * table_size;
        if (((reinterpret_cast<uintptr_t>(tables) | (uintptr_t)table_size) & 15u) == 0) {
            const long long pieces = table_size / 16;
            for (long long i = threadIdx.x; i < (end - first) * pieces; i += 256) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(tables) + i);
                if ((v.x | v.y | v.z | v.w) & 0x80808080u) s_esc[i / pieces] = 1;
            }
        } else {
            for (long long i = threadIdx.x; i < (end - first) * table_size; i += 256)
                if (__ldg(tables + i) & 0x80u) s_esc[i / table_size] = 1;
        }
        __syncthreads();
    }
    int32_t chunk[kOwnerPositions / 256];
#pragma unroll
    for (int i = 0; i < kOwnerPositions / 256; ++i) {
        const long long p = p0 + threadIdx.x + 256 * i;
        chunk[i] = p < p1 ? __ldcs(stream_ids + p) : -1;
    }
#pragma unroll
    for (int i = 0; i < kOwnerPositions / 256; ++i) {
        const long long p = p0 + threadIdx.x + 256 * i;
        if (chunk[i] < 0 || chunk[i] >= num_chunks) continue;
        long long lo = first, hi = end;
        while (hi - lo > 1) {
            const long long mid = (lo + hi) >> 1;
            if (__ldg(stream_ofs + mid) <= p) lo = mid; else hi = mid;
        }
        owner[chunk[i]] = (T)lo | (T)(MARKS && (!look || s_esc[lo - first]) ? kEscMark<T> : (T)0);
    }
}

template <typename T, bool MARKS>
__global__ void __launch_bounds__(256, 8)
shared_chunk_decode_kernel(const uint64_t* __restrict__ bs, long long nwords, const int16_t* __restrict__ syms,
                           const uint8_t* __restrict__ nbits, long long table_size, const long long* __restrict__ scale_bit_base,
                           long long num_scales, const uint32_t* __restrict__ chunk_startbit, const uint32_t* __restrict__ chunk_out_base,
                           const uint32_t* __restrict__ chunk_meta, const int32_t* __restrict__ chunk_scale_id, long long num_chunks,
                           const T* __restrict__ owner, const int32_t* __restrict__ out_idx, long long out_len, int L,
                           int16_t* __restrict__ out) {
    constexpr int J = kSharedJ;
    constexpr T kNone = (T)~(T)0;
    for (long long c0 = (long long)blockIdx.x * (256 * J); c0 < num_chunks; c0 += (long long)gridDim.x * (256 * J)) {
        T own[J];
        bool esc[J];
        int32_t sid[J];
        uint32_t take[J], flat[J], peek[J], nb[J];
        long long bit[J];
        int32_t dst[J];
        int16_t sym[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const long long c = c0 + threadIdx.x + 256 * j;
            const bool in = c < num_chunks;
            own[j] = in ? __ldcs(owner + c) : kNone;
            sid[j] = in ? __ldcs(chunk_scale_id + c) : -1;
            take[j] = in ? __ldcs(chunk_meta + c) >> 8 : 0u;
            flat[j] = in ? __ldcs(chunk_out_base + c) : 0u;
            bit[j] = in ? (long long)__ldcs(chunk_startbit + c) : 0;
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (own[j] == kNone || sid[j] < 0 || sid[j] >= num_scales) take[j] = 0u;
            esc[j] = !MARKS || (own[j] & kEscMark<T>) != 0;
            if (MARKS) own[j] &= (T)~kEscMark<T>;
            peek[j] = 0u;
            dst[j] = -1;
            if (take[j]) {
                if (flat[j] < out_len) dst[j] = __ldcs(out_idx + flat[j]);
                bit[j] += __ldg(scale_bit_base + sid[j]);
                peek[j] = peek_bits_global(bs, nwords, bit[j], L);
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            nb[j] = 0u; sym[j] = 0;
            if (take[j]) {
                // (nothing follows a chunk's only symbol whose length is then not asked for)
                if (esc[j] || take[j] > 1u) nb[j] = __ldg(nbits + (long long)own[j] * table_size + peek[j]);
                sym[j] = __ldg(syms + (long long)own[j] * table_size + peek[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            for (uint32_t i = 0; i < take[j]; ++i) {
                if (i) {   // (the first symbol's entry is here already)
                    const uint32_t t = peek_bits_global(bs, nwords, bit[j], L);
                    nb[j] = __ldg(nbits + (long long)own[j] * table_size + t);
                    sym[j] = __ldg(syms + (long long)own[j] * table_size + t);
                }
                bit[j] += nb[j] & 0x7Fu;
                if (nb[j] & 0x80u) {
                    sym[j] = (int16_t)peek_bits_global(bs, nwords, bit[j], 16);
                    bit[j] += 16;
                }
                const long long q = (long long)flat[j] + i;
                if (i) dst[j] = q < out_len ? __ldcs(out_idx + q) : -1;
                if (dst[j] >= 0 && dst[j] < out_len) out[dst[j]] = sym[j];
            }
        }
    }
}

// Whether streams are marked: where their numbers leave a bit for it, and tables are long enough for the lengths not looked up
// to pay for a look at each table.
// us, lengths always looked up | marks: 4096 x 4096, 6 bits 218 | 224, 7 bits 265 | 269, 8 bits 259 | 263, 9 bits 253 | 257 where one
// table in six holds an ESC and 236 | 226 where none does, 10 bits 245 | 241, 11 bits 253 | 233; 512 x 4096, 11 bits 62 | 60.
constexpr int64_t kMarksMinLen = 9;
static bool marks_pay(int64_t num_streams, bool narrow, int64_t max_len) {
    return max_len >= kMarksMinLen && num_streams < (narrow ? 0x7FFF : 0x7FFFFFFF);
}

static int shared_check(int64_t bitstream_words, int64_t num_streams, int64_t num_scales_plus1, int64_t num_chunks, int64_t out_len,
                        int64_t max_len) {
    if (max_len <= 0 || max_len > 20) { set_error("max_len must be in (0,20]"); return MPS_ERR_INVALID; }
    if (num_streams < 0 || num_chunks < 0 || out_len < 0 || num_scales_plus1 < 1 || bitstream_words < 0) {
        set_error("mps_decode_awq_shared_table: negative size");
        return MPS_ERR_INVALID;
    }
    return MPS_OK;
}

}  // namespace mps

using namespace mps;

extern "C" int mps_decode_awq_shared_table(const uint64_t* bitstream_u64, int64_t bitstream_words,
                                           const int16_t* decode_syms_i16, const uint8_t* decode_nbits_u8,
                                           int64_t num_streams, const int64_t* scale_bit_base_i64, int64_t num_scales_plus1,
                                           const uint32_t* chunk_startbit_rel_u32, const uint32_t* chunk_out_base_u32,
                                           const uint32_t* chunk_meta_u32, const int32_t* chunk_scale_id_i32,
                                           int64_t num_chunks, const int32_t* out_idx_i32,
                                           const int64_t* stream_chunk_ofs_i64, const int32_t* stream_chunk_ids_i32,
                                           int64_t out_len, int64_t max_len, int16_t* out_i16, void* stream) {
    const int rc = shared_check(bitstream_words, num_streams, num_scales_plus1, num_chunks, out_len, max_len);
    if (rc) return rc;
    if (num_chunks == 0 || num_streams == 0 || out_len == 0) return MPS_OK;
    if (!bitstream_u64 || !decode_syms_i16 || !decode_nbits_u8 || !scale_bit_base_i64 || !chunk_startbit_rel_u32 ||
        !chunk_out_base_u32 || !chunk_meta_u32 || !chunk_scale_id_i32 || !out_idx_i32 || !stream_chunk_ofs_i64 ||
        !stream_chunk_ids_i32 || !out_i16) {
        set_error("mps_decode_awq_shared_table: null device pointer");
        return MPS_ERR_INVALID;
    }
    const int threads = 256;
    long long blocks = (num_chunks + threads - 1) / threads;
    if (blocks > 148LL * 64) blocks = 148LL * 64;
    shared_table_decode_kernel<<<(int)blocks, threads, 0, static_cast<cudaStream_t>(stream)>>>(
        bitstream_u64, bitstream_words, decode_syms_i16, decode_nbits_u8, 1LL << max_len, num_streams,
        reinterpret_cast<const long long*>(scale_bit_base_i64), num_scales_plus1 - 1, chunk_startbit_rel_u32,
        chunk_out_base_u32, chunk_meta_u32, chunk_scale_id_i32, num_chunks, out_idx_i32,
        reinterpret_cast<const long long*>(stream_chunk_ofs_i64), stream_chunk_ids_i32, out_len, (int)max_len, out_i16);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

extern "C" size_t mps_shared_workspace_bytes(int64_t num_streams, int64_t num_chunks) {
    if (num_chunks <= 0) return 0;
    return (size_t)num_chunks * (num_streams < 0xFFFF ? sizeof(uint16_t) : sizeof(uint32_t));
}

extern "C" int mps_decode_awq_shared_table_ws(const uint64_t* bitstream_u64, int64_t bitstream_words,
                                              const int16_t* decode_syms_i16, const uint8_t* decode_nbits_u8,
                                              int64_t num_streams, const int64_t* scale_bit_base_i64, int64_t num_scales_plus1,
                                              const uint32_t* chunk_startbit_rel_u32, const uint32_t* chunk_out_base_u32,
                                              const uint32_t* chunk_meta_u32, const int32_t* chunk_scale_id_i32,
                                              int64_t num_chunks, const int32_t* out_idx_i32,
                                              const int64_t* stream_chunk_ofs_i64, const int32_t* stream_chunk_ids_i32,
                                              int64_t out_len, int64_t max_len, int16_t* out_i16, void* workspace,
                                              size_t workspace_bytes, void* stream) {
    const int rc = shared_check(bitstream_words, num_streams, num_scales_plus1, num_chunks, out_len, max_len);
    if (rc) return rc;
    if (num_chunks == 0 || num_streams == 0 || out_len == 0) return MPS_OK;
    if (!bitstream_u64 || !decode_syms_i16 || !decode_nbits_u8 || !scale_bit_base_i64 || !chunk_startbit_rel_u32 ||
        !chunk_out_base_u32 || !chunk_meta_u32 || !chunk_scale_id_i32 || !out_idx_i32 || !stream_chunk_ofs_i64 ||
        !stream_chunk_ids_i32 || !out_i16) {
        set_error("mps_decode_awq_shared_table_ws: null device pointer");
        return MPS_ERR_INVALID;
    }
    const size_t need = mps_shared_workspace_bytes(num_streams, num_chunks);
    const bool narrow = num_streams < 0xFFFF;
    if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 3u) != 0) {
        set_error("mps_decode_awq_shared_table_ws: workspace missing, too small or misaligned");
        return MPS_ERR_WORKSPACE;
    }
    const long long owner_blocks = (num_chunks + kOwnerPositions - 1) / kOwnerPositions;
    if (owner_blocks > 0x7FFFFFFFLL) { set_error("mps_decode_awq_shared_table_ws: too many chunks"); return MPS_ERR_INVALID; }
    long long blocks = (num_chunks + 256 * kSharedJ - 1) / (256 * kSharedJ);
    if (blocks > 148LL * 64) blocks = 148LL * 64;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    MPS_CUDA_TRY(cudaMemsetAsync(workspace, 0xFF, need, st));
    auto run = [&](auto* owner, auto marks) {
        using T = std::remove_pointer_t<decltype(owner)>;
        constexpr bool kMarks = decltype(marks)::value;
        shared_owner_kernel<T, kMarks><<<(unsigned)owner_blocks, 256, 0, st>>>(reinterpret_cast<const long long*>(stream_chunk_ofs_i64), num_streams,
                                                                    stream_chunk_ids_i32, num_chunks, decode_nbits_u8, 1LL << max_len, owner);
        shared_chunk_decode_kernel<T, kMarks><<<(unsigned)blocks, 256, 0, st>>>(
            bitstream_u64, bitstream_words, decode_syms_i16, decode_nbits_u8, 1LL << max_len,
            reinterpret_cast<const long long*>(scale_bit_base_i64), num_scales_plus1 - 1, chunk_startbit_rel_u32, chunk_out_base_u32,
            chunk_meta_u32, chunk_scale_id_i32, num_chunks, owner, out_idx_i32, out_len, (int)max_len, out_i16);
    };
    const bool marks = marks_pay(num_streams, narrow, max_len);
    if (narrow) marks ? run(static_cast<uint16_t*>(workspace), std::true_type()) : run(static_cast<uint16_t*>(workspace), std::false_type());
    else marks ? run(static_cast<uint32_t*>(workspace), std::true_type()) : run(static_cast<uint32_t*>(workspace), std::false_type());
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}
