// Direct path for tensors made of tiny buckets (AWQ with one bucket per 128-element group, small per-channel
// weights): staging 128 KB of fused tables per bucket would cost far more than decoding it, so codes are looked
// up in the sidecar's own tables in global memory (they stay in L2).  Parallelism comes from the number of
// sub-streams, which is what such tensors have plenty of.
//
// A warp takes a unit, up to `per_unit` neighbouring sub-streams of one bucket: what belongs to the bucket is read
// once per warp and not once per sub-stream.  Where a sub-stream is one symbol (a bucket of no more elements than
// sub-streams, the rule for INT4 on this path) a lane takes J of them, 32 apart: their loads are all in flight
// together and coalesced.  A length that nothing follows is only needed for its ESC mark, and an ESC code of the INT4
// formats has L bits: the mark is read only where the sub-stream has as many, some one symbol in ten.  (FP8's may have
// fewer: read always.  16 raw bits need not follow, the encoder leaves them out behind a symbol that equals the ESC
// symbol; what is there instead is read all the same, as everywhere.)  Bound: the latency of dependent loads, the L1's
// request path half busy; a divergent gather is what a symbol costs there, and little more than one is left of two.
// Measured, 4096 x 4096 INT4 of 131072 buckets x 256 sub-streams: 103 us (112 with eight CTAs' worth of blocks per place of the
// GPU and every unit's numbers read when it begins);
// 498 us with a thread per sub-stream and both lookups (half the threads without an element, every one of them reading its
// bucket's five numbers); two in flight instead of four: 155 us.  Tensors of few buckets: decode_direct.
#pragma once

#include "mps_common.cuh"

namespace mps {

constexpr int kDirectThreads = 256;

// A bucket as this path sees it (uniform across the warp).
struct DirectBucket {
    const uint32_t* bs32;
    const uint32_t* startbit;
    const int32_t* btab;
    uint32_t lim, bit_lo;
    long long row_a, col_start, col_len;
};

// Element `rr`, `cc` (row of the bucket, column in it): its offset in the tensor, or -1 where the row list is bad.
__device__ __forceinline__ long long direct_element(const mps_bucket_tensor& T, const DirectBucket& B, int mode, long long rr,
                                                    long long cc) {
    const long long row = T.row_indices[B.row_a + rr];
    const long long c0 = (mode == 2) ? (long long)T.group_col_start[B.row_a + rr] : B.col_start;
    const bool good = row >= 0 && row < T.n && c0 >= 0 && c0 + B.col_len <= T.m;
    return good ? row * T.m + c0 + cc : -1;
}

// Sub-streams [t_begin, t_end) of a bucket, any number of symbols each.
template <int L>
__device__ __forceinline__ void direct_run(const mps_bucket_tensor& T, const DirectBucket& B, int mode, uint32_t t_begin, uint32_t t_end,
                                           uint32_t k_eff, long long total) {
    constexpr int TS = 1 << L;
    for (uint32_t t = t_begin + (threadIdx.x & 31u); t < t_end; t += 32u) {
        BitWin win;
        win_init(win, B.bs32, B.lim, B.startbit[t] + B.bit_lo);
        for (long long e = t; e < total; e += k_eff) {
            const long long rr = e / B.col_len, cc = e - rr * B.col_len;
            const long long idx = direct_element(T, B, mode, rr, cc);
            const uint32_t ctx = idx >= 0 ? ((L == 7) ? T.ctx_bytes[idx] : (T.ctx_bytes[idx] & 0xFu)) : 0u;
            int32_t gid = B.btab[ctx];
            if (gid >= T.num_tables) gid = -1;
            const uint32_t peek = win.hi >> (32 - L);
            uint32_t sym = 0, len = 0, esc = 0;
            if (gid >= 0) {
                const uint32_t nib = (__ldg(T.decode_lens + (long long)gid * (TS / 2) + (peek >> 1)) >> ((peek & 1u) * 4u)) & 0xFu;
                sym = __ldg(T.decode_syms + (long long)gid * TS + peek);
                if constexpr (L == 7) { len = nib & 7u; esc = nib & 8u; }
                else { esc = (nib == 15u); len = esc ? (uint32_t)L : nib; }
            } else if constexpr (L != 7) {
                esc = 1u; len = (uint32_t)L;  // AWQ: a context without a table reads as an ESC
            }
            win_consume(win, len);
            if (esc) {
                sym = win.hi >> 16;
                win_consume(win, 16);
            }
            if (idx >= 0) T.out[idx] = (uint16_t)sym;
            if (win.avail <= 32) win_refill(win, B.bs32, B.lim);
        }
    }
}

// Sub-streams [t_begin, t_end) of a bucket in which each is one symbol.  ONE_ROW: of a bucket of one row, whose place is
// worked out once and not once per element.
template <int L, int J, bool ONE_ROW>
__device__ __forceinline__ void direct_run_one(const mps_bucket_tensor& T, const DirectBucket& B, int mode, uint32_t t_begin,
                                               uint32_t t_end) {
    constexpr int TS = 1 << L;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t col_len = (uint32_t)B.col_len;   // at most as many elements as sub-streams
    int32_t gid16 = -1;
    if constexpr (L == 11) {
        gid16 = B.btab[lane & 15u];
        if (gid16 >= T.num_tables) gid16 = -1;
    }
    const long long row = ONE_ROW ? direct_element(T, B, mode, 0, 0) : 0;
    for (uint32_t t0 = t_begin; t0 < t_end; t0 += 32u * J) {
        uint32_t bit[J], nbits[J], hi[J], lo[J], ctx[J];
        long long at[J];    // the element's offset in the tensor, -1 where the row list is bad (ONE_ROW: unused)
        int32_t gid[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint32_t t = t0 + 32u * j + lane;
            const uint32_t tc = t < t_end ? t : t_end - 1u;
            bit[j] = B.startbit[tc];
            nbits[j] = B.startbit[tc + 1u] - bit[j];    // (k + 1 start bits, and tc < k)
            if constexpr (!ONE_ROW) {
                const uint32_t rr = tc / col_len;
                at[j] = direct_element(T, B, mode, rr, tc - rr * col_len);
                ctx[j] = at[j] >= 0 ? (uint32_t)T.ctx_bytes[at[j]] : 0u;
            } else {
                at[j] = row;
                ctx[j] = row >= 0 ? (uint32_t)T.ctx_bytes[row + tc] : 0u;
            }
            bit[j] += B.bit_lo;
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const uint32_t u = bit[j] >> 5;
            hi[j] = ld_unit(B.bs32, u, B.lim);
            lo[j] = ld_unit(B.bs32, u + 1u, B.lim);
        }
        uint32_t sym[J], nib[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if constexpr (L == 11) {
                gid[j] = __shfl_sync(0xFFFFFFFFu, gid16, (int)(ctx[j] & 0xFu));
            } else {
                gid[j] = B.btab[ctx[j]];
                if (gid[j] >= T.num_tables) gid[j] = -1;
            }
            hi[j] = __funnelshift_l(lo[j], hi[j], bit[j]);
            lo[j] <<= (bit[j] & 31u);
            const uint32_t peek = hi[j] >> (32 - L);
            sym[j] = 0u;
            nib[j] = (L == 7) ? 0u : 15u;               // AWQ: a context without a table reads as an ESC of L bits
            if (gid[j] >= 0) {
                sym[j] = __ldg(T.decode_syms + (long long)gid[j] * TS + peek);
                nib[j] = 0u;
                if (L == 7 || nbits[j] >= (uint32_t)L)
                    nib[j] = (__ldg(T.decode_lens + (long long)gid[j] * (TS / 2) + (peek >> 1)) >> ((peek & 1u) * 4u)) & 0xFu;
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const bool esc = (L == 7) ? (nib[j] & 8u) != 0u : nib[j] == 15u;
            const uint32_t len = (L == 7) ? (nib[j] & 7u) : (uint32_t)L;
            if (esc) sym[j] = __funnelshift_l(lo[j], hi[j], len) >> 16;   // 33 bits of the window are valid at least
            const uint32_t t = t0 + 32u * j + lane;
            if (t < t_end && at[j] >= 0) st_stream_u16(T.out + (ONE_ROW ? row + t : at[j]), sym[j]);
        }
    }
}

// What belongs to a bucket, as it lies in memory (uniform across the warp).
struct DirectNumbers { int32_t row_a, row_e, col_start, col_len; long long bit_base; };
__device__ __forceinline__ DirectNumbers direct_numbers(const mps_bucket_tensor& T, long long b) {
    DirectNumbers n;
    n.row_a = T.bucket_row_offsets[b];
    n.row_e = T.bucket_row_offsets[b + 1];
    n.col_start = 0;
    n.col_len = T.group_size;
    if (T.mode != 2) { n.col_start = T.bucket_col_start[b]; n.col_len = T.bucket_col_len[b]; }
    n.bit_base = T.bucket_bit_base[b];
    return n;
}

constexpr int kDirectResident = 4;   // CTAs per SM with four symbols in flight per lane
template <int L, int J>
__global__ void __launch_bounds__(kDirectThreads, J == 4 ? kDirectResident : 0)
direct_decode_kernel(const __grid_constant__ mps_bucket_tensor T, uint32_t per_unit, uint32_t parts, long long units) {
    constexpr int NCTX = (L == 7) ? 256 : 16;
    const int mode = T.mode;
    const long long k = T.k;
    const long long warps = (long long)gridDim.x * (kDirectThreads / 32);
    long long u = (long long)blockIdx.x * (kDirectThreads / 32) + (threadIdx.x >> 5);
    // Four in flight, a warp after many units: the next unit's numbers are on their way while one is decoded, one trip to memory
    // of four that depend on each other.  The others have a unit or two per warp, and more warps per SM without (INT4
    // 4096 x 2048, k = 64, us: 100 | 107 with).
    constexpr bool kAhead = J == 4;
    DirectNumbers next;
    if constexpr (kAhead) {
        if (u >= units) return;
        next = direct_numbers(T, parts == 1u ? u : u / parts);
    }
    for (; u < units; u += warps) {
        const long long b = parts == 1u ? u : u / parts;
        const uint32_t t_begin = (uint32_t)(u - b * parts) * per_unit;
        DirectBucket B;
        long long row_e, bit_base;
        if constexpr (kAhead) {
            const DirectNumbers num = next;
            if (u + warps < units) next = direct_numbers(T, parts == 1u ? u + warps : (u + warps) / parts);
            B.row_a = num.row_a; row_e = num.row_e; B.col_start = num.col_start; B.col_len = num.col_len; bit_base = num.bit_base;
        } else {
            B.row_a = T.bucket_row_offsets[b];
            row_e = T.bucket_row_offsets[b + 1];
            B.col_start = 0;
            B.col_len = T.group_size;
            if (mode != 2) { B.col_start = T.bucket_col_start[b]; B.col_len = T.bucket_col_len[b]; }
            bit_base = T.bucket_bit_base[b];
        }
        const long long nrows = row_e - B.row_a;
        const long long wb = bit_base >> 6;
        const bool ok = nrows > 0 && B.col_len > 0 && B.row_a >= 0 && B.row_a + nrows <= T.num_rows &&
                        (mode == 2 || (B.col_start >= 0 && B.col_start + B.col_len <= T.m)) && bit_base >= 0 && wb < T.bitstream_words;
        if (!ok) continue;
        const long long total = nrows * B.col_len;
        const uint32_t k_eff = (total < k) ? (uint32_t)total : (uint32_t)k;
        if (t_begin >= k_eff) continue;
        const uint32_t t_end = k_eff - t_begin < per_unit ? k_eff : t_begin + per_unit;
        B.bs32 = reinterpret_cast<const uint32_t*>(T.bitstream) + 2 * wb;
        const long long units32 = 2 * (T.bitstream_words - wb);
        B.lim = (uint32_t)((units32 > 0x7FFFFFFELL ? 0x7FFFFFFELL : units32) - 1);
        B.startbit = T.thread_startbit + b * (k + 1);
        B.btab = T.bucket_table + b * NCTX;
        B.bit_lo = (uint32_t)(bit_base & 63);
        if constexpr (J > 1) {
            if (total <= k) {
                if (nrows == 1) direct_run_one<L, J, true>(T, B, mode, t_begin, t_end);
                else direct_run_one<L, J, false>(T, B, mode, t_begin, t_end);
                continue;
            }
        }
        direct_run<L>(T, B, mode, t_begin, t_end, k_eff, total);
    }
}

}  // namespace mps
