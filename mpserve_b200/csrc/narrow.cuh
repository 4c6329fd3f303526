// Decode of work items that are 256 sub-streams wide, one per thread: buckets of at most 256
// sub-streams (every by-scale sidecar the reference's script writes, per-channel sidecars of the builder's default), and
// tensors of so few sub-streams that wider items would leave SMs without work.
//
// Bound: latency and issue slots.  A sub-stream is a serial chain -- table lookup, shift, next lookup -- and an item has
// eight warps of it:
//  * the tables stay as the sidecar stores them, 16-bit symbols and 4-bit lengths: 80 KB instead of the 128 KB of fused
//    entries, so that two CTAs share an SM and one's start (tables, row list, first chunks) hides behind the other's
//    decoding; nothing is expanded (with fused entries and one CTA per SM a step is no faster, and staging takes 8 us an
//    item: by-scale 291 instead of 176 us), and the symbol's lookup is off the chain;
//  * the next bits wait in a 64-bit window whose refill comes from a unit read one refill earlier; refill, requests and
//    ESC are predicated, not branches, so that a block of steps is one stretch of code to schedule, short enough for the
//    instruction cache (three blocks unrolled: a third more time, waiting for instructions);
//  * a ninth warp brings the context bytes, two stages of sixteen steps ahead, through plain loads, so that any row
//    length and alignment takes this path; a load to registers in the decoding warps themselves costs its whole latency
//    once per block, however early it is issued: what waits for a table lookup then waits for it too (203 -> 230 us);
//  * the bitstream runs through the ring of four 16-byte chunks per sub-stream of the wide kernel.
// Measured (before: the wide kernel with one chain per thread): INT4 by scale 14336 x 4096 147 us (254), 4096 x 4096 76
// (94), FP8 2047 x 3000 31 (76), 4096 x 4096 with one scale 45 (51).  Where the wide kernel stays: narrow_pays.
#pragma once

#include <type_traits>

#include "stream_common.cuh"

namespace mps {
namespace narrow {

constexpr int kSpan = 256;            // sub-streams of an item
constexpr int kThreads = kSpan;       // decoding threads; one more warp brings context bytes
constexpr int kAll = kThreads + 32;
constexpr int kEntries = 32768;       // 256 contexts x 2^7 == 16 contexts x 2^11
constexpr int kRows = 1024;           // rows / groups of a bucket kept in shared memory
constexpr int kBlock = 8;             // steps per block
constexpr int kStage = 16;            // steps per stage of the ring of context bytes, which has two
constexpr int kChunks = 4;            // 16-byte chunks of bitstream per sub-stream

struct Smem {
    uint16_t syms[kEntries];
    uint8_t lens[kEntries / 2];       // two 4-bit entries per byte, low half first
    uint4 ring[kSpan * kChunks];
    uint8_t ctxring[2 * kStage * kSpan];
    uint32_t rowbase[kRows];          // element offset of every row's first element (an invalid row leaves the fast path)
    int32_t gid[256];                 // context -> table id of the staged tables
    mps_bucket_tensor tensor;
    int next_item;
    uint16_t order[kOrderMost];       // buckets of a lone tensor, longest first
};
static_assert(sizeof(Smem) <= 113 * 1024, "two CTAs per SM");

template <int L> struct Fmt {
    static constexpr int kCtx = (L == 7) ? 256 : 16;
    static constexpr int TS = 1 << L;
    // symbols between two refills: the window holds at least 33 bits after one
    static constexpr int kPerRefill = (L == 7) ? 4 : 2;
    static constexpr uint32_t kCtxMask = (L == 7) ? 0xFFu : 0x0Fu;
};

// ---- the 64-bit window over a sub-stream's ring ------------------------------------------------------
// hi:lo hold the next `avail` bits, left-aligned, zeros below; nx is unit r of the stream (units of 32 bits in bit
// order), the first that is not in the window.  Unit x lies at bytes 4 * (x ^ 1).
struct Win {
    uint32_t hi, lo, nx;
    int avail;
    uint32_t r4;      // 4 * r
};

__device__ __forceinline__ uint32_t ring_ld(uint32_t ring, uint32_t r4) { return lds_ordered(ring + ((r4 ^ 4u) & 60u)); }

__device__ __forceinline__ void win_start(Win& w, uint32_t ring, uint32_t pos) {
    const uint32_t u4 = (pos >> 5) << 2, off = pos & 31u;
    const uint32_t a = ring_ld(ring, u4), b = ring_ld(ring, u4 + 4u);
    w.hi = __funnelshift_l(b, a, off);
    w.lo = b << off;
    w.avail = 64 - (int)off;
    w.r4 = u4 + 8u;
    w.nx = ring_ld(ring, w.r4);
}

// Appends unit r where the window has room for it (avail <= 32; its low half is empty then) and reads the next.
__device__ __forceinline__ void win_fill(Win& w, uint32_t ring) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 t, a;\n\t"
        "setp.le.s32 p, %3, 32;\n\t"
        "shf.r.clamp.b32 t, %2, 0, %3;\n\t"       // (nothing where avail > 32)
        "or.b32 %0, %0, t;\n\t"
        "@p shf.r.clamp.b32 %1, 0, %2, %3;\n\t"
        "@p add.s32 %3, %3, 32;\n\t"
        "@p add.u32 %4, %4, 4;\n\t"
        "lop3.b32 a, %4, 4, 60, 0x28;\n\t"        // (r4 ^ 4) & 60
        "add.u32 a, a, %5;\n\t"
        "@p ld.shared.u32 %2, [a];\n\t}"
        : "+r"(w.hi), "+r"(w.lo), "+r"(w.nx), "+r"(w.avail), "+r"(w.r4) : "r"(ring) : "memory");
}

__device__ __forceinline__ void win_take(Win& w, uint32_t n) {
    w.hi = __funnelshift_l(w.lo, w.hi, n);
    w.lo <<= n;
    w.avail -= (int)n;
}

// One chunk of the bitstream into the ring: nothing past its end, the last 8 bytes alone where it ends mid-chunk.
__device__ __forceinline__ void fetch_chunk(uint32_t ring, const BitOrigin& bo, uint32_t ofs) {
    const uint32_t dst = ring + (ofs & 63u);
    if (ofs <= bo.last_ofs) cp_async_16(dst, bo.base + ofs);
    else if (ofs == bo.tail_ofs) cp_async_8(dst, bo.base + ofs);
}

// The same, predicated, for the next chunk of a ring if it is due: chunks below the one three after unit r + 1 must be on
// their way.
__device__ __forceinline__ void request(const Win& w, uint32_t& next, uint32_t ring, const BitOrigin& bo) {
    const uint32_t need = ((w.r4 + 4u) >> 4) + kChunks;
    const uint32_t ofs = next << 4;
    asm volatile(
        "{\n\t.reg .pred p, q, r;\n\t"
        "setp.lt.u32 p, %0, %1;\n\t"
        "setp.le.and.u32 q, %4, %5, p;\n\t"
        "setp.eq.and.u32 r, %4, %6, p;\n\t"
        "@q cp.async.cg.shared.global [%2], [%3], 16;\n\t"
        "@r cp.async.ca.shared.global [%2], [%3], 8;\n\t"
        "@p add.u32 %0, %0, 1;\n\t}"
        : "+r"(next) : "r"(need), "r"(ring + (ofs & 63u)), "l"(bo.base + ofs), "r"(ofs), "r"(bo.last_ofs), "r"(bo.tail_ofs) : "memory");
}

struct Item {
    const uint8_t* ctx;
    uint16_t* out;
    uint32_t t;                      // first sub-stream of this thread's
    uint32_t total, k_eff, col_len, nrows;
    uint32_t item_steps;             // most symbols of a sub-stream of the item
    BitOrigin bo;
    __device__ __forceinline__ uint32_t steps(uint32_t sub) const { return sub < k_eff ? (total - sub - 1u) / k_eff + 1u : 0u; }
};

// (row, column) of a sub-stream's element, moved on by k_eff elements a step; past the bucket's end it stays in its last row
struct Walk {
    uint32_t row4, col, last4;       // shared-memory address of the row's base, column, address of the last row's base
    uint32_t d_row4, d_col, col_len;
};

__device__ __forceinline__ uint32_t walk_next(Walk& w) {
    uint32_t base;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(base) : "r"(w.row4));
    const uint32_t ofs = base + w.col;
    w.row4 += w.d_row4;
    w.col += w.d_col;
    if (w.col >= w.col_len) { w.col -= w.col_len; w.row4 += 4u; }
    w.row4 = w.row4 < w.last4 ? w.row4 : w.last4;
    return ofs;
}

__device__ __forceinline__ Walk walk_from(const Smem& sm, const Item& it, uint32_t t) {
    Walk w;
    const uint32_t rr = t / it.col_len, q = it.k_eff / it.col_len;
    w.col_len = it.col_len;
    w.last4 = smem_u32(sm.rowbase) + (it.nrows - 1u) * 4u;
    w.row4 = smem_u32(sm.rowbase) + (rr < it.nrows ? rr : it.nrows - 1u) * 4u;
    w.col = t - rr * it.col_len;
    w.d_row4 = q * 4u;
    w.d_col = it.k_eff - q * it.col_len;
    return w;
}

// Hardware barriers between the warp that brings context bytes and the decoding ones: 1, 2: a stage is full; 3, 4: it
// may be overwritten.  Both sides go through the same number of stages.
__device__ __forceinline__ void named_sync(uint32_t id) { asm volatile("barrier.sync %0, %1;" ::"r"(id), "n"(kAll) : "memory"); }
__device__ __forceinline__ void named_arrive(uint32_t id) { asm volatile("barrier.arrive %0, %1;" ::"r"(id), "n"(kAll) : "memory"); }

// The context bytes of an item, step by step.  WIDE: rows and steps come in eights, a lane has eight neighbouring
// sub-streams; else it has every 32nd, a byte each.
template <bool WIDE>
__device__ __forceinline__ void bring_ctx(Smem& sm, const Item& it, uint32_t t_begin) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stages = (it.item_steps + kStage - 1) / kStage;
    if constexpr (WIDE) {
        Walk w = walk_from(sm, it, t_begin + 8u * lane);
        for (uint32_t j = 0; j < stages; ++j) {
            uint2 v[kStage];
#pragma unroll
            for (int u = 0; u < kStage; ++u) v[u] = ld_stream_u64(it.ctx + walk_next(w));
            if (j >= 2u) named_sync(3u + (j & 1u));
            uint8_t* dst = sm.ctxring + (j & 1u) * (kStage * kSpan) + 8u * lane;
#pragma unroll
            for (int u = 0; u < kStage; ++u) *reinterpret_cast<uint2*>(dst + u * kSpan) = v[u];
            named_arrive(1u + (j & 1u));
        }
    } else {
        Walk w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = walk_from(sm, it, t_begin + lane + 32u * i);
        for (uint32_t j = 0; j < stages; ++j) {
            if (j >= 2u) named_sync(3u + (j & 1u));
            uint8_t* dst = sm.ctxring + (j & 1u) * (kStage * kSpan) + lane;
#pragma unroll 1
            for (int u = 0; u < kStage; u += 4) {
                uint32_t v[4][8];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[q][i] = ld_stream_u8(it.ctx + walk_next(w[i]));
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) dst[(u + q) * kSpan + 32 * i] = (uint8_t)v[q][i];
            }
            named_arrive(1u + (j & 1u));
        }
    }
}

// idx = context << L | next L bits: the 4-bit entry is nibble idx of the lengths
__device__ __forceinline__ uint32_t lens_at(uint32_t lens, uint32_t idx) {
    uint32_t w;
    asm("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(lens + ((idx >> 1) & ~3u)));
    return __funnelshift_r(w, 0u, idx << 2) & 0xFu;
}
__device__ __forceinline__ uint32_t sym_at(uint32_t syms, uint32_t idx) {
    uint32_t v;
    asm("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(syms + idx * 2u));
    return v;
}

// One sub-stream; called by all decoding threads.  Returns whether the loop without ESC met a length that is none (a
// context without a table, L = 11).
template <int L, bool ESC>
__device__ __forceinline__ bool run(Smem& sm, const Item& it, uint32_t pos) {
    constexpr int kMaxBits = ESC ? L + 16 : L;             // most bits of one step
    constexpr int kPeriod = ESC ? kBlock / 2 : kBlock;     // steps between requests for bitstream
    // (an ESC symbol and its 16 raw bits come out of one window: no branch, at the price of a refill per symbol)
    constexpr int kPerRefill = ESC ? 1 : Fmt<L>::kPerRefill;
    static_assert(kPerRefill * kMaxBits <= 33, "the window holds at least 33 bits after a refill");
    // a request sees the unit it stands at; that unit moves on by at most one chunk between two requests ...
    static_assert(kPeriod * kMaxBits + 31 < 5 * 32, "one request per period is enough");
    // ... and a chunk must have landed when it has moved on by three.  Without ESC that takes at least kNeed steps (the
    // window's filling level accounts for up to 31 bits), so groups of requests older than kLag periods must have landed.
    // With ESC the same reasoning would leave two periods, less than a trip to memory: every step would wait for it,
    // for the sake of codes that are one in a thousand.  There kLag periods are right as long as no period moves on by
    // more than kUnits units: kLag * kUnits <= 9 - 1, the chunk of unit r + 4 then lies below the first one not asked
    // for kLag periods ago, ((r' + 1) >> 2) + 4.  A period that does is followed by kLag of waits for everything.
    constexpr int kNeed = (3 * 128 - 31 + L - 1) / L;
    constexpr int kUnits = (L == 7) ? 1 : 2;
    constexpr int kLag = ESC ? 8 / kUnits : kNeed / kPeriod - 2;
    static_assert(kLag >= 0, "the ring is too short");
    const uint32_t syms = smem_u32(sm.syms), lens = smem_u32(sm.lens), ring = smem_u32(sm.ring) + threadIdx.x * 64u;
    const uint32_t ctx0 = smem_u32(sm.ctxring) + threadIdx.x;
    Win w;
    win_start(w, ring, pos);
    uint32_t next = (pos >> 7) + kChunks, most = 0;
    Walk walk = walk_from(sm, it, it.t);
    const uint32_t steps = it.steps(it.t);
    uint32_t last4 = w.r4, strict = 0;   // (ESC) unit of the last request, periods yet to wait for everything
    request(w, next, ring, it.bo);
    cp_async_commit();
    // (steps past the end are decoded like any other, from whatever bits and bytes there are, and not stored: one copy of
    // the code, small enough for the instruction cache)
#pragma unroll 1
    for (uint32_t s = 0; s < it.item_steps; s += kBlock) {
        const uint32_t stage = (s / kStage) & 1u;
        if (s % kStage == 0) named_sync(1u + stage);
        const uint32_t ctx = ctx0 + stage * (kStage * kSpan) + (s % kStage) * kSpan;
        uint32_t val[kBlock], ofs[kBlock];
#pragma unroll
        for (int u = 0; u < kBlock; ++u) asm volatile("ld.shared.u8 %0, [%1];" : "=r"(val[u]) : "r"(ctx + u * kSpan) : "memory");
#pragma unroll
        for (int u = 0; u < kBlock; ++u) ofs[u] = walk_next(walk);
        const uint32_t left = steps > s ? steps - s : 0u;
#pragma unroll
        for (int u = 0; u < kBlock; ++u) {
            if (u % kPerRefill == 0) win_fill(w, ring);
            const uint32_t idx = __funnelshift_l(w.hi, val[u] & Fmt<L>::kCtxMask, L);
            uint32_t len = lens_at(lens, idx), sym = sym_at(syms, idx);
            if constexpr (ESC) {       // 16 raw bits follow the code
                if constexpr (L == 7) {
                    const uint32_t raw = __funnelshift_l(w.lo, w.hi, len & 7u) >> 16;
                    sym = (len & 8u) ? raw : sym;
                    len += len & 8u;                   // 8 + code length -> 16 + code length
                } else {
                    const bool esc = len == 15u;       // a code of L bits
                    sym = esc ? w.hi >> (32 - L - 16) : sym;   // (the low 16 bits are stored)
                    len = esc ? (uint32_t)(L + 16) : len;
                }
            } else if constexpr (L == 11) {
                if ((uint32_t)u < left) most = most > len ? most : len;
            }
            win_take(w, len);
            uint16_t* dst;
            asm("mad.wide.u32 %0, %1, 2, %2;" : "=l"(dst) : "r"(ofs[u]), "l"(it.out));
            if ((uint32_t)u < left) st_stream_u16(dst, sym);
            if ((u + 1) % kPeriod == 0) {
                request(w, next, ring, it.bo);
                cp_async_commit();
                if constexpr (ESC) {
                    strict = w.r4 - last4 > 4u * kUnits ? kLag + 1u : strict;
                    last4 = w.r4;
                    if (strict) { --strict; cp_async_wait<0>(); }
                }
                cp_async_wait<kLag>();
            }
        }
        if (s % kStage != 0 && s + kBlock + kStage < (it.item_steps + kStage - 1) / kStage * kStage) named_arrive(3u + stage);
    }
    cp_async_wait<0>();
    return most > (uint32_t)L;
}

// Items outside the fast path: rows that are invalid or too many for shared memory, offsets of more than 32 bits, a
// bitstream whose chunks cannot be copied.  One element at a time, 64-bit indices, every access checked.
template <int L>
__device__ void run_general(const Smem& sm, const mps_bucket_tensor& T, const uint32_t* __restrict__ bs32, uint32_t lim, uint32_t bit,
                            uint32_t t, uint32_t k_eff, long long col_len, long long col_start, long long row_a, long long total) {
    BitWin w;
    win_init(w, bs32, lim, bit);
    for (long long e = t; e < total; e += k_eff) {
        const long long rr = e / col_len, cc = e - rr * col_len;
        const long long row = T.row_indices[row_a + rr];
        const long long c0 = (T.mode == 2) ? (long long)T.group_col_start[row_a + rr] : col_start;
        const bool good = row >= 0 && row < T.n && c0 >= 0 && c0 + col_len <= T.m;
        const long long at = row * T.m + c0 + cc;
        const uint32_t ctx = good ? (T.ctx_bytes[at] & Fmt<L>::kCtxMask) : 0u;
        const uint32_t idx = (ctx << L) + (w.hi >> (32 - L));
        uint32_t len = (sm.lens[idx >> 1] >> ((idx & 1u) * 4u)) & 0xFu, sym = sm.syms[idx];
        bool esc;
        if constexpr (L == 7) { esc = (len & 8u) != 0u; len &= 7u; }
        else { esc = (len == 15u); len = esc ? (uint32_t)L : len; }
        win_consume(w, len);
        if (esc) { sym = w.hi >> 16; win_consume(w, 16u); }
        if (good) T.out[at] = (uint16_t)sym;
        if (w.avail <= 32) win_refill(w, bs32, lim);
    }
}

// Raw tables of all contexts into shared memory (asynchronously where the alignment allows; the caller waits).  A
// context without a table: the FP8 decoder emits zeros and consumes nothing, the AWQ decoders read an ESC of L bits.
template <int L>
__device__ __forceinline__ void stage(Smem& sm, const mps_bucket_tensor& T) {
    constexpr int TS = Fmt<L>::TS;
    constexpr int kSymPieces = TS / 8, kLenPieces = TS / 32;      // 16-byte pieces of a context's symbols and lengths
    const bool aligned = ((reinterpret_cast<uintptr_t>(T.decode_syms) | reinterpret_cast<uintptr_t>(T.decode_lens)) & 15u) == 0;
    constexpr uint32_t kFill = (L == 7) ? 0u : 0xFFFFFFFFu;
    // the threads that copy one context's symbols (lengths) are kSymPieces (kLenPieces) neighbours, or all of them
    constexpr int kSymThreads = kSymPieces < kThreads ? kSymPieces : kThreads;
    constexpr int kLenThreads = kLenPieces < kThreads ? kLenPieces : kThreads;
    auto piece = [&](uint8_t* dst, const uint8_t* src, int32_t gid, uint32_t fill) {
        if (gid < 0) *reinterpret_cast<uint4*>(dst) = make_uint4(fill, fill, fill, fill);
        else if (aligned) cp_async_16(smem_u32(dst), src);
        else for (int q = 0; q < 16; ++q) dst[q] = src[q];
    };
    const int tid = threadIdx.x;
#pragma unroll 4
    for (int c = tid / kSymThreads; c < Fmt<L>::kCtx; c += kThreads / kSymThreads) {
        const int32_t gid = sm.gid[c];
        const uint8_t* src = reinterpret_cast<const uint8_t*>(T.decode_syms) + (long long)gid * (TS * 2);
        uint8_t* dst = reinterpret_cast<uint8_t*>(sm.syms) + c * (TS * 2);
#pragma unroll
        for (int i = tid % kSymThreads; i < kSymPieces; i += kSymThreads) piece(dst + i * 16, src + i * 16, gid, 0u);
    }
#pragma unroll 4
    for (int c = tid / kLenThreads; c < Fmt<L>::kCtx; c += kThreads / kLenThreads) {
        const int32_t gid = sm.gid[c];
        const uint8_t* src = T.decode_lens + (long long)gid * (TS / 2);
        uint8_t* dst = sm.lens + c * (TS / 2);
#pragma unroll
        for (int i = tid % kLenThreads; i < kLenPieces; i += kLenThreads) piece(dst + i * 16, src + i * 16, gid, kFill);
    }
}

// Does any staged length carry the ESC mark?  (this thread's share)
template <int L>
__device__ __forceinline__ bool any_esc(const Smem& sm) {
    uint32_t any = 0;
#pragma unroll
    for (int i = threadIdx.x; i < kEntries / 32; i += kThreads) {
        if (L == 11 && sm.gid[i / (Fmt<L>::TS / 32)] < 0) continue;   // (no table: the loop without ESC finds out if it is met)
        const uint4 v = reinterpret_cast<const uint4*>(sm.lens)[i];
        auto mark = [](uint32_t x) { return L == 7 ? x : (x & (x >> 1) & (x >> 2) & (x >> 3)); };   // top (L = 7) or low bit of a nibble
        any |= mark(v.x) | mark(v.y) | mark(v.z) | mark(v.w);
    }
    any &= (L == 7) ? 0x88888888u : 0x11111111u;
    return any != 0u;
}

// ORDERED: a lone tensor whose buckets are taken longest first (orders_itself).  ONE: no more items than CTAs and no order but
// their numbers'; without the questions that the others ask, none of them in the loop over the steps, such launches are 1.5 %
// faster (FP8 2047 x 3000 of 290 buckets, three weights, us: 34.6, 33.3, 32.4 | 35.1, 33.8, 32.9 with).
template <int L, bool ORDERED, bool ONE>
__global__ void __launch_bounds__(kAll, 2)
narrow_decode_kernel(const __grid_constant__ BatchArgs args, unsigned int* __restrict__ ws) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    constexpr int NCTX = Fmt<L>::kCtx;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool decoding = tid < kThreads;
    constexpr int kGids = (NCTX + kThreads - 1) / kThreads;
    int item = (int)blockIdx.x;      // a CTA's first item is the one of its number: the queue counts from the grid size on
    int staged_ti = -1;
    bool esc = false;
    if constexpr (ORDERED) order_by_length<kAll / 32>(args.single, reinterpret_cast<uint32_t*>(sm.syms), sm.order);
    while (item < args.total_items) {
        int ti = 0;
        long long local = item;
        [[maybe_unused]] uint4 entry = make_uint4(0u, 0u, 0u, 0u);
        if (!ONE && args.order != nullptr) {
            entry = args.order[item];
            ti = (int)entry.x;
        } else if (args.tensors != nullptr) {
            int lo = 0, hi = args.count;  // largest ti with prefix[ti] <= item
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (args.item_prefix[mid] <= item) lo = mid; else hi = mid;
            }
            ti = lo;
            local = item - args.item_prefix[ti];
        }
        if constexpr (ONE) { if (tid == kThreads) sm.next_item = args.total_items; }
        if (ti != staged_ti) {
            const uint32_t* src = reinterpret_cast<const uint32_t*>((args.tensors != nullptr) ? &args.tensors[ti] : &args.single);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&sm.tensor);
            for (int i = tid; i < (int)(sizeof(mps_bucket_tensor) / 4); i += kAll) dst[i] = src[i];
            __syncthreads();
        }
        const mps_bucket_tensor& T = sm.tensor;
        const int mode = T.mode;
        const uint32_t k = (uint32_t)T.k;
        const uint32_t chunks = (k + kSpan - 1) / kSpan;
        long long b = !ONE && args.order != nullptr ? (long long)entry.y : local / chunks;
        const uint32_t t_begin = !ONE && args.order != nullptr ? entry.z : (uint32_t)(local - b * chunks) * kSpan;
        if constexpr (ORDERED) b = sm.order[b];
        const uint32_t t = t_begin + tid;
        // everything that depends on the bucket's number alone is requested before any of it is used
        const long long row_a = T.bucket_row_offsets[b];
        const long long row_e = T.bucket_row_offsets[b + 1];
        long long col_start = 0, col_len = T.group_size;
        if (mode != 2) { col_start = T.bucket_col_start[b]; col_len = T.bucket_col_len[b]; }
        const long long bit_base = T.bucket_bit_base[b];
        const uint32_t* const startbit = T.thread_startbit + b * ((long long)k + 1);
        const uint32_t bits_k = startbit[k];
        const uint32_t my_start = startbit[t < k ? t : k];
        int32_t gid[kGids];
#pragma unroll
        for (int i = 0; i < kGids; ++i) gid[i] = tid + i * kThreads < NCTX ? T.bucket_table[b * NCTX + tid + i * kThreads] : -1;
        const long long nrows = row_e - row_a;
        const long long total = nrows * col_len;
        const long long wb = bit_base >> 6;
        const uint32_t k_eff = total < (long long)k ? (uint32_t)(total > 0 ? total : 1) : k;
        const bool ok = nrows > 0 && col_len > 0 && row_a >= 0 && row_a + nrows <= T.num_rows &&
                        (mode == 2 || (col_start >= 0 && col_start + col_len <= T.m)) && bit_base >= 0 && wb < T.bitstream_words &&
                        t_begin < k_eff;
        if (ok) {    // (uniform)
            // ---- where the bits lie
            const uint32_t bit_lo = (uint32_t)(bit_base & 63);
            const uint8_t* bytes = reinterpret_cast<const uint8_t*>(T.bitstream) + 8 * wb;
            const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(bytes) & 15u);   // 0 or 8
            long long valid = 8 * (T.bitstream_words - wb) + mis;
            const long long bits = (long long)(k_eff == k ? bits_k : startbit[k_eff]) + 8 * mis + bit_lo;
            if (valid > 0x7FFFFFF0LL) valid = 0x7FFFFFF0LL;
            // (the bucket's own bits must lie inside the bitstream; look-ahead past its end is never copied)
            bool fast = (mis == 0u || wb > 0) && valid >= 16 && ((bits + 7) >> 3) <= valid && nrows <= kRows &&
                        T.n * T.m < 0xFFFFFFFFLL && total < 0x7FFFFFFFLL;
            Item it;
            it.bo.base = bytes - mis;
            it.bo.last_ofs = (uint32_t)((valid - 16) & ~15LL);
            it.bo.tail_ofs = (valid & 8) ? it.bo.last_ofs + 16u : 0xFFFFFFFFu;
            it.bo.bit_delta = 8 * mis + bit_lo;
            const uint32_t pos = my_start + it.bo.bit_delta;
            const bool mine = decoding && t < k_eff;
            if (fast) {
                // first chunks of the rings: four neighbouring lanes fetch the 64 bytes of one sub-stream
                const uint32_t rings = smem_u32(sm.ring) + (uint32_t)(tid & ~31) * 64u;
                const uint32_t live = __ballot_sync(0xFFFFFFFFu, mine);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t owner = j * 8 + (lane >> 2);
                    const uint32_t p = __shfl_sync(0xFFFFFFFFu, pos, owner);
                    if ((live >> owner) & 1u) fetch_chunk(rings + owner * 64u, it.bo, ((p >> 7) + (lane & 3u)) << 4);
                }
            }
            // ---- rows, tables
            int bad = 0;
            uint32_t low = (uint32_t)col_len | k_eff | (uint32_t)reinterpret_cast<uintptr_t>(T.ctx_bytes);   // low bits of offsets
            if (fast) {
                for (int i = tid; i < (int)nrows; i += kAll) {
                    const long long row = T.row_indices[row_a + i];
                    const long long c0 = (mode == 2) ? (long long)T.group_col_start[row_a + i] : col_start;
                    const bool good = row >= 0 && row < T.n && c0 >= 0 && c0 + col_len <= T.m;
                    const uint32_t base = good ? (uint32_t)(row * T.m + c0) : 0u;
                    sm.rowbase[i] = base;
                    bad |= !good;
                    low |= base;
                }
            }
            int differs = ti != staged_ti;
#pragma unroll
            for (int i = 0; i < kGids; ++i) {
                const int c = tid + i * kThreads;
                if (decoding && c < NCTX) {
                    if (gid[i] >= T.num_tables) gid[i] = -1;
                    if (differs || sm.gid[c] != gid[i]) { differs = 1; sm.gid[c] = gid[i]; }
                }
            }
            if (__syncthreads_or(bad)) fast = false;
            const bool eights = !__syncthreads_or((int)(low & 7u));
            const bool restage = __syncthreads_or(differs) != 0;
            if (restage && decoding) stage<L>(sm, T);
            staged_ti = ti;
            cp_async_commit();
            cp_async_wait<0>();
            __syncthreads();
            if (restage) esc = __syncthreads_or(decoding && any_esc<L>(sm) ? 1 : 0) != 0;
            // ---- decode
            it.ctx = T.ctx_bytes; it.out = T.out;
            it.t = t; it.total = (uint32_t)total; it.k_eff = k_eff; it.col_len = (uint32_t)col_len; it.nrows = (uint32_t)nrows;
            it.item_steps = it.steps(t_begin);
            bool one_by_one = !fast;
            if (fast) {
                if (!decoding) {
                    if (eights) bring_ctx<true>(sm, it, t_begin);
                    else bring_ctx<false>(sm, it, t_begin);
                } else if (esc) {
                    run<L, true>(sm, it, pos);
                } else {
                    one_by_one = run<L, false>(sm, it, pos);
                }
            }
            if (one_by_one && mine) {
                const long long units = 2 * (T.bitstream_words - wb);
                const uint32_t lim = (uint32_t)((units > 0x7FFFFFFELL ? 0x7FFFFFFELL : units) - 1);
                run_general<L>(sm, T, reinterpret_cast<const uint32_t*>(T.bitstream) + 2 * wb, lim, my_start + bit_lo, t, k_eff, col_len,
                               col_start, row_a, total);
            }
        } else if (ti != staged_ti) {
            staged_ti = -1;          // the descriptor in shared memory is not the one the tables belong to
        }
        // (taken when the item's last context bytes are on their way, not at its start: what a CTA holds waits for it)
        if (!ONE && tid == kThreads)
            sm.next_item = args.total_items > (int)gridDim.x ? (int)(atomicAdd(&ws[0], 1u) + gridDim.x) : args.total_items;
        __syncthreads();             // tables, rings, rows and the next item's number
        item = sm.next_item;
        __syncthreads();
    }
    // the last CTA out re-zeroes the queue so that the next launch on this stream can reuse the workspace
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ws[1], 1u) == gridDim.x - 1) {
            ws[0] = 0u;
            ws[1] = 0u;
            __threadfence();
        }
    }
}

template <int L, bool ORDERED, bool ONE>
static int launch_as(const BatchArgs& a, int grid, unsigned int* ws, cudaStream_t st) {
    static bool attr_set[64] = {false};  // per instantiation and device
    int dev = 0;
    MPS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        MPS_CUDA_TRY(cudaFuncSetAttribute(narrow_decode_kernel<L, ORDERED, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    narrow_decode_kernel<L, ORDERED, ONE><<<grid, kAll, sizeof(Smem), st>>>(a, ws);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

template <int L>
static int launch(const BatchArgs& a, unsigned int* ws, cudaStream_t st) {
    int grid = 2 * sm_count();
    if (a.total_items < grid) grid = a.total_items;
    if (grid <= 0) return MPS_OK;
    if (a.total_items <= grid && a.order == nullptr) return launch_as<L, false, true>(a, grid, ws, st);
    if constexpr (L == 11) {
        if (orders_itself(a, grid, kSpan)) return launch_as<L, true, false>(a, grid, ws, st);
    }
    return launch_as<L, false, false>(a, grid, ws, st);
}

}  // namespace narrow
}  // namespace mps
