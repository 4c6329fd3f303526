// Layout and emission of the bucketed bitstream (kernel/build_huffman.cu:811-918 in the reference, which looks
// every element up in two hash maps, twice, on one thread).
//
//   codes    looks up the code of every element once, stores it in bucket order (16 bits an element for
//            tables of up to 2^11 entries) and counts the bits of every sub-stream
//   starts   start bit of every sub-stream in its bucket, then the 64-bit aligned start of every bucket
//   emit     reads the codes back, assembles the bits and writes the bitstream
//
// A unit of work is a bucket's range of neighbouring sub-streams, cut so that a unit has some tens of
// thousands of elements.  Neighbouring sub-streams are neighbouring elements, so a step of a unit is one
// contiguous read, and neighbouring sub-streams are one contiguous run of bits, so a unit assembles its
// bits in shared memory and writes them out coalesced; only its first and last word may be shared with a
// neighbour.  The threads of a CTA form teams, a thread holding V neighbouring sub-streams; every team
// takes a stretch of the steps, and where its bits start in each sub-stream is the sum of what the teams
// before it counted, which the first pass leaves behind.
//
// How an element's code is found: a context of a quantised weight sees a few dozen neighbouring BF16
// patterns of one sign, or two such runs, one of either sign, so each (context, sign) gets a map indexed
// by (magnitude pattern - the smallest one), all in shared memory: two loads per element.  A bucket whose
// maps do not fit, or whose tables are not one run of table ids, and buckets too small to pay for the maps,
// are searched in the sorted item lists in global memory.
#pragma once

#include "mps_common.cuh"

namespace mps {

struct RectGeom {
    const uint16_t* sym;              // [n*m] BF16 bit patterns
    const uint8_t* ctx;               // [n*m]
    const int32_t* bucket_table;      // [B, nctx]
    const int32_t* col_start;         // [B]
    const int32_t* col_len;           // [B]
    const int32_t* row_ofs;           // [B+1]
    const int32_t* rows;              // row lists
    const int32_t* group_col;         // ragged buckets: column start of every listed group, else nullptr
    long long B, m;
    int k, nctx, group_size;          // group_size: elements per group (ragged buckets)
    uint32_t ctx_mask;
};

struct CodeBook {
    const unsigned long long* items;
    const int* ctx_ofs;
    const uint32_t* enc;
    const uint32_t* esc;
    const uint16_t* escsym;
};

// (code, length) of one element, ESC expansion included: returns total bits, code(s) via out params
__device__ __forceinline__ int element_code(const CodeBook& cb, int gid, uint32_t sym, uint32_t& code, int& len,
                                            bool& raw) {
    const int a = cb.ctx_ofs[gid], b = cb.ctx_ofs[gid + 1];
    int lo = a, hi = b - 1, j = -1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const uint32_t v = (uint32_t)(cb.items[mid] & 0xFFFF);
        if (v == sym) { j = mid; break; }
        if (v < sym) lo = mid + 1; else hi = mid - 1;
    }
    raw = false;
    if (j < 0) return -1;
    uint32_t lc = cb.enc[j];
    if (lc == 0) {                       // not in the codebook: ESC code, then the raw 16 bits ...
        lc = cb.esc[gid];
        if (lc == 0) return -1;
        raw = (sym != cb.escsym[gid]);   // ... unless the symbol equals the synthetic ESC symbol, which the
    }                                    // reference's encoder map resolves to the bare ESC code
    code = lc & 0xFFFF;
    len = (int)(lc >> 16);
    return len + (raw ? 16 : 0);
}

namespace lay {

constexpr int kThreads = 512;
constexpr int kMaxV = 4;
constexpr int kNotFours = 5;   // error flag: buckets whose columns do not come in V (layout starts over with V = 1)

// A stored code: length and code in one word; 0: the context's ESC code; kNone: no code.
template <typename E> struct Packed;
template <> struct Packed<uint16_t> {      // tables of up to 2^11 entries
    static constexpr uint32_t kNone = 0xFFFFu;
    static __device__ __forceinline__ uint32_t pack(uint32_t lc) { return ((lc >> 16) << 11) | (lc & 0x7FFu); }
    static __device__ __forceinline__ uint32_t len(uint32_t e) { return e >> 11; }
    static __device__ __forceinline__ uint32_t code(uint32_t e) { return e & 0x7FFu; }
};
template <> struct Packed<uint32_t> {
    static constexpr uint32_t kNone = 0xFFFFFFFFu;
    static __device__ __forceinline__ uint32_t pack(uint32_t lc) { return lc; }
    static __device__ __forceinline__ uint32_t len(uint32_t e) { return e >> 16; }
    static __device__ __forceinline__ uint32_t code(uint32_t e) { return e & 0xFFFFu; }
};

struct Args {
    RectGeom g;
    CodeBook cb;
    long long G, numel;
    const unsigned long long* ebase;   // [B+1] first element of every bucket, in bucket order
    void* codes;                       // uint16 or uint32 [numel], in bucket order
    uint32_t* bits;                    // [B*k] bits of every sub-stream
    uint32_t* part;                    // [units][kThreads * kMaxV] bits in front of every team's stretch; null: one team
    uint32_t unit;                     // elements a unit should have
    uint32_t map_cap;                  // entries of the code maps in shared memory; 0: search, do not stage
    uint32_t buf_words;                // 32-bit words of the emit buffer
    const uint32_t* startbit;          // [B, k+1]
    const long long* bit_base;         // [B+1]
    unsigned long long* stream;
    int* err;
};

struct Unit {          // a bucket's range of sub-streams
    uint32_t row_a, col_len, col_start, k_eff, total;
    uint32_t R;        // sub-streams per unit, a multiple of V; the last unit of a bucket may have fewer
    uint32_t T, teams; // threads per team, teams
    uint32_t splits;
    unsigned long long ebase, part;   // first code of the bucket, first unit
};

// false: an empty bucket, buckets of more elements than the tensor has, or widths that V does not divide
__device__ __forceinline__ bool bucket_units(const Args& A, long long b, int V, Unit& u) {
    const RectGeom& g = A.g;
    const unsigned long long e0 = A.ebase[b], e1 = A.ebase[b + 1];
    if (e1 <= e0 || A.ebase[g.B] > (unsigned long long)A.numel) return false;
    u.row_a = (uint32_t)g.row_ofs[b];
    u.col_len = (uint32_t)(g.group_col ? g.group_size : g.col_len[b]);
    u.col_start = g.group_col ? 0u : (uint32_t)g.col_start[b];
    u.total = (uint32_t)(e1 - e0);
    u.k_eff = u.total < (uint32_t)g.k ? u.total : (uint32_t)g.k;
    if ((u.col_len | u.k_eff | (uint32_t)e0) & (uint32_t)(V - 1)) { atomicExch(A.err, kNotFours); return false; }
    const uint32_t splits = (u.total + A.unit - 1) / A.unit;
    u.R = ((u.k_eff + splits - 1) / splits + V - 1) / V * V;
    if (u.R > blockDim.x * (uint32_t)V) u.R = blockDim.x * (uint32_t)V;
    u.splits = (u.k_eff + u.R - 1) / u.R;
    u.T = u.R / V;
    u.teams = A.part ? blockDim.x / u.T : 1u;
    u.ebase = e0;
    u.part = (unsigned long long)b * (1u + (uint32_t)g.k / (blockDim.x * (uint32_t)V)) + e0 / A.unit;
    return true;
}

// row and column of the elements t + s * k_eff, one step after the other
struct Walk {
    uint32_t rr, cc, dr, dc, col_len;
    __device__ __forceinline__ Walk(const Unit& u, uint32_t e) {
        col_len = u.col_len;
        rr = e / col_len; cc = e - rr * col_len;
        dr = u.k_eff / col_len; dc = u.k_eff - dr * col_len;
    }
    __device__ __forceinline__ void step() {
        rr += dr; cc += dc;
        if (cc >= col_len) { cc -= col_len; ++rr; }
    }
};

__device__ __forceinline__ long long element_at(const RectGeom& g, const Unit& u, uint32_t rr, uint32_t cc) {
    return (long long)g.rows[u.row_a + rr] * g.m + (g.group_col ? (uint32_t)g.group_col[u.row_a + rr] : u.col_start) + cc;
}

// The code maps of a bucket in shared memory.
struct Maps {
    uint2 at[512];           // by context and sign: first entry of the map, smallest magnitude pattern | entries << 16
    int32_t gid[256];
    uint32_t lo[512], hi[512];
    uint32_t red[4];         // smallest table id, tables, first item, end of the items
    uint32_t warp[kThreads / 32];
};

// Fills the maps of bucket b; false: they do not fit or its tables are not one run of ids.  Called by the whole CTA of
// kThreads threads.
template <typename E>
__device__ bool stage_maps(const Args& A, long long b, Maps& M, E* map) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nctx = A.g.nctx;
    if (tid == 0) { M.red[0] = 0xFFFFFFFFu; M.red[1] = 0; M.red[2] = 0xFFFFFFFFu; M.red[3] = 0; }
    M.lo[tid] = 1; M.hi[tid] = 0;
    __syncthreads();
    int32_t gid = -1;
    if (tid < 256) {
        if (tid < nctx) {
            gid = A.g.bucket_table[b * nctx + tid];
            if (gid >= A.G) gid = -1;
        }
        M.gid[tid] = gid;
        if (gid >= 0) {
            atomicMin(&M.red[0], (uint32_t)gid);
            atomicAdd(&M.red[1], 1u);
            atomicMin(&M.red[2], (uint32_t)A.cb.ctx_ofs[gid]);
            atomicMax(&M.red[3], (uint32_t)A.cb.ctx_ofs[gid + 1]);
        }
    }
    __syncthreads();
    const uint32_t i0 = M.red[2], i1 = M.red[3];
    // one run of ids, each of its own context
    const bool odd = gid >= 0 && ((uint32_t)gid - M.red[0] >= M.red[1] || ((uint32_t)(A.cb.items[A.cb.ctx_ofs[gid]] >> 16) & 0xFFu) != (uint32_t)tid);
    if (__syncthreads_or(odd) || M.red[1] == 0) return false;
    // items are in (context, symbol) order: the first and last of every (context, sign) bound its map, and where a context
    // has symbols of either sign a search tells where the second begins
    if (gid >= 0) {
        uint32_t i = (uint32_t)A.cb.ctx_ofs[gid];
        const uint32_t e = (uint32_t)A.cb.ctx_ofs[gid + 1];
        const uint32_t first = (uint32_t)A.cb.items[i] & 0xFFFFu, last = (uint32_t)A.cb.items[e - 1] & 0xFFFFu;
        if (!((first ^ last) & 0x8000u)) {
            M.lo[2 * tid + (first >> 15)] = first & 0x7FFFu;
            M.hi[2 * tid + (first >> 15)] = last & 0x7FFFu;
        } else {
            uint32_t z = e - 1;      // items[i] is positive, items[z] negative
            while (z - i > 1) {
                const uint32_t mid = (i + z) >> 1;
                if ((uint32_t)A.cb.items[mid] & 0x8000u) z = mid; else i = mid;
            }
            M.lo[2 * tid] = first;
            M.hi[2 * tid] = (uint32_t)A.cb.items[i] & 0x7FFFu;
            M.lo[2 * tid + 1] = (uint32_t)A.cb.items[z] & 0x7FFFu;
            M.hi[2 * tid + 1] = last & 0x7FFFu;
        }
    }
    __syncthreads();
    const uint32_t span = M.hi[tid] >= M.lo[tid] ? M.hi[tid] - M.lo[tid] + 1u : 0u;
    uint32_t incl = span;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) M.warp[w] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) { if (i < w) before += M.warp[i]; total += M.warp[i]; }
    if (total > A.map_cap) return false;
    M.at[tid] = make_uint2(before + incl - span, (span ? M.lo[tid] : 0u) | (span << 16));
    for (uint32_t i = tid; i < total; i += kThreads) map[i] = (E)Packed<E>::kNone;
    __syncthreads();
#pragma unroll 4
    for (uint32_t i = i0 + tid; i < i1; i += kThreads) {
        const uint32_t v = (uint32_t)A.cb.items[i], h = (v >> 15) & 0x1FFu;
        map[M.at[h].x + (v & 0x7FFFu) - (M.at[h].y & 0xFFFFu)] = (E)Packed<E>::pack(A.cb.enc[i]);
    }
    __syncthreads();
    return true;
}

constexpr int kRowsKept = 1024;   // rows / groups of a bucket whose element offsets a CTA keeps in shared memory

// Pass 1.  Bound: two dependent lookups in shared memory and some thirty instructions per element, at half the warp slots.
// 14336 x 4096 FP8: 130 us; 205 with a search for every element's row in global memory, a branch per element and maps whose
// bounds came from a walk over all items.
template <typename E, int V, int NT>
__global__ void __launch_bounds__(NT) codes_kernel(const __grid_constant__ Args A) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_part[NT * V];
    __shared__ int32_t s_gid[256];
    __shared__ uint32_t s_row[V == 4 ? kRowsKept : 1];   // (fewer than 2^31 elements)
    const RectGeom& g = A.g;
    const long long b = blockIdx.x;
    Unit u;
    if (!bucket_units(A, b, V, u)) {
        if (blockIdx.y == 0)
            for (int t = threadIdx.x; t < g.k; t += NT) A.bits[b * g.k + t] = 0;
        return;
    }
    if (blockIdx.y >= u.splits) return;
    const uint32_t tid = threadIdx.x;
    bool mapped = false;
    const int32_t* gids = s_gid;
    Maps& M = *reinterpret_cast<Maps*>(s_raw);
    E* const map = reinterpret_cast<E*>(s_raw + sizeof(Maps));
    if constexpr (NT == kThreads) {
        if (A.map_cap) { mapped = stage_maps<E>(A, b, M, map); gids = M.gid; }
    }
    if (!A.map_cap) {
        for (int c = tid; c < g.nctx; c += NT) {
            const int32_t gid = g.bucket_table[b * g.nctx + c];
            s_gid[c] = gid >= A.G ? -1 : gid;
        }
        __syncthreads();
    }
    const uint32_t nrows = u.total / u.col_len;
    const bool rows_kept = V == 4 && nrows <= (uint32_t)kRowsKept;
    if (rows_kept) {
        for (uint32_t r = tid; r < nrows; r += NT) s_row[r] = (uint32_t)element_at(g, u, r, 0u);
        __syncthreads();
    }
    E* const codes = reinterpret_cast<E*>(A.codes) + u.ebase;
    // an element that the maps do not settle: its stored code, and its bits
    auto search = [&](uint32_t c, uint32_t sym, uint32_t& bits) -> uint32_t {
        uint32_t code = 0; int len = 0; bool raw = false;
        const int32_t gid = gids[c];
        const int nb = gid >= 0 ? element_code(A.cb, gid, sym, code, len, raw) : -1;
        if (nb < 0) { atomicExch(A.err, 3); bits = 0; return Packed<E>::kNone; }
        bits = (uint32_t)nb;
        // the ESC code proper is told from the ESC'd symbol's by emit, which looks at the symbol again
        return (raw || A.cb.esc[gid] == (((uint32_t)len << 16) | code)) ? 0u : Packed<E>::pack(((uint32_t)len << 16) | code);
    };
    for (uint32_t sp = blockIdx.y; sp < u.splits; sp += gridDim.y) {
        const uint32_t team = tid / u.T, lt = tid - team * u.T;
        const uint32_t t = sp * u.R + lt * V;
        const bool active = team < u.teams && t < u.k_eff;
        uint32_t acc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = 0;
        if (active) {
            const uint32_t steps = (u.total - t - 1) / u.k_eff + 1;   // V sub-streams side by side have the same number
            const uint32_t all = (u.total + u.k_eff - 1) / u.k_eff, per = (all + u.teams - 1) / u.teams;
            uint32_t s = team * per;
            const uint32_t s1 = (s + per < steps) ? s + per : steps;
            Walk at(u, t + s * u.k_eff);
            constexpr int UN = 4;
            for (; s < s1; s += UN) {
                uint32_t c[UN], sy[UN][(V + 1) / 2];
#pragma unroll
                for (int q = 0; q < UN; ++q) {
                    if (s + q < s1) {
                        const long long i = rows_kept ? (long long)(s_row[at.rr] + at.cc) : element_at(g, u, at.rr, at.cc);
                        if constexpr (V == 4) {
                            if ((i & 3) == 0) {
                                c[q] = *reinterpret_cast<const uint32_t*>(g.ctx + i);
                                const uint2 x = *reinterpret_cast<const uint2*>(g.sym + i);
                                sy[q][0] = x.x; sy[q][1] = x.y;
                            } else {   // a caller's group that starts between four-element boundaries
                                c[q] = g.ctx[i] | (g.ctx[i + 1] << 8) | (g.ctx[i + 2] << 16) | ((uint32_t)g.ctx[i + 3] << 24);
                                sy[q][0] = g.sym[i] | ((uint32_t)g.sym[i + 1] << 16);
                                sy[q][1] = g.sym[i + 2] | ((uint32_t)g.sym[i + 3] << 16);
                            }
                        } else { c[q] = g.ctx[i]; sy[q][0] = g.sym[i]; }
                        at.step();
                    }
                }
#pragma unroll
                for (int q = 0; q < UN; ++q) {
                    if (s + q < s1) {
                        uint32_t e[V];
                        bool settled = mapped;
                        if (mapped) {
#pragma unroll
                            for (int v = 0; v < V; ++v) {
                                const uint32_t cx = (c[q] >> (8 * v)) & g.ctx_mask;
                                const uint32_t sym = (sy[q][v >> 1] >> (16 * (v & 1))) & 0xFFFFu;
                                const uint2 at_h = M.at[(cx << 1) | (sym >> 15)];
                                const uint32_t d = (sym & 0x7FFFu) - (at_h.y & 0xFFFFu);
                                // (a symbol that the analysis did not see under this context is left to the search, which says so)
                                e[v] = Packed<E>::kNone;
                                if (d < (at_h.y >> 16)) e[v] = (uint32_t)map[at_h.x + d];
                                settled = settled && e[v] - 1u < Packed<E>::kNone - 1u;
                            }
                        }
                        if (settled) {
#pragma unroll
                            for (int v = 0; v < V; ++v) acc[v] += Packed<E>::len(e[v]);
                        } else {
#pragma unroll
                            for (int v = 0; v < V; ++v) {
                                if (mapped && e[v] - 1u < Packed<E>::kNone - 1u) { acc[v] += Packed<E>::len(e[v]); continue; }
                                uint32_t nb;
                                e[v] = search((c[q] >> (8 * v)) & g.ctx_mask, (sy[q][v >> 1] >> (16 * (v & 1))) & 0xFFFFu, nb);
                                acc[v] += nb;
                            }
                        }
                        E* dst = codes + (t + (s + q) * u.k_eff);
                        if constexpr (V == 4 && sizeof(E) == 2)
                            *reinterpret_cast<uint2*>(dst) = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
                        else if constexpr (V == 4)
                            *reinterpret_cast<uint4*>(dst) = make_uint4(e[0], e[1], e[2], e[3]);
                        else *dst = (E)e[0];
                    }
                }
            }
        }
        // bits in front of every team's stretch, and of every sub-stream as a whole
        const uint32_t here = u.k_eff - sp * u.R < u.R ? u.k_eff - sp * u.R : u.R;
        if (u.teams == 1) {
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (active) A.bits[b * g.k + t + v] = acc[v];
        } else {
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (team < u.teams) s_part[team * u.R + lt * V + v] = acc[v];
            __syncthreads();
            uint32_t* part = A.part + (u.part + sp) * (uint32_t)(kThreads * kMaxV);
            for (uint32_t i = tid; i < here; i += NT) {
                uint32_t sum = 0;
                for (uint32_t q = 0; q < u.teams; ++q) {
                    const uint32_t x = s_part[q * u.R + i];
                    part[q * u.R + i] = sum;
                    sum += x;
                }
                A.bits[b * g.k + sp * u.R + i] = sum;
            }
            __syncthreads();
        }
    }
    // sub-streams that a bucket of few elements does not have
    if (blockIdx.y == 0)
        for (uint32_t t = u.k_eff + tid; t < (uint32_t)g.k; t += NT) A.bits[b * g.k + t] = 0;
}

// Pass 3.  A thread appends its codes to a 64-bit register per sub-stream and ORs whole 32-bit words into
// the unit's buffer (units of the stream in bit order); a unit whose bits do not fit the buffer ORs them
// into the bitstream itself.  GRP codes of at most 32 bits together are put side by side first and appended at once: what
// an append costs, 64-bit shifts and the question whether a word is full, which some lane of a warp always answers with
// yes, is then paid per group.  14336 x 4096 FP8: 77 us, 191 with an append per code.  (Four codes of up to 8 bits, two of up
// to 15.)
template <typename E, int V, int NT, int GRP>
__global__ void __launch_bounds__(NT, 1024 / NT) emit_kernel(const __grid_constant__ Args A) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    uint32_t* const buf = reinterpret_cast<uint32_t*>(s_raw);
    const RectGeom& g = A.g;
    const long long b = blockIdx.x;
    Unit u;
    if (!bucket_units(A, b, V, u) || blockIdx.y >= u.splits) return;
    const uint32_t tid = threadIdx.x;
    const E* const codes = reinterpret_cast<const E*>(A.codes) + u.ebase;
    const uint32_t* const startbit = A.startbit + b * ((long long)g.k + 1);
    const unsigned long long base = (unsigned long long)A.bit_base[b];
    for (uint32_t sp = blockIdx.y; sp < u.splits; sp += gridDim.y) {
        const uint32_t t_a = sp * u.R, t_b = t_a + u.R < u.k_eff ? t_a + u.R : u.k_eff;
        const unsigned long long w0 = (base + startbit[t_a]) >> 6, w1 = (base + startbit[t_b] + 63) >> 6;
        const uint32_t words = (uint32_t)(w1 - w0) * 2u;
        const bool local = (unsigned long long)(w1 - w0) * 2u <= A.buf_words;
        if (local)
            for (uint32_t i = tid; i < words; i += NT) buf[i] = 0;
        __syncthreads();
        const uint32_t team = tid / u.T, lt = tid - team * u.T;
        const uint32_t t = t_a + lt * V;
        if (team < u.teams && t < u.k_eff) {
            const uint32_t steps = (u.total - t - 1) / u.k_eff + 1;
            const uint32_t all = (u.total + u.k_eff - 1) / u.k_eff, per = (all + u.teams - 1) / u.teams;
            uint32_t s = team * per;
            const uint32_t s1 = (s + per < steps) ? s + per : steps;
            const uint32_t* part = (u.teams > 1) ? A.part + (u.part + sp) * (uint32_t)(kThreads * kMaxV) + team * u.R + lt * V : nullptr;
            unsigned long long acc[V];
            uint32_t fill[V], at[V];   // bits held, next 32-bit word from w0 on
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const unsigned long long pos = base + startbit[t + v] + (part ? part[v] : 0u) - (w0 << 6);
                at[v] = (uint32_t)(pos >> 5);
                fill[v] = (uint32_t)pos & 31u;
                acc[v] = 0;
            }
            auto put = [&](uint32_t at_v, uint32_t word) {
                if (local) atomicOr(&buf[at_v], word);
                else atomicOr(reinterpret_cast<uint32_t*>(A.stream + w0) + (at_v ^ 1u), word);   // high half of a word first
            };
            auto append = [&](int v, uint32_t val, uint32_t nb) {     // fill < 32, nb <= 32
                acc[v] = (acc[v] << nb) | val;
                fill[v] += nb;
                if (fill[v] >= 32u) {
                    fill[v] -= 32u;
                    put(at[v]++, (uint32_t)(acc[v] >> fill[v]));
                }
            };
            auto append_one = [&](int v, uint32_t x, uint32_t step) {
                uint32_t val = Packed<E>::code(x), nb = Packed<E>::len(x);
                if (x == 0u) {   // the context's ESC code, then the 16 raw bits of the symbol
                    const uint32_t e = t + v + step * u.k_eff, rr = e / u.col_len;
                    const long long i = element_at(g, u, rr, e - rr * u.col_len);
                    const int32_t gid = g.bucket_table[b * g.nctx + (g.ctx[i] & g.ctx_mask)];
                    const uint32_t lc = gid >= 0 ? A.cb.esc[gid] : 0u, sym = g.sym[i];
                    val = lc & 0xFFFFu; nb = lc >> 16;
                    if (lc && sym != A.cb.escsym[gid]) { val = (val << 16) | sym; nb += 16; }
                } else if (x == Packed<E>::kNone) nb = val = 0;
                append(v, val, nb);
            };
            constexpr int UN = 4;
            static_assert(UN % GRP == 0, "a block of steps holds whole groups");
            for (; s < s1; s += UN) {
                uint32_t x[UN][V];
#pragma unroll
                for (int q = 0; q < UN; ++q) {
                    const E* src = codes + (t + (s + q) * u.k_eff);
                    if constexpr (V == 4 && sizeof(E) == 2) {
                        uint2 y = make_uint2(0u, 0u);
                        if (s + q < s1) y = *reinterpret_cast<const uint2*>(src);
                        x[q][0] = y.x & 0xFFFFu; x[q][1] = y.x >> 16; x[q][2] = y.y & 0xFFFFu; x[q][3] = y.y >> 16;
                    } else if constexpr (V == 4) {
                        uint4 y = make_uint4(0u, 0u, 0u, 0u);
                        if (s + q < s1) y = *reinterpret_cast<const uint4*>(src);
                        x[q][0] = y.x; x[q][1] = y.y; x[q][2] = y.z; x[q][3] = y.w;
                    } else x[q][0] = s + q < s1 ? (uint32_t)*src : 0u;
                }
#pragma unroll
                for (int q = 0; q < UN; q += GRP) {
#pragma unroll
                    for (int v = 0; v < V; ++v) {
                        uint32_t val = 0, nb = 0;
                        bool plain = true;      // (steps past the end read as 0, which is not)
#pragma unroll
                        for (int i = 0; i < GRP; ++i) {
                            const uint32_t n = Packed<E>::len(x[q + i][v]);
                            val = (val << (n & 31u)) | Packed<E>::code(x[q + i][v]);   // (n > 31: not plain)
                            nb += n;
                            plain = plain && x[q + i][v] - 1u < Packed<E>::kNone - 1u;
                        }
                        if (plain) append(v, val, nb);
                        else
#pragma unroll
                            for (int i = 0; i < GRP; ++i)
                                if (s + q + i < s1) append_one(v, x[q + i][v], s + q + i);
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (fill[v]) {
                    const uint32_t rest = (uint32_t)(acc[v] << (32u - fill[v]));
                    if (rest) put(at[v], rest);
                }
        }
        __syncthreads();
        if (local) {
            unsigned long long* const out = A.stream + w0;
            for (uint32_t i = tid; i < words / 2; i += NT) {
                const unsigned long long v = ((unsigned long long)buf[2 * i] << 32) | buf[2 * i + 1];
                if (i == 0 || i + 1 == words / 2) { if (v) atomicOr(&out[i], v); }   // shared with the neighbours
                else out[i] = v;
            }
        }
        __syncthreads();
    }
}

// Running sums over the buckets by one CTA of 1024 threads: f(b) is the value of bucket b, put(b, sum of those before it).
template <typename F, typename P>
__device__ __forceinline__ unsigned long long scan_buckets(long long B, F&& f, P&& put) {
    constexpr int PER = 4;
    __shared__ unsigned long long s_warp[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned long long carry = 0;
    for (long long b0 = 0; b0 < B; b0 += 1024 * PER) {
        unsigned long long v[PER], mine = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const long long b = b0 + tid * PER + i;
            v[i] = b < B ? f(b) : 0ull;
            mine += v[i];
        }
        unsigned long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) s_warp[w] = incl;
        __syncthreads();
        if (w == 0) {
            unsigned long long x = s_warp[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            s_warp[lane] = x;
        }
        __syncthreads();
        unsigned long long sum = carry + incl - mine + (w ? s_warp[w - 1] : 0ull);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const long long b = b0 + tid * PER + i;
            if (b < B) put(b, sum);
            sum += v[i];
        }
        carry += s_warp[31];
        __syncthreads();
    }
    return carry;
}

// first element of every bucket in bucket order, [B]: all elements; sets the error flag when there are more than the tensor has
__global__ void __launch_bounds__(1024) element_bases_kernel(RectGeom g, long long numel, unsigned long long* __restrict__ ebase, int* __restrict__ err) {
    const unsigned long long all = scan_buckets(g.B,
        [&](long long b) {
            const long long rows = (long long)g.row_ofs[b + 1] - g.row_ofs[b], cols = g.group_col ? g.group_size : g.col_len[b];
            return rows > 0 && cols > 0 ? (unsigned long long)(rows * cols) : 0ull;
        },
        [&](long long b, unsigned long long sum) { ebase[b] = sum; });
    if (threadIdx.x == 0) {
        ebase[g.B] = all;
        if (all > (unsigned long long)numel) atomicExch(err, 4);
    }
}

// start bit of every sub-stream relative to its bucket (build_huffman.cu:869-879), and the bucket's bits; a warp per bucket
__global__ void __launch_bounds__(256) starts_kernel(const uint32_t* __restrict__ bits, long long B, int k, uint32_t* __restrict__ startbit,
                                                     unsigned long long* __restrict__ bucket_bits) {
    const int lane = threadIdx.x & 31;
    for (long long b = blockIdx.x * 8LL + (threadIdx.x >> 5); b < B; b += gridDim.x * 8LL) {
        uint32_t* st = startbit + b * ((long long)k + 1);
        unsigned long long rel = 0;
        if (lane == 0) st[0] = 0;
        for (int t0 = 0; t0 < k; t0 += 128) {   // (sub-streams without elements have no bits: their start repeats the last one)
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = (t0 + 32 * i + lane < k) ? bits[b * k + t0 + 32 * i + lane] : 0u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t incl = v[i];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += x;
                }
                const int t = t0 + 32 * i + lane;
                if (t < k) st[t + 1] = (uint32_t)(rel + incl);
                rel += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
        }
        if (lane == 0) bucket_bits[b] = rel;
    }
}

struct Totals { long long bits; int err, codebook_err; };

// 64-bit aligned start of every bucket, [B] = end of the stream (build_huffman.cu:811-817, 918); what the host asks for, side by side
__global__ void __launch_bounds__(1024) bit_bases_kernel(const unsigned long long* __restrict__ bucket_bits, long long B, const int* __restrict__ err,
                                                         long long* __restrict__ bit_base, Totals* __restrict__ totals) {
    const unsigned long long all = scan_buckets(B, [&](long long b) { return (bucket_bits[b] + 63ull) & ~63ull; },
                                                [&](long long b, unsigned long long sum) { bit_base[b] = (long long)sum; });
    if (threadIdx.x == 0) {
        const unsigned long long last = B > 0 ? bucket_bits[B - 1] : 0ull;
        const long long end = (long long)(all - (((last + 63ull) & ~63ull) - last));
        bit_base[B] = end;
        totals->bits = end;
        totals->err = err[0];
        totals->codebook_err = err[1];
    }
}

// Host side -----------------------------------------------------------------------------------------------

struct Shape { bool small, wide, short_codes; int v;   // short_codes: four fit 32 bits
               uint32_t unit, map_cap, buf_words; unsigned splits; };

// Sizes of the launches.  Buckets of fewer than kSmallBucket elements on average (one per group of an INT4 weight) are searched
// by small CTAs, a bucket each: filling maps of some 5 K entries costs as much as looking up that many elements.  Whole builds,
// us, searched | mapped, 4096 x 4096 INT4 by scale, by elements per bucket: 255: 2029 | 7781, 1010: 1552 | 2830, 3851: 1486 |
// 1585, 7228: 1479 | 1377, 36551: 3406 | 1292; 1024 x 4096: 3418: 914 | 918, 5737: 964 | 902.  (FP8 buckets, whose maps are
// smaller, meet earlier: 2048 x 128, 1846 elements 810 | 793; 2048 x 512, 9118: 739 | 549.)
// Otherwise a unit has up to 64 K elements (7-bit tables: 32 KB of code) or 32 K, fewer when that leaves SMs idle.
constexpr long long kSmallBucket = 4096;
inline Shape shape_of(long long numel, long long B, long long largest, int k, int L, bool vec, int sms) {
    Shape s;
    s.small = numel / (B > 0 ? B : 1) < kSmallBucket;
    s.wide = L > 11;
    s.short_codes = L <= 8;
    s.v = (vec && !s.small) ? 4 : 1;
    const long long most = L <= 7 ? 65536 : 32768;
    long long unit = numel / (4LL * sms);
    unit = unit < 8192 ? 8192 : (unit > most ? most : unit);
    s.unit = (uint32_t)unit;
    s.map_cap = s.small ? 0u : (L <= 7 ? 28672u : (s.wide ? 22528u : 45056u));
    s.buf_words = s.small ? 1024u : (L <= 7 ? 14336u : 14336u);
    if (largest > numel) largest = numel;
    long long splits = (largest + unit - 1) / unit, by_k = (k + 127) / 128;   // (by_k: a CTA takes at least 128 sub-streams)
    if (splits < by_k) splits = by_k;
    s.splits = (unsigned)(splits < 1 ? 1 : (splits > 1024 ? 1024 : splits));
    return s;
}

template <typename E, int V, int NT>
static int launch_codes_as(const Args& a, const Shape& s, cudaStream_t st) {
    const size_t smem = a.map_cap ? sizeof(Maps) + (size_t)a.map_cap * sizeof(E) : 0;
    if (smem) MPS_CUDA_TRY(cudaFuncSetAttribute(codes_kernel<E, V, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    codes_kernel<E, V, NT><<<dim3((unsigned)a.g.B, s.splits), NT, smem, st>>>(a);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}
template <typename E, int V, int NT, int GRP>
static int launch_emit_as(const Args& a, const Shape& s, cudaStream_t st) {
    const size_t smem = (size_t)a.buf_words * 4;
    MPS_CUDA_TRY(cudaFuncSetAttribute(emit_kernel<E, V, NT, GRP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    emit_kernel<E, V, NT, GRP><<<dim3((unsigned)a.g.B, s.splits), NT, smem, st>>>(a);
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}
static int launch_codes(const Args& a, const Shape& s, cudaStream_t st) {
    if (s.small) return s.wide ? launch_codes_as<uint32_t, 1, 128>(a, s, st) : launch_codes_as<uint16_t, 1, 128>(a, s, st);
    if (s.v == 4) return s.wide ? launch_codes_as<uint32_t, 4, kThreads>(a, s, st) : launch_codes_as<uint16_t, 4, kThreads>(a, s, st);
    return s.wide ? launch_codes_as<uint32_t, 1, kThreads>(a, s, st) : launch_codes_as<uint16_t, 1, kThreads>(a, s, st);
}
static int launch_emit(const Args& a, const Shape& s, cudaStream_t st) {
    if (s.small) return s.wide ? launch_emit_as<uint32_t, 1, 128, 2>(a, s, st) : launch_emit_as<uint16_t, 1, 128, 2>(a, s, st);
    if (s.wide) return s.v == 4 ? launch_emit_as<uint32_t, 4, kThreads, 2>(a, s, st) : launch_emit_as<uint32_t, 1, kThreads, 2>(a, s, st);
    if (s.short_codes) return s.v == 4 ? launch_emit_as<uint16_t, 4, kThreads, 4>(a, s, st) : launch_emit_as<uint16_t, 1, kThreads, 4>(a, s, st);
    return s.v == 4 ? launch_emit_as<uint16_t, 4, kThreads, 2>(a, s, st) : launch_emit_as<uint16_t, 1, kThreads, 2>(a, s, st);
}

}  // namespace lay
}  // namespace mps
