// Codebook of every (scale, context): which symbols get a code, length-limited code lengths
// (package-merge, kernel/build_huffman.cu:46-118 in the reference), canonical codes in item order
// (:171-203), the 2^L-entry lookup table with its packed lengths (:205-239), and the code of every
// histogram item for the encoder.
//
// A group of threads -- a warp, two, or a CTA for contexts with many symbols -- owns one context and keeps
// everything in shared memory:
//   * items come in symbol order and are sorted by count, stably, a byte at a time (up to 32 items, and lists with an ESC
//     item in them, by a bitonic network over both);
//   * a level of package-merge is the merge of two sorted lists, the leaves and the sums of neighbouring
//     pairs of the level before: every thread finds where its share of the output begins on the merge
//     path (one binary search along a diagonal) and merges a few elements from there.  All that the
//     lengths need of a level is how many leaves lie among its first `take` items, so a level leaves one
//     bit per item behind, counted with popcounts on the way back down;
//   * a leaf is then as long as the number of levels that took it, and because those are prefixes of the
//     leaf list, the items of one length are one run of the sorted list: codes and table slots follow
//     from the run boundaries alone, and the table is written slot by slot, coalesced.
//
// Bound by shared-memory latency (dependent binary-search and merge steps), which some thirty resident
// warps per SM overlap.  The 6539 contexts of a 4096 x 4096 INT4 weight (some 300 symbols of up to 11 bits
// each): 0.21 ms, against 0.46 with the network for all, a branch per merged element and a search over the lengths per slot,
// and 190 ms with one thread per context and its arrays in global memory; the 23 K
// contexts of a 14336 x 4096 FP8 weight (some 26 symbols of up to 7 bits): 59 us, against 308 us and 200 us of
// device-wide sorts of the items before it.
#pragma once

#include "mps_common.cuh"

namespace mps {

enum { V_FP8 = 0, V_AWQ_BUCKET = 1, V_AWQ_BYSCALE = 2, V_AWQ_SHARED = 3 };

namespace cbk {

constexpr int kMaxL = 15;
constexpr int kWarpItems7 = 128;    // symbols a warp handles: all of a 7-bit table's
constexpr int kWarpItems = 512;     // symbols of a wider one that a small group handles
constexpr int kWarps = 4;           // warps (contexts in flight) of a CTA of the warp kernel
constexpr int kGroupThreads = 64;  // threads of a context of up to kWarpItems symbols of a wider table
constexpr int kCtaThreads = 256;
constexpr int kCtaItems = 2048;     // symbols a CTA handles in shared memory: all of an 11-bit table's

struct Args {
    const unsigned long long* items;   // scale << 32 | ctx << 16 | symbol, ascending
    const int* counts;
    const int* ctx_ofs;                // [G+1]
    int G, L, variant;
    int wide;                          // sums of L x the elements may pass 2^32 - 2: look before using 32-bit sums
    const int* row_of;                 // table row of every context (shared-table layout), else null: its number
    uint16_t* out_syms;
    uint8_t* out_lens;
    int pairs;                         // two slots can be stored at once: symbols lie on a multiple of 4 bytes, byte lengths on one of 2
    uint32_t* enc;                     // [N] len << 16 | code of each item, 0: not coded
    uint32_t* esc;                     // [G] len << 16 | code of the ESC code, 0: none
    uint16_t* escsym;
    int* err;
    int* big;                          // [G] contexts left to the CTA kernel
    unsigned int* big_count;
    unsigned int* queue;
};

template <int NT>
__device__ __forceinline__ void group_barrier() {
    if constexpr (NT == 32) __syncwarp(); else __syncthreads();
}

// run boundaries and first codes of a context's code lengths, in shared memory
struct Lengths {
    int q[kMaxL + 2];          // items of at least l bits: indices 0 .. q[l]-1 (ascending weights)
    uint32_t first[kMaxL + 2]; // first canonical code of l bits
    uint32_t cnt[kMaxL + 2];   // codes of l bits
    int ok;
};

// keys: count << 32 | symbol << 16 | position of the item in its context
__device__ __forceinline__ uint32_t key_weight(unsigned long long k) { return (uint32_t)(k >> 32); }
__device__ __forceinline__ uint32_t key_sym(unsigned long long k) { return (uint32_t)(k >> 16) & 0xFFFFu; }
__device__ __forceinline__ uint32_t key_pos(unsigned long long k) { return (uint32_t)k & 0xFFFFu; }

template <int NT>
__device__ void sort_keys(unsigned long long* keys, int n, int r) {
    if (NT == 32 && n <= 32) {
        unsigned long long v = r < n ? keys[r] : ~0ull;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1) {
                const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, v, j);
                const bool keep_low = ((r & k) == 0) == ((r & j) == 0);
                v = (keep_low == (o < v)) ? o : v;
            }
        if (r < n) keys[r] = v;
        __syncwarp();
        return;
    }
    int P = 64;
    while (P < n) P <<= 1;
    for (int i = n + r; i < P; i += NT) keys[i] = ~0ull;
    group_barrier<NT>();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int h = r; h < P / 2; h += NT) {
                const int a = ((h & ~(j - 1)) << 1) | (h & (j - 1)), b = a + j;
                const unsigned long long x = keys[a], y = keys[b];
                if ((x > y) == ((a & k) == 0)) { keys[a] = y; keys[b] = x; }
            }
            group_barrier<NT>();
        }
}

// Items in ascending symbol order by count: a stable sort by the count alone is enough, eight bits of it at a time and
// only the bytes that differ -- one pass where no symbol occurs 256 times.  Every warp of the group takes a stretch of the
// items and has its own 256 counters.  `other`: room for n keys, `hist`: for 256 counters per warp.  (300 items: some 400
// instructions a pass for a warp, the bitonic network 5000.)
template <int NT>
__device__ void sort_by_count(unsigned long long* keys, unsigned long long* other, uint32_t* hist, int n, int r) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, w = NT == 32 ? 0 : r >> 5;
    const int per = ((n + NW - 1) / NW + 31) & ~31, begin = w * per, end = begin + per < n ? begin + per : n;
    uint32_t* const mine = hist + 256 * w;
    uint32_t differ = 0;
    const uint32_t first = key_weight(keys[0]);
    for (int i = lane; i < n; i += 32) differ |= key_weight(keys[i]) ^ first;    // (every warp for itself)
    differ = __reduce_or_sync(0xFFFFFFFFu, differ);
    unsigned long long *from = keys, *to = other;
    for (int sh = 0; sh < 32; sh += 8) {
        if (!((differ >> sh) & 255u)) continue;
        for (int i = lane; i < 256; i += 32) mine[i] = 0u;
        __syncwarp();
        for (int i = begin + lane; i < end; i += 32) atomicAdd(&mine[(key_weight(from[i]) >> sh) & 255u], 1u);
        group_barrier<NT>();
        // where every (digit, warp) begins: a warp for all digits, every 32nd to a lane
        if (w == 0) {
            uint32_t at[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) at[d] = 0u;
#pragma unroll 1
            for (int q = 0; q < NW; ++q)
#pragma unroll
                for (int d = 0; d < 8; ++d) at[d] += hist[256 * q + 32 * d + lane];
            uint32_t before = 0;
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                uint32_t incl = at[d];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += x;
                }
                const uint32_t all = __shfl_sync(0xFFFFFFFFu, incl, 31);
                at[d] = before + incl - at[d];
                before += all;
            }
#pragma unroll 1
            for (int q = 0; q < NW; ++q)
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                    const uint32_t c = hist[256 * q + 32 * d + lane];
                    hist[256 * q + 32 * d + lane] = at[d];
                    at[d] += c;
                }
        }
        group_barrier<NT>();
        for (int i0 = begin; i0 < end; i0 += 32) {
            const int i = i0 + lane;
            const unsigned long long k = i < end ? from[i] : 0ull;
            const uint32_t d = i < end ? (key_weight(k) >> sh) & 255u : 256u + (uint32_t)lane;
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, d);
            const uint32_t before = (uint32_t)__popc(same & ((1u << lane) - 1u));
            if (i < end) to[mine[d] + before] = k;
            __syncwarp();
            if (i < end && before == 0u) mine[d] += (uint32_t)__popc(same);
            __syncwarp();
        }
        group_barrier<NT>();
        unsigned long long* t = from; from = to; to = t;
    }
    if (from != keys) {
        for (int i = r; i < n; i += NT) keys[i] = from[i];
        group_barrier<NT>();
    }
}

// Package-merge over keys[0, n), n >= 2, ascending by weight; fills ls.q.  `words`: 32-bit words of item
// flags per level.  keys[n] is overwritten.  IN_SHARED: keys and cur lie in shared memory.
constexpr uint32_t kEnd = 0xFFFFFFFFu;      // (sums of 32 bits stay below)
template <int NT, bool IN_SHARED, typename W>
__device__ void package_merge(unsigned long long* keys, int n, int L, W* cur, W* nxt, uint32_t* bits, int words,
                              Lengths& ls, int r) {
    for (int i = r; i < n; i += NT) cur[i] = key_weight(keys[i]);
    for (int i = r; i < (L - 1) * words; i += NT) bits[i] = 0;
    if (r == 0) keys[n] = (unsigned long long)kEnd << 32;
    group_barrier<NT>();
    int have = n;   // items of the level before; never more than 2 n - 1, so nothing is ever cut off
    for (int p = 1; p < L; ++p) {
        const int npk = have >> 1, total = n + npk;
        const int per = ((total + NT - 1) / NT) | 1;      // (odd: the threads' shares begin in different banks)
        const int d0 = r * per < total ? r * per : total, d1 = d0 + per < total ? d0 + per : total;
        int lo = d0 > npk ? d0 - npk : 0, hi = d0 < n ? d0 : n;
        while (lo < hi) {   // leaves among the first d0 items: a leaf goes before a package of the same weight
            const int mid = (lo + hi) >> 1, j = d0 - 1 - mid;
            if ((W)key_weight(keys[mid]) <= cur[2 * j] + cur[2 * j + 1]) lo = mid + 1; else hi = mid;
        }
        int i = lo, j = d0 - lo;
        uint32_t* flags = bits + (p - 1) * words;
        uint32_t acc = 0;
        if constexpr (sizeof(W) == 4) {
            // Both lists end in a weight above all others (the caller's, and the one below), and what comes next is one
            // read of eight bytes from either: a key, whose upper half is its weight, or two neighbours to be added up.
            uint32_t leaf = key_weight(keys[i]), pkg = j < npk ? cur[2 * j] + cur[2 * j + 1] : kEnd;
            const uint32_t key0 = IN_SHARED ? (uint32_t)__cvta_generic_to_shared(keys) : 0u, cur0 = IN_SHARED ? (uint32_t)__cvta_generic_to_shared(cur) : 0u;
            for (int o = d0; o < d1; ++o) {
                const bool is_leaf = leaf <= pkg;
                nxt[o] = is_leaf ? leaf : pkg;
                acc |= (is_leaf ? 1u : 0u) << (o & 31);
                i += is_leaf ? 1 : 0;
                j += is_leaf ? 0 : 1;
                uint32_t x = kEnd, y = 0u;
                if (is_leaf || j < npk) {
                    if constexpr (IN_SHARED) {
                        const uint32_t at = is_leaf ? key0 + 8u * (uint32_t)i : cur0 + 8u * (uint32_t)j;
                        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x), "=r"(y) : "r"(at) : "memory");
                    } else {
                        const uint2 v = is_leaf ? reinterpret_cast<const uint2*>(keys)[i] : reinterpret_cast<const uint2*>(cur)[j];
                        x = v.x; y = v.y;
                    }
                }
                leaf = is_leaf ? y : leaf;
                pkg = is_leaf ? pkg : x + y;
                if (((o & 31) == 31 || o + 1 == d1) && acc) { atomicOr(&flags[o >> 5], acc); acc = 0; }
            }
        } else {
            W leaf = i < n ? (W)key_weight(keys[i]) : 0, pkg = j < npk ? cur[2 * j] + cur[2 * j + 1] : 0;
            for (int o = d0; o < d1; ++o) {
                if (i < n && (j >= npk || leaf <= pkg)) {
                    nxt[o] = leaf;
                    acc |= 1u << (o & 31);
                    if (++i < n) leaf = key_weight(keys[i]);
                } else {
                    nxt[o] = pkg;
                    if (++j < npk) pkg = cur[2 * j] + cur[2 * j + 1];
                }
                if (((o & 31) == 31 || o + 1 == d1) && acc) { atomicOr(&flags[o >> 5], acc); acc = 0; }
            }
        }
        group_barrier<NT>();
        W* t = cur; cur = nxt; nxt = t;
        have = total;
    }
    // leaves taken at every level, from the top; lane l of every warp keeps level l's number
    const int lane = threadIdx.x & 31;
    int take = 2 * (n - 1), mine = -1;
    const bool enough = have >= take;
    for (int lvl = L - 1; lvl >= 0; --lvl) {
        int c = take;                            // the lowest level holds leaves only
        if (lvl > 0) {
            const uint32_t* flags = bits + (lvl - 1) * words;
            uint32_t part = 0;
            for (int w = lane; w * 32 < take; w += 32) {
                uint32_t f = flags[w];
                if (take - w * 32 < 32) f &= (1u << (take - w * 32)) - 1u;
                part += __popc(f);
            }
            c = (int)__reduce_add_sync(0xFFFFFFFFu, part);
        }
        if (lane == lvl) mine = c;
        take = 2 * (take - c);
    }
    // an item's length is the number of levels that took it: q[l] is the l-th largest of those numbers
    int rank = 0;
    for (int l = 0; l < L; ++l) {
        const int o = __shfl_sync(0xFFFFFFFFu, mine, l);
        if (o > mine || (o == mine && l < lane)) ++rank;
    }
    if (r < 32 && lane < L) ls.q[rank + 1] = mine;
    if (r == 0) { ls.q[L + 1] = 0; ls.ok = enough ? 1 : 0; }
    group_barrier<NT>();
}

__device__ __forceinline__ int length_of(const Lengths& ls, int i, int L) {
    int len = 0;
    for (int l = 1; l <= L; ++l) len += ls.q[l] > i ? 1 : 0;
    return len;
}

// Two neighbouring slots of a table whose rows start at `tsym` and `tlen`; a caller's arrays may lie anywhere.
__device__ __forceinline__ void put_slots(const Args& A, uint16_t* tsym, uint8_t* tlen, int s2, uint32_t sy0, uint32_t sy1, uint32_t nb0,
                                          uint32_t nb1) {
    if (A.pairs) {
        reinterpret_cast<uint32_t*>(tsym)[s2] = sy0 | (sy1 << 16);
    } else {
        tsym[2 * s2] = (uint16_t)sy0;
        tsym[2 * s2 + 1] = (uint16_t)sy1;
    }
    if (A.variant != V_AWQ_SHARED) {
        tlen[s2] = (uint8_t)((nb0 & 0xFu) | (nb1 << 4));
    } else if (A.pairs) {
        reinterpret_cast<uint16_t*>(tlen)[s2] = (uint16_t)(nb0 | (nb1 << 8));
    } else {
        tlen[2 * s2] = (uint8_t)nb0;
        tlen[2 * s2 + 1] = (uint8_t)nb1;
    }
}

template <int NT>
__device__ __forceinline__ uint32_t group_sum(uint32_t v, uint32_t* s_red) {
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    if constexpr (NT > 32) {
        __syncthreads();
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
        __syncthreads();
        v = 0;
        for (int i = 0; i < NT / 32; ++i) v += s_red[i];
    }
    return v;
}

// Canonical codes, the items' codes and the table of a context whose n items lie in `keys` in item order
// (esc_at: index of the ESC item, or -1).
template <int NT>
__device__ void write_codes(const Args& A, long long g, int a, const unsigned long long* keys, int n, int esc_at, uint32_t esc_sym,
                            Lengths& ls, int r) {
    const int L = A.L, TS = 1 << L;
    // the AWQ bucket formats force the ESC code to L bits (:1812-1816)
    const bool force = esc_at >= 0 && (A.variant == V_AWQ_BUCKET || A.variant == V_AWQ_BYSCALE);
    const int esc_len = esc_at >= 0 ? length_of(ls, esc_at, L) : 0;
    const bool moved = force && esc_len != L;
    if (r == 0) {
        uint32_t code = 0, before = 0;
        for (int l = 1; l <= L; ++l) {
            uint32_t c = (uint32_t)(ls.q[l] - ls.q[l + 1]);
            if (moved && l == esc_len) --c;
            if (moved && l == L) ++c;
            code = (code + before) << 1;
            ls.first[l] = code;
            ls.cnt[l] = before = c;
        }
    }
    group_barrier<NT>();
    for (int i = r; i < n; i += NT) {
        int len = length_of(ls, i, L);
        uint32_t rank = (uint32_t)(i - ls.q[len + 1]);
        if (moved) {
            if (i == esc_at) { len = L; rank = ls.cnt[L] - 1; }
            else if (len == esc_len && i > esc_at) --rank;
        }
        const uint32_t packed = ((uint32_t)len << 16) | (ls.first[len] + rank);
        if (i == esc_at) { A.esc[g] = packed; A.escsym[g] = (uint16_t)esc_sym; }
        else A.enc[a + key_pos(keys[i])] = packed;
    }
    // the table, two slots (one byte of packed lengths) per thread and step
    const bool bytes = A.variant == V_AWQ_SHARED;
    const long long row = A.row_of ? A.row_of[g] : g;
    uint16_t* tsym = A.out_syms + row * TS;
    uint8_t* tlen = A.out_lens + (bytes ? row * TS : row * (TS / 2));
    // slots ascend with the codes, and those with their lengths: end[l] is the first slot behind the codes of l bits
    uint32_t end[kMaxL];
    const uint32_t covered = ls.first[L] + ls.cnt[L];
#pragma unroll
    for (int l = 1; l < kMaxL; ++l) end[l] = l <= L ? (ls.first[l] + ls.cnt[l]) << (L - l) : 0xFFFFFFFFu;
    auto slot = [&](uint32_t s, uint32_t& sy, uint32_t& nb) -> int {
        int l = 1;
#pragma unroll
        for (int q = 1; q < kMaxL; ++q) l += s >= end[q] ? 1 : 0;
        sy = 0; nb = 0;       // a slot that no code covers
        if (s >= covered) return L;
        const uint32_t rank = (s >> (L - l)) - ls.first[l];
        int i = ls.q[l + 1] + (int)rank;
        if (moved) {
            if (l == L && rank == ls.cnt[L] - 1) i = esc_at;
            else if (l == esc_len && i >= esc_at) ++i;
        }
        sy = key_sym(keys[i]);
        nb = (uint32_t)l;
        if (A.variant == V_FP8 && i == esc_at) nb |= 8u;
        // every slot that shows the ESC symbol is marked (:1822-1829, :2410-2415)
        if (esc_at >= 0 && sy == esc_sym) {
            if (force) nb = 15u;
            else if (bytes) nb |= 0x80u;
        }
        return l;
    };
    for (int s2 = r; s2 < TS / 2; s2 += NT) {
        uint32_t sy[2], nb[2];
        if (slot(2u * s2, sy[0], nb[0]) < L) { sy[1] = sy[0]; nb[1] = nb[0]; }
        else slot(2u * s2 + 1u, sy[1], nb[1]);
        put_slots(A, tsym, tlen, s2, sy[0], sy[1], nb[0], nb[1]);
    }
}

// A context with one symbol: length 1, code 0, every slot (:464-472); with none: an empty table.
template <int NT>
__device__ void write_trivial(const Args& A, long long g, int a, int cnt, int r) {
    const int TS = 1 << A.L;
    const bool bytes = A.variant == V_AWQ_SHARED;
    const long long row = A.row_of ? A.row_of[g] : g;
    const uint32_t sy = cnt ? (uint32_t)(A.items[a] & 0xFFFFu) : 0u, nb = cnt ? 1u : 0u;
    uint16_t* tsym = A.out_syms + row * TS;
    uint8_t* tlen = A.out_lens + (bytes ? row * TS : row * (TS / 2));
    for (int s2 = r; s2 < TS / 2; s2 += NT) put_slots(A, tsym, tlen, s2, sy, sy, nb, nb);
    if (cnt && r == 0) A.enc[a] = 1u << 16;
}

template <int ITEMS>
struct WarpSpace {
    unsigned long long keys[ITEMS + 2];          // (one behind the last is written, and pairs of 16 bytes)
    alignas(16) uint32_t cur[2 * ITEMS], nxt[2 * ITEMS];
    uint32_t bits[(kMaxL - 1) * (2 * ITEMS / 32)];
    Lengths ls;
};

// One group of NT threads per context of at most ITEMS symbols that all get a code (kWarps warps to a CTA, or one larger group);
// the others are listed for the CTA kernel.
template <int ITEMS, int NT>
__global__ void __launch_bounds__(NT == 32 ? kWarps * 32 : NT) group_kernel(const __grid_constant__ Args A) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    constexpr int kGroups = NT == 32 ? kWarps : 1;
    const int r = threadIdx.x % NT, w = threadIdx.x / NT;
    WarpSpace<ITEMS>& S = reinterpret_cast<WarpSpace<ITEMS>*>(s_raw)[w];
    const int TS = 1 << A.L;
    for (long long g = (long long)blockIdx.x * kGroups + w; g < A.G; g += (long long)gridDim.x * kGroups) {
        const int a = A.ctx_ofs[g], cnt = A.ctx_ofs[g + 1] - a;
        if (r == 0) { A.esc[g] = 0; A.escsym[g] = 0; }
        if (cnt <= 1) { write_trivial<NT>(A, g, a, cnt, r); continue; }
        bool mine = cnt <= ITEMS && cnt <= TS;
        if (mine && A.wide) {       // (every warp for itself)
            unsigned long long part = 0;
            for (int i = r & 31; i < cnt; i += 32) part += (uint32_t)A.counts[a + i];
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
            mine = part * (unsigned)A.L < kEnd;
        }
        if (!mine) {
            if (r == 0) A.big[atomicAdd(A.big_count, 1u)] = (int)g;
            continue;
        }
        group_barrier<NT>();
        for (int i = r; i < cnt; i += NT)
            S.keys[i] = ((unsigned long long)(uint32_t)A.counts[a + i] << 32) | ((A.items[a + i] & 0xFFFFull) << 16) | (uint32_t)i;
        group_barrier<NT>();
        static_assert(sizeof(S.nxt) >= NT / 32 * 256 * 4, "the warps' counters");
        if (NT == 32 && cnt <= 32) sort_keys<NT>(S.keys, cnt, r);
        else sort_by_count<NT>(S.keys, reinterpret_cast<unsigned long long*>(S.cur), S.nxt, cnt, r);
        package_merge<NT, true>(S.keys, cnt, A.L, S.cur, S.nxt, S.bits, (2 * cnt + 31) / 32, S.ls, r);
        if (!S.ls.ok) { if (r == 0) atomicExch(A.err, 2); continue; }
        write_codes<NT>(A, g, a, S.keys, cnt, -1, 0, S.ls, r);
        group_barrier<NT>();
    }
}

// What a CTA works in: shared memory for tables of up to kCtaItems entries and 32-bit sums, else global scratch.
template <typename W>
struct CtaSpace {
    unsigned long long* keys;   // [items]
    W *cur, *nxt;               // [2 * items] each
    uint32_t* bits;             // [(L - 1) * 2 * items / 32]
    static __host__ __device__ int items_of(int L) { return (1 << L) < 64 ? 64 : (1 << L); }   // the sort pads to 64
    static __host__ __device__ size_t bytes(int L) {
        const int items = items_of(L);
        return (size_t)(items + 2) * 8 + (size_t)items * 4 * sizeof(W) + (size_t)(L - 1) * ((size_t)items / 16 + 1) * 4 + 64;
    }
    __device__ void carve(unsigned char* p, int L) {
        const int items = items_of(L);
        keys = reinterpret_cast<unsigned long long*>(p);
        cur = reinterpret_cast<W*>(keys + items + 2);
        nxt = cur + 2 * items;
        bits = reinterpret_cast<uint32_t*>(nxt + 2 * items);
    }
};

// One CTA per listed context.  A context with more symbols than table slots keeps the 2^L - 1 most
// frequent ones (ties: smaller symbol first) and folds the rest into one ESC item (:479-535).
template <typename W, bool IN_SHARED>
__global__ void __launch_bounds__(kCtaThreads) cta_kernel(const __grid_constant__ Args A, unsigned char* __restrict__ scratch, size_t stride) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ Lengths ls;
    __shared__ uint32_t s_red[kCtaThreads / 32], s_hist[256], s_next, s_low, s_prefix, s_need;
    const int r = threadIdx.x, lane = r & 31, w = r >> 5;
    const int L = A.L, TS = 1 << L;
    CtaSpace<W> S;
    S.carve(IN_SHARED ? s_raw : scratch + (size_t)blockIdx.x * stride, L);

    // exclusive prefix of a flag over the CTA, and its total
    auto prefix = [&](bool f, uint32_t& total) -> uint32_t {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, f);
        __syncthreads();
        if (lane == 0) s_red[w] = __popc(m);
        __syncthreads();
        uint32_t before = 0;
        total = 0;
        for (int i = 0; i < kCtaThreads / 32; ++i) { if (i < w) before += s_red[i]; total += s_red[i]; }
        return before + __popc(m & ((1u << lane) - 1u));
    };

    for (;;) {
        if (r == 0) s_next = atomicAdd(A.queue, 1u);
        __syncthreads();
        const uint32_t turn = s_next;
        __syncthreads();
        if (turn >= *A.big_count) break;
        const long long g = A.big[turn];
        const int a = A.ctx_ofs[g], cnt = A.ctx_ofs[g + 1] - a;
        const bool use_esc = cnt > TS;
        const int keep = use_esc ? TS - 1 : cnt;
        int n = cnt, esc_at = -1;
        uint32_t esc_sym = 0;
        if (!use_esc) {
            for (int i = r; i < cnt; i += kCtaThreads)
                S.keys[i] = ((unsigned long long)(uint32_t)A.counts[a + i] << 32) | ((A.items[a + i] & 0xFFFFull) << 16) | (uint32_t)i;
        } else {
            // the keep-th largest count, eight bits at a time
            if (r == 0) { s_prefix = 0; s_need = (uint32_t)keep; s_low = 0x10000u; }
            for (int sh = 24; sh >= 0; sh -= 8) {
                for (int h = r; h < 256; h += kCtaThreads) s_hist[h] = 0;
                __syncthreads();
                const uint32_t want = s_prefix;
                for (int i = r; i < cnt; i += kCtaThreads) {
                    const uint32_t c = (uint32_t)A.counts[a + i];
                    if (sh == 24 || (c >> (sh + 8)) == want) atomicAdd(&s_hist[(c >> sh) & 255u], 1u);
                }
                __syncthreads();
                if (r == 0) {
                    uint32_t left = s_need;
                    int d = 255;
                    while (d > 0 && s_hist[d] < left) left -= s_hist[d--];
                    s_need = left;
                    s_prefix = (want << 8) | (uint32_t)d;
                }
                __syncthreads();
            }
            const uint32_t edge = s_prefix, of_edge = s_need;   // keep all above `edge` and the first `of_edge` at it
            uint32_t seen = 0, kept = 0;
            unsigned long long lost = 0;
            for (int i0 = 0; i0 < cnt; i0 += kCtaThreads) {      // items are in ascending symbol order
                const int i = i0 + r;
                const uint32_t c = i < cnt ? (uint32_t)A.counts[a + i] : 0u;
                const uint32_t sy = i < cnt ? (uint32_t)(A.items[a + i] & 0xFFFFull) : 0u;
                uint32_t all_edge, all_kept;
                const uint32_t at_edge = prefix(i < cnt && c == edge, all_edge);
                const bool keep_it = i < cnt && (c > edge || (c == edge && seen + at_edge < of_edge));
                const uint32_t at = kept + prefix(keep_it, all_kept);
                if (keep_it) S.keys[at] = ((unsigned long long)c << 32) | ((unsigned long long)sy << 16) | (uint32_t)i;
                else if (i < cnt) { lost += c; A.enc[a + i] = 0; }
                // smallest symbol not among the kept ones (by-scale: not in the context at all): the first
                // whose place in their ascending list is not its own value
                if (A.variant == V_AWQ_BYSCALE) { if (i < cnt && sy != (uint32_t)i) atomicMin(&s_low, (uint32_t)i); }
                else if (keep_it && sy != at) atomicMin(&s_low, at);
                seen += all_edge;
                kept += all_kept;
            }
            // 2^31 elements at most, so the sum's halves fit 32-bit reductions
            const uint32_t lost_lo = group_sum<kCtaThreads>((uint32_t)(lost & 0xFFFFu), s_red);
            const uint32_t lost_hi = group_sum<kCtaThreads>((uint32_t)(lost >> 16), s_red);
            lost = ((unsigned long long)lost_hi << 16) + lost_lo;
            __syncthreads();
            const uint32_t dense = A.variant == V_AWQ_BYSCALE ? (uint32_t)cnt : (uint32_t)keep;
            esc_sym = s_low < dense ? s_low : dense;
            if (esc_sym > 0xFFFFu) esc_sym = 0xFFFFu;
            int weight = (int)lost;                              // the reference accumulates in int
            if (A.variant == V_AWQ_SHARED) weight = lost > 2147483647ull ? 2147483647 : (int)lost;   // (:2345-2352)
            if ((A.variant == V_AWQ_BUCKET || A.variant == V_AWQ_SHARED) && weight <= 0) weight = 1;
            if (r == 0) S.keys[keep] = ((unsigned long long)(uint32_t)weight << 32) | ((unsigned long long)esc_sym << 16);
            n = keep + 1;
        }
        __syncthreads();
        const unsigned long long esc_key = use_esc ? S.keys[keep] : 0ull;
        __syncthreads();
        // (the ESC item stands last whatever its symbol: the network compares symbols too)
        if (!use_esc && 2 * CtaSpace<W>::items_of(L) * sizeof(W) >= kCtaThreads / 32 * 256 * sizeof(uint32_t))
            sort_by_count<kCtaThreads>(S.keys, reinterpret_cast<unsigned long long*>(S.cur), reinterpret_cast<uint32_t*>(S.nxt), n, r);
        else
            sort_keys<kCtaThreads>(S.keys, n, r);
        package_merge<kCtaThreads, IN_SHARED, W>(S.keys, n, L, S.cur, S.nxt, S.bits, (2 * n + 31) / 32, ls, r);
        if (!ls.ok) { if (r == 0) atomicExch(A.err, 2); __syncthreads(); continue; }
        if (use_esc && A.variant == V_AWQ_BYSCALE) {
            // The by-scale builder keeps its items in DESCENDING order of count (ascending symbol inside a
            // count) with the ESC item last and does not re-sort them (build_huffman.cu:1283-1301), while the
            // lengths it pairs them with by position are those of the ASCENDING weights.
            for (int i = r; i < n; i += kCtaThreads) {
                const unsigned long long k = S.keys[i];
                S.keys[i] = k == esc_key ? ~0ull : (k ^ 0xFFFFFFFF00000000ull);
            }
            __syncthreads();
            sort_keys<kCtaThreads>(S.keys, n, r);
            if (r == 0) S.keys[n - 1] = esc_key;
            __syncthreads();
            esc_at = n - 1;
        } else if (use_esc) {
            for (int i = r; i < n; i += kCtaThreads)
                if (S.keys[i] == esc_key) s_low = (uint32_t)i;
            __syncthreads();
            esc_at = (int)s_low;
        }
        write_codes<kCtaThreads>(A, g, a, S.keys, n, esc_at, esc_sym, ls, r);
        __syncthreads();
    }
}

// Scratch the CTA kernel needs in global memory (0: it works in shared memory), and its grid.
struct CtaShape { bool in_shared, wide; int grid; size_t stride; };
inline CtaShape cta_shape(int L, int wide, int sms, size_t scratch_bytes) {
    CtaShape c;
    c.wide = wide != 0;
    c.in_shared = !c.wide && (1 << L) <= kCtaItems;
    c.stride = c.wide ? CtaSpace<unsigned long long>::bytes(L) : CtaSpace<uint32_t>::bytes(L);
    c.stride = (c.stride + 255) / 256 * 256;
    c.grid = 4 * sms;
    if (!c.in_shared && (size_t)c.grid * c.stride > scratch_bytes) c.grid = (int)(scratch_bytes / c.stride);
    return c;
}

template <typename K>
static int allow_smem(K kernel, size_t bytes) {
    MPS_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return MPS_OK;
}

// All codebooks of a histogram.  `scratch`: at least one cta_shape().stride bytes when it is not in shared memory.
static int launch(const Args& A, const CtaShape& c, int sms, unsigned char* scratch, cudaStream_t st) {
    if (A.G <= 0) return MPS_OK;
    if (c.grid < 1) { set_error("codebook scratch too small for max_len=%d", A.L); return MPS_ERR_WORKSPACE; }
    const bool narrow = (1 << A.L) <= kWarpItems7;
    // What limits how many contexts an SM works on is their shared memory, 14 KB for 512 symbols: sixteen warps if each has its
    // own.  Two share one: a 4096 x 4096 INT4 weight's whole build 785 us, 834 with one, 802 with four (a CTA per larger context
    // of 128, 256 or 512 threads: 790, 785, 811).
    const int per_cta = narrow ? kWarps : 1;
    const size_t smem = narrow ? kWarps * sizeof(WarpSpace<kWarpItems7>) : sizeof(WarpSpace<kWarpItems>);
    int grid = (A.G + per_cta - 1) / per_cta;
    const int most = sms * (narrow ? 12 : 2048 / kGroupThreads);
    if (grid > most) grid = most;
    if (narrow) {
        if (int rc = allow_smem(group_kernel<kWarpItems7, 32>, smem)) return rc;
        group_kernel<kWarpItems7, 32><<<grid, kWarps * 32, smem, st>>>(A);
    } else {
        if (int rc = allow_smem(group_kernel<kWarpItems, kGroupThreads>, smem)) return rc;
        group_kernel<kWarpItems, kGroupThreads><<<grid, kGroupThreads, smem, st>>>(A);
    }
    const int ctas = c.grid < A.G ? c.grid : A.G;
    if (c.wide) cta_kernel<unsigned long long, false><<<ctas, kCtaThreads, 0, st>>>(A, scratch, c.stride);
    else if (!c.in_shared) cta_kernel<uint32_t, false><<<ctas, kCtaThreads, 0, st>>>(A, scratch, c.stride);
    else {
        if (int rc = allow_smem(cta_kernel<uint32_t, true>, c.stride)) return rc;
        cta_kernel<uint32_t, true><<<ctas, kCtaThreads, c.stride, st>>>(A, nullptr, 0);
    }
    MPS_CUDA_TRY(cudaGetLastError());
    return MPS_OK;
}

}  // namespace cbk
}  // namespace mps
