// query_impl.cuh -- the CTA-level query body shared by the plain query kernel
// (query.cu) and the persistent batch kernel (batch.cu).
//
// It replaces RTX_blocks' ray programs (src/rtx_kernels.cu:85-193 for
// values, 350-465 for indices). The reference fires up to three rays per
// query: one through the fully covered blocks lB+1..rB-1, one through the
// left partial block and one through the right partial block, and keeps the
// closest hit. Here the same decomposition is answered from arrays:
//   left partial block   -> suf[l]   (random HBM lookup)
//   right partial block  -> pre[r]   (random HBM lookup)
//   full blocks between  -> two sparse-table entries (L2-resident)
// and it is needed only for the few queries a cheaper test does not settle:
// every query first probes a small L2-resident table over all the units it
// touches (blocks lB..rB, or with the sub-block level the 32-element
// micro-blocks l/32..r/32), and when the leftmost best of that superset
// lies inside [l, r] it is the answer without any per-element lookup. A
// query inside one micro-block is settled by a scan of that 128-byte line,
// 8 lanes per query; without the sub-block level a query inside one block that
// the probe does not settle reads pre / suf at a block edge, or is scanned
// by the whole warp (__reduce_min_sync over the composites). All
// comparisons are unsigned minima of the composites of common.cuh; only the
// final answer is decoded.
//
// Differences from the reference kept on purpose: ties between rays are
// resolved leftmost (the reference compares rays with strict `<` in the
// order middle, left, right, src/rtx_kernels.cu:451-465), values are the
// exact bits of A[idx] (the reference returns payload + min, rtx.h:109,
// rtx_kernels.cu:179), and a miss cannot overwrite a minimum
// (src/rtx_kernels.cu:80-83).
#pragma once

#include "common.cuh"

namespace rmq {

// One built array: values A[off .. off + n) of the buffer A (loads never go
// past A[limit - 1]); structure arrays are array-relative.
struct V1View {
    const float *A;
    int64_t off;
    int64_t limit;
    uint32_t n;
    uint32_t bs;
    uint32_t nb;
    Div31 dv;
    const Entry *pre;
    const Entry *suf;
    const Entry *st;
    // sub-block level: 32-element micro-blocks (local index / 32), whatever
    // the block size; null when the index has none (same-block queries then
    // use the warp-cooperative scan)
    const Entry *mst;   // micro-block minima (micro-table level 0)
    const void *moff;   // levels 1..: offsets of each window's best micro-block
    uint32_t moff_bytes;
    uint32_t nmicro;
    const Entry *mpre;  // in-micro-block prefix / suffix minima
    const Entry *msuf;
    uint32_t kmode;     // KeyMode: element type and minimum / maximum
    uint32_t levels;    // sparse-table levels (st holds levels * nb entries)
    uint32_t mlevels;   // micro-table levels (moff holds mlevels - 1 rows of nmicro)
    // 2^mlevels - 1: a query whose end micro-blocks ml < mr have
    // mr - ml < micro_span is probed through the micro table (0: no micro level)
    uint32_t micro_span;
};

// Range-checked accesses (rmq_chk, common.cuh): element loads by absolute
// index into A, table entries by index into a table of `size` entries.
__device__ __forceinline__ uint32_t ld_elem(const V1View &v, int64_t g) {
    return rmq_chk(g >= 0 && g < v.limit) ? ld_u1(v.A + g) : 0u;
}
__device__ __forceinline__ uint4 ld_elem4(const V1View &v, int64_t g) {
    return rmq_chk(g >= 0 && g + 3 < v.limit) ? ld_u4(v.A + g) : make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ Entry ld_entry(const Entry *t, uint64_t i, uint64_t size) {
    return rmq_chk(i < size) ? t[i] : kEntryNone;
}

// The same, as a streaming load (evict-first in L1 and L2), for the random
// per-element sub-block entries: they are read once, and the micro table
// they would otherwise evict is read by every same-block query.
__device__ __forceinline__ Entry ld_entry_cs(const Entry *t, uint64_t i, uint64_t size) {
    return rmq_chk(i < size) ? __ldcs(reinterpret_cast<const unsigned long long *>(t) + i)
                             : kEntryNone;
}

// The small tables every query probes (the sparse table over block minima,
// the micro table) are read with an L2 evict-last policy (PTX createpolicy +
// ld.L2::cache_hint), so that the per-element lines and the query stream
// passing through L2 evict them last. No L2 carve-out is set aside, unlike a
// persisting access-policy window. The policy is made once per step.
__device__ __forceinline__ uint64_t l2_keep_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ Entry ld_entry_keep(const Entry *t, uint64_t i, uint64_t size,
                                               uint64_t pol) {
    if (!rmq_chk(i < size)) return kEntryNone;
    unsigned long long v;
    asm volatile("ld.global.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(t + i), "l"(pol));
    return v;
}

// Offset i of the micro table's levels 1.. (moff_bytes wide, the same for
// every query of an index, so the branch does not diverge).
__device__ __forceinline__ uint32_t ld_moff(const V1View &v, uint64_t i, uint64_t pol) {
    if (!rmq_chk(i < static_cast<uint64_t>(v.mlevels - 1u) * v.nmicro)) return 0u;
    uint32_t r;
    if (v.moff_bytes == 1u)
        asm volatile("ld.global.L2::cache_hint.u8 %0, [%1], %2;"
                     : "=r"(r) : "l"(static_cast<const uint8_t *>(v.moff) + i), "l"(pol));
    else if (v.moff_bytes == 2u)
        asm volatile("ld.global.L2::cache_hint.u16 %0, [%1], %2;"
                     : "=r"(r) : "l"(static_cast<const uint16_t *>(v.moff) + i), "l"(pol));
    else
        asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;"
                     : "=r"(r) : "l"(static_cast<const uint32_t *>(v.moff) + i), "l"(pol));
    return r;
}

// The aligned 8-byte word of the 1-byte micro-table offsets that holds
// offset i (the table starts 256-byte aligned; its tail is padded to 256
// bytes, so the word never passes the allocation).
__device__ __forceinline__ uint64_t ld_moff_word(const V1View &v, uint64_t i, uint64_t pol) {
    const uint64_t w = i >> 3;
    if (!rmq_chk(w < (static_cast<uint64_t>(v.mlevels - 1u) * v.nmicro + 7) / 8)) return 0u;
    uint64_t r;
    asm volatile("ld.global.L2::cache_hint.u64 %0, [%1], %2;"
                 : "=l"(r) : "l"(static_cast<const uint64_t *>(v.moff) + w), "l"(pol));
    return r;
}

struct QueryOut {
    const int2 *Q;        // queries of this array (local l, r)
    float *val;           // outputs aligned with Q, may be null
    int32_t *idx;         // may be null
    unsigned long long *invalid;
    int64_t span;         // entries of Q / val / idx from these pointers on
};

__device__ __forceinline__ void put_bits_idx(const QueryOut &o, int64_t i, uint32_t bits,
                                             uint32_t idx) {
    if (!rmq_chk(i >= 0 && i < o.span)) return;
    if (o.val) __stcs(reinterpret_cast<unsigned int *>(o.val) + i, bits);
    if (o.idx) __stcs(o.idx + i, static_cast<int32_t>(idx));
}

__device__ __forceinline__ void put_result(const QueryOut &o, int64_t i, Entry e, uint32_t mode) {
    put_bits_idx(o, i, o.val ? entry_bits(e, mode) : 0u, entry_idx(e));
}

__device__ __forceinline__ void put_invalid(const QueryOut &o, int64_t i) {
    if (!rmq_chk(i >= 0 && i < o.span)) return;
    if (o.val) __stcs(reinterpret_cast<unsigned int *>(o.val) + i, 0x7fc00000u);
    if (o.idx) __stcs(o.idx + i, -1);
    if (o.invalid) atomicAdd(o.invalid, 1ull);
}

// Leftmost minimum of local A[l..r] computed by the whole warp. All 32 lanes
// call it with the same (l, r); every lane gets the result. ALIGNED: the
// buffer base is 16-byte aligned, so 16-byte loads on absolute indices are.
template <bool ALIGNED>
__device__ __forceinline__ Entry warp_scan_range(const V1View &v, uint32_t l, uint32_t r,
                                                 int lane, uint32_t mode) {
    Entry best = kEntryNone;
    const int64_t al = v.off + l, ar = v.off + r;
    if (ALIGNED) {
        for (int64_t p = (al & ~int64_t(3)) + 4 * lane; p <= ar; p += 128) {
            uint32_t b[4];
            if (p + 3 < v.limit) {
                const uint4 f = ld_elem4(v, p);
                b[0] = f.x;
                b[1] = f.y;
                b[2] = f.z;
                b[3] = f.w;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    b[c] = (p + c <= ar) ? ld_elem(v, p + c) : 0u;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int64_t g = p + c;
                if (g >= al && g <= ar)
                    best = better(best, make_entry(b[c], static_cast<uint32_t>(g - v.off), mode));
            }
        }
    } else {
        for (int64_t g = al + lane; g <= ar; g += 32)
            best = better(best, make_entry(ld_elem(v, g), static_cast<uint32_t>(g - v.off), mode));
    }
    // 64-bit minimum across the warp: the key word first, then the low word
    // among the lanes that hold that key
    const uint32_t key = static_cast<uint32_t>(best >> 32);
    const uint32_t kmin = __reduce_min_sync(0xffffffffu, key);
    const uint32_t cand = (key == kmin) ? static_cast<uint32_t>(best) : 0xffffffffu;
    const uint32_t lo = __reduce_min_sync(0xffffffffu, cand);
    return (static_cast<uint64_t>(kmin) << 32) | lo;
}

// Answer queries [q0, q1) of one array with the whole CTA. The loop is
// uniform across the CTA (warp-cooperative scans need full warps).
// QPT queries per thread per iteration keep several independent lookups in
// flight per thread.
// Queries base + threadIdx.x + k * blockDim.x (k < QPT) of [.., q1), loaded
// ahead of use (the query stream may come from host memory over the host
// link, so a caller can issue the next step's loads before answering the
// current step).
template <int QPT>
__device__ __forceinline__ void load_queries(const QueryOut &o, int64_t base, int64_t q1,
                                             int2 (&qq)[QPT]) {
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const int64_t i = base + threadIdx.x + static_cast<int64_t>(k) * blockDim.x;
        qq[k] = make_int2(0, 0);
        if (i < q1 && rmq_chk(i < o.span)) qq[k] = __ldcs(o.Q + i);
    }
}

// ---- per-query work --------------------------------------------------------
//
// Every probe of a small table returns the leftmost best element of a set of
// whole units (blocks of the sparse table, micro-blocks of the micro table)
// that contains [l, r]. If that element's index lies in [l, r], it is the
// answer: it beats every element of the superset, and an equal element
// further left inside [l, r] would have been chosen instead. Otherwise the
// best lies outside on one side, say left of l in unit a; then the answer is
// better(S[l], best of units a+1..b) when the latter falls at or before r
// (S[l] covers [l, end of a]), and the three-part decomposition of the
// reference (left partial, units between, right partial) only when it does
// not. The per-element entries S / P, the random HBM lookups, are read only
// on those two fallbacks.

// Query counters of a measurement launch (rmq_query_stats); the normal
// kernels compile them out.
enum QStat : int {
    kStatFirst = 0,   // settled by the superset probe
    kStatSecond,      // settled by the second probe and one per-element entry
    kStatFull,        // three-part decomposition: two entries and a middle probe
    kStatMicroScan,   // inside one micro-block: its line of values is scanned
    kStatBlockEdge,   // one block, no sub-block level: pre / suf at a block edge
    kStatWarpScan,    // one block, no sub-block level: warp-cooperative scan
    kStatEntries,     // per-element entries read (pre, suf, mpre, msuf)
    kStatTable,       // small-table words read (sparse table, micro offsets and minima)
    kStatSectors,     // 32-byte sectors of A read by scans
    kStatInvalid,     // invalid queries
    kStatCount
};
struct QStats {
    uint32_t c[kStatCount];
};

// Leftmost best of blocks a..b (a <= b < nb) from the sparse table: two
// entries of level floor(log2(b - a + 1)), one when the window is exact.
template <bool STATS>
__device__ __forceinline__ Entry st_probe(const V1View &v, uint32_t a, uint32_t b, uint64_t pol,
                                          QStats &s) {
    const int lev = ilog2(b - a + 1u);
    const uint64_t row = static_cast<uint64_t>(lev) * v.nb;
    const uint64_t size = static_cast<uint64_t>(v.levels) * v.nb;
    const uint32_t c = b + 1u - (1u << lev);
    const Entry x = ld_entry_keep(v.st, row + a, size, pol);
    Entry y = x;
    if (c != a) y = ld_entry_keep(v.st, row + c, size, pol);
    if constexpr (STATS) s.c[kStatTable] += (c != a) ? 2u : 1u;
    return better(x, y);
}

// Leftmost best of micro-blocks a..b (a <= b, b - a + 1 < 2^mlevels): the
// offsets of the two windows' best micro-blocks, then their minima.
template <bool STATS>
__device__ __forceinline__ Entry micro_probe(const V1View &v, uint32_t a, uint32_t b, uint64_t pol,
                                             QStats &s) {
    const int lev = ilog2(b - a + 1u);
    uint32_t x = a, y = b + 1u - (1u << lev);
    if (lev > 0) {
        const uint64_t row = static_cast<uint64_t>(lev - 1) * v.nmicro;
        const bool two = y != x;
        const uint32_t ox = ld_moff(v, row + x, pol);
        const uint32_t oy = two ? ld_moff(v, row + y, pol) : ox;
        if constexpr (STATS) s.c[kStatTable] += two ? 2u : 1u;
        x += ox;
        y += oy;
    }
    const Entry ex = ld_entry_keep(v.mst, x, v.nmicro, pol);
    Entry ey = ex;
    if (y != x) ey = ld_entry_keep(v.mst, y, v.nmicro, pol);
    if constexpr (STATS) s.c[kStatTable] += (y != x) ? 2u : 1u;
    return better(ex, ey);
}

template <bool STATS>
__device__ __forceinline__ Entry unit_probe(const V1View &v, bool micro, uint32_t a, uint32_t b,
                                            uint64_t pol, QStats &s) {
    return micro ? micro_probe<STATS>(v, a, b, pol, s) : st_probe<STATS>(v, a, b, pol, s);
}

// S[l]: best of A[l .. end of l's unit]; P[r]: best of A[start of r's unit .. r].
// The micro-level entries are read with streaming loads (they are read once,
// and would otherwise push the micro table out of L2).
template <bool STATS>
__device__ __forceinline__ Entry left_entry(const V1View &v, bool micro, uint32_t l, QStats &s) {
    if constexpr (STATS) s.c[kStatEntries] += 1u;
    return micro ? ld_entry_cs(v.msuf, l, v.n) : ld_entry(v.suf, l, v.n);
}
template <bool STATS>
__device__ __forceinline__ Entry right_entry(const V1View &v, bool micro, uint32_t r, QStats &s) {
    if constexpr (STATS) s.c[kStatEntries] += 1u;
    return micro ? ld_entry_cs(v.mpre, r, v.n) : ld_entry(v.pre, r, v.n);
}

// 32-byte sectors of the local range A[a..b]
__device__ __forceinline__ uint32_t range_sectors(const V1View &v, uint32_t a, uint32_t b) {
    return static_cast<uint32_t>(((v.off + b) >> 3) - ((v.off + a) >> 3) + 1);
}

// ---- the queued form (query_kernel, batch_kernel's query phase) -------------
//
// Settling a query that its probe leaves open inside the same step would
// make a warp wait for the slowest lane's chain of dependent loads (entry,
// narrower probe, then maybe the rest). The queued form is specialised at
// compile time on the key mode and on whether the index has the sub-block
// level, and its main pass does only the superset probe: a query the probe
// settles is stored at once; one it leaves open, or that lies inside one
// micro-block, goes into a per-warp queue in shared memory, and whenever 32
// are waiting the warp settles them together (drain_misses).

// ---- lines of values, settled by the warp ---------------------------------
//
// A query inside one micro-block, and a miss of the light index, needs the
// best of part of one 32-element line. Scanned by the lane that owns the
// query, a load instruction touches up to 32 different 128-byte lines, one
// L1 tag lookup each, for up to 9 instructions, and a warp waits for its
// longest scan. Here 8 lanes take one request, 16 bytes each: a load
// instruction touches 4 lines and each line is looked up once. What bounds
// it is the random lines' DRAM traffic. Measured (2^26 queries, ms): ranges
// of 32 over n = 1e8 2.78 -> 1.81; light index, uniform 0.527 -> 0.346, short
// (lr=-3) 1.18 -> 1.09, ranges of 32 4.99 -> 3.2 (those took 40 KB of shared
// memory per CTA for the lines besides, and ran 3 CTAs per SM).

// The best of one lane's chunk b[0..3] among the elements whose bit of `nib`
// is set, in key mode MODE: its key, and its position | (-0.0 flag << 2).
// With no element set, or every set element at the largest key, the key is
// the largest one (the caller then takes the request's first element).
template <uint32_t MODE>
__device__ __forceinline__ void chunk_best(const uint32_t (&b)[4], uint32_t nib, uint32_t &key,
                                           uint32_t &info) {
    if constexpr (MODE == kFloatMin || MODE == kFloatMax) {
        // the IEEE minimum (maximum) skips NaN, which orders last; the first
        // value equal to it is the leftmost best and gives the key
        float x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            x[k] = __uint_as_float((nib >> k) & 1u ? b[k] : 0x7fc00000u);
        const float m = MODE == kFloatMin ? fminf(fminf(x[0], x[1]), fminf(x[2], x[3]))
                                          : fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
        const uint32_t p = x[0] == m ? 0u : x[1] == m ? 1u : x[2] == m ? 2u : 3u;
        const uint32_t wb = p == 0u ? b[0] : p == 1u ? b[1] : p == 2u ? b[2] : b[3];
        key = m == m ? key_of(wb, MODE) : 0xffffffffu;
        info = p | (negzero_of(wb, MODE) << 2);
    } else {
        key = 0xffffffffu;
        info = 0u;
#pragma unroll
        for (int k = 3; k >= 0; --k) {
            const uint32_t kk = (nib >> k) & 1u ? key_of(b[k], MODE) : 0xffffffffu;
            if (kk <= key) {
                key = kk;
                info = static_cast<uint32_t>(k);
            }
        }
    }
}

// One chunk of values: elements 4 sub .. 4 sub + 3 of the 32-element line
// `line` (array-relative), of which only those set in `nib` are read when the
// 16-byte load is not possible (values not 16-byte aligned, or the chunk
// passes the end of the buffer).
template <bool ALIGNED>
__device__ __forceinline__ void load_chunk(const V1View &v, uint32_t line, uint32_t sub,
                                           uint32_t nib, uint32_t (&b)[4]) {
    const int64_t g = v.off + static_cast<int64_t>(line) * 32 + 4 * sub;
#pragma unroll
    for (int k = 0; k < 4; ++k) b[k] = 0u;
    if (nib == 0u) return;
    if (ALIGNED && (v.off & 3) == 0 && g + 4 <= v.limit) {
        const uint4 f = ld_elem4(v, g);
        b[0] = f.x;
        b[1] = f.y;
        b[2] = f.z;
        b[3] = f.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((nib >> k) & 1u) b[k] = ld_elem(v, g + k);
    }
}

// Rounds of 4 requests whose loads are in flight together. Two: four cost 9
// to 16 more registers in the main pass they share a kernel with (uniform
// lengths, n = 1e8, q = 2^26: 0.309 ms with two, 0.341 with four) and settle
// misses no faster.
constexpr int kLineRounds = 2;

// Leftmost best of the elements of line `line` whose bits are set in `bits`,
// for every lane with bits != 0, kEntryNone for the others; the whole warp
// calls it.
template <bool ALIGNED, uint32_t MODE>
__device__ __forceinline__ Entry warp_lines(const V1View &v, uint32_t line, uint32_t bits) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, grp = lane >> 3;
    const uint32_t act = __ballot_sync(0xffffffffu, bits != 0u);
    Entry out = kEntryNone;
#pragma unroll 1
    for (uint32_t h = 0; h < 32u; h += 4u * kLineRounds) {
        if (((act >> h) & ((1u << (4 * kLineRounds)) - 1u)) == 0u) continue;  // warp-uniform
        uint32_t b[kLineRounds][4];
#pragma unroll
        for (int t = 0; t < kLineRounds; ++t) {
            const uint32_t ln = __shfl_sync(0xffffffffu, line, h + 4u * t + grp);
            const uint32_t m = __shfl_sync(0xffffffffu, bits, h + 4u * t + grp);
            load_chunk<ALIGNED>(v, ln, sub, (m >> (4u * sub)) & 15u, b[t]);
        }
#pragma unroll
        for (int t = 0; t < kLineRounds; ++t) {
            const uint32_t m = __shfl_sync(0xffffffffu, bits, h + 4u * t + grp);
            uint32_t gk, info;
            chunk_best<MODE>(b[t], (m >> (4u * sub)) & 15u, gk, info);
            const uint32_t key = gk;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) gk = min(gk, __shfl_xor_sync(0xffffffffu, gk, o, 8));
            const uint32_t own = (__ballot_sync(0xffffffffu, key == gk) >> (8u * grp)) & 0xffu;
            const uint32_t w = __ffs(own) - 1u;
            info = __shfl_sync(0xffffffffu, info, 8u * grp + w);
            // every set element at the largest key: the first of them
            const uint32_t pos = gk == 0xffffffffu ? __ffs(m) - 1u : 4u * w + (info & 3u);
            const uint32_t nz = gk == 0xffffffffu ? 0u : info >> 2;
            // to the lane that asked: h + 4 t + its group
            const uint32_t rk = __shfl_sync(0xffffffffu, gk, 8u * (lane & 3u));
            const uint32_t rl = __shfl_sync(0xffffffffu, (pos << 1) | nz, 8u * (lane & 3u));
            if (bits != 0u && (lane >> 2) == (h >> 2) + t)
                out = (static_cast<uint64_t>(rk) << 32) | ((line << 6) + rl);
        }
    }
    return out;
}

// Bits lo .. hi (inclusive, 0 <= lo <= hi <= 31)
__device__ __forceinline__ uint32_t bit_range(uint32_t lo, uint32_t hi) {
    return (0xffffffffu >> (31u - hi)) & (0xffffffffu << lo);
}

// With per-element entries, the part of a query in its end unit on the
// left, [l, end of l's unit] (micro-block, or block), and on the right,
// [start of r's unit, r]: one entry each.
template <bool STATS>
__device__ __forceinline__ Entry left_part(const V1View &v, bool micro, uint32_t l, QStats &s) {
    return left_entry<STATS>(v, micro, l, s);
}
template <bool STATS>
__device__ __forceinline__ Entry right_part(const V1View &v, bool micro, uint32_t r, QStats &s) {
    return right_entry<STATS>(v, micro, r, s);
}

// Light index: the query's part in its end unit on one side, [l, end of
// l's unit] (left) or [start of r's unit, r] (right): part of one line of
// values inside the end micro-block (its line and element bits), plus for a
// block unit the best of the block's whole micro-blocks on that side. The
// side is a value, not a branch, so that lanes settling left and right parts
// run the same code.
template <bool STATS>
__device__ __forceinline__ Entry light_rest(const V1View &v, bool micro, bool left, uint32_t a,
                                            uint32_t b, uint32_t l, uint32_t r, uint64_t pol,
                                            QStats &s, uint32_t &line, uint32_t &bits) {
    line = (left ? l : r) >> 5;
    // the left end's unit lies before the right end's, so its line is whole
    bits = left ? 0xffffffffu << (l & 31u) : 0xffffffffu >> (31u - (r & 31u));
    if constexpr (STATS) s.c[kStatSectors] += range_sectors(v, left ? l : (r & ~31u), left ? l | 31u : r);
    if (micro) return kEntryNone;
    // block a is full when a < b: its last micro-block ends inside the array
    const uint32_t ml = l >> 5, me = (((a + 1u) * v.bs) >> 5) - 1u;
    const uint32_t mr = r >> 5, ms = (b * v.bs) >> 5;
    const bool has = left ? ml < me : ms < mr;
    if (!has) return kEntryNone;
    return micro_probe<STATS>(v, left ? ml + 1u : ms, left ? me : mr - 1u, pol, s);
}

// Settles one query whose superset best lay outside [l, r] (or, without
// the sub-block level, inside one block at an edge) from the per-element
// entries: the query's part in the end unit on that side and a narrower
// probe, loaded together, then only if needed the other end's part and the
// middle units.
template <bool STATS>
__device__ __forceinline__ Entry finish_miss(const V1View &v, bool micro, bool left, uint32_t l,
                                             uint32_t r, uint64_t pol, QStats &s) {
    const uint32_t a = micro ? (l >> 5) : div31(l, v.dv);
    const uint32_t b = micro ? (r >> 5) : div31(r, v.dv);
    if (a == b) {
        // one block, without the sub-block level: the query touches an edge
        if constexpr (STATS) s.c[kStatBlockEdge] += 1u;
        const uint32_t bend = min(a * v.bs + v.bs, v.n) - 1u;
        return r == bend ? left_entry<STATS>(v, false, l, s) : right_entry<STATS>(v, false, r, s);
    }
    // the narrower probe first: its loads are in flight while the part's
    // entry is loaded
    const Entry e2 = left ? unit_probe<STATS>(v, micro, a + 1u, b, pol, s)
                          : unit_probe<STATS>(v, micro, a, b - 1u, pol, s);
    const Entry e1 = left ? left_part<STATS>(v, micro, l, s) : right_part<STATS>(v, micro, r, s);
    const uint32_t m2 = entry_idx(e2);
    if (left ? m2 <= r : m2 >= l) {
        if constexpr (STATS) s.c[kStatSecond] += 1u;
        return better(e1, e2);
    }
    if constexpr (STATS) s.c[kStatFull] += 1u;
    const Entry mid = (b - a >= 2u) ? unit_probe<STATS>(v, micro, a + 1u, b - 1u, pol, s)
                                    : kEntryNone;
    const Entry other = left ? right_part<STATS>(v, micro, r, s) : left_part<STATS>(v, micro, l, s);
    return better(better(e1, other), mid);
}

// One warp's queue: up to 31 waiting queries plus the 32 that each query
// slot of a step can add, 12 bytes each (what it takes from the L1 matters:
// the block table's upper levels live there). `id` numbers the queries of
// the CTA in the order it takes them: step * step size + place in the step.
template <int QPT>
struct MissQueue {
    static constexpr int kCap = 32 * (QPT + 1);
    uint32_t l[kCap];   // kMissLeft set: the probe's best lay left of l
    uint32_t r[kCap];
    uint32_t id[kCap];
};
constexpr uint32_t kMissLeft = 0x80000000u;  // above every index

// The queries a CTA takes: steps of `chunk` consecutive ones, `stride` apart.
struct StepMap {
    int64_t first;
    int64_t stride;
    __device__ __forceinline__ int64_t query(uint32_t id, uint32_t chunk) const {
        return first + static_cast<int64_t>(id / chunk) * stride + id % chunk;
    }
};

// Settles the last min(count, 32) queued queries, one per lane; the whole
// warp calls it (count is warp-uniform). Queries inside one micro-block, and
// the light index's misses, read lines of values, the warp together.
template <bool ALIGNED, bool MICRO, bool LIGHT, uint32_t MODE, bool STATS, int THREADS, int QPT>
__device__ __forceinline__ void drain_misses(const V1View &v, const QueryOut &o,
                                             const StepMap &map, MissQueue<QPT> &mq,
                                             uint32_t &count, uint64_t pol, QStats &s) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t take = count < 32u ? count : 32u;
    __syncwarp();
    const uint32_t e = count - take + lane;
    const bool act = lane < take;
    const uint32_t lq = act ? mq.l[e] : 0u, r = act ? mq.r[e] : 0u;
    const uint32_t l = lq & ~kMissLeft;
    const bool left = (lq & kMissLeft) != 0u;
    const bool micro = MICRO && (r >> 5) - (l >> 5) < v.micro_span;
    const bool scan = MICRO && act && (l >> 5) == (r >> 5);
    const bool miss = act && !scan;
    Entry res = kEntryNone;
    uint32_t line = l >> 5, bits = scan ? bit_range(l & 31u, r & 31u) : 0u;
    if constexpr (!LIGHT) {
        if (MICRO && __any_sync(0xffffffffu, scan)) res = warp_lines<ALIGNED, MODE>(v, line, bits);
        if (miss) res = finish_miss<STATS>(v, micro, left, l, r, pol, s);
    } else {
        const uint32_t a = micro ? (l >> 5) : div31(l, v.dv);
        const uint32_t b = micro ? (r >> 5) : div31(r, v.dv);
        Entry e2 = kEntryNone;
        if (miss) {
            e2 = unit_probe<STATS>(v, micro, left ? a + 1u : a, left ? b : b - 1u, pol, s);
            res = light_rest<STATS>(v, micro, left, a, b, l, r, pol, s, line, bits);
        }
        // one copy of the line scan's code: the second pass (the other end,
        // after the middle units) runs only for the rare query the narrower
        // probe does not settle
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            res = better(res, warp_lines<ALIGNED, MODE>(v, line, bits));
            if (pass == 1) break;
            bits = 0u;
            bool more = false;
            if (miss) {
                const uint32_t m2 = entry_idx(e2);
                more = left ? m2 > r : m2 < l;
                if constexpr (STATS) s.c[more ? kStatFull : kStatSecond] += 1u;
                if (!more) {
                    res = better(res, e2);
                } else {
                    if (b - a >= 2u)
                        res = better(res, unit_probe<STATS>(v, micro, a + 1u, b - 1u, pol, s));
                    res = better(res, light_rest<STATS>(v, micro, !left, a, b, l, r, pol, s, line, bits));
                }
            }
            if (!__any_sync(0xffffffffu, more)) break;
        }
    }
    if (act) put_result(o, map.query(mq.id[e], THREADS * QPT), res, MODE);
    __syncwarp();
    count -= take;
}

// The bits of an entry's element for key mode MODE, without branches
// (unkey for a mode known at compile time).
template <uint32_t MODE>
__device__ __forceinline__ uint32_t decode_bits(Entry e) {
    const uint32_t k = static_cast<uint32_t>(e >> 32);
    if constexpr (MODE == kIntMin) {
        return k ^ 0x80000000u;
    } else if constexpr (MODE == kIntMax) {
        return k ^ 0x7fffffffu;
    } else {
        const uint32_t nz = static_cast<uint32_t>(e) & 1u;
        // f = fkey(bits): bits | 2^31 for a positive value (2^31 for +-0,
        // negzero telling them apart), ~bits for a negative one
        const uint32_t f = (MODE == kFloatMax) ? ~k : k;
        const uint32_t b = (f & 0x80000000u) ? ((f & 0x7fffffffu) | (nz << 31)) : ~f;
        return k == 0xffffffffu ? 0x7fc00000u : b;  // NaN: the canonical quiet NaN
    }
}

// The superset probe of the queued form for a valid query not inside one
// micro-block: through the micro table when the query's micro-blocks fit
// it (`mic`), else through the block table (two entries, one straight
// sequence).
template <bool MICRO, bool STATS>
__device__ __forceinline__ Entry superset_probe(const V1View &v, uint32_t l, uint32_t r,
                                                uint64_t pol, QStats &s, bool &mic) {
    const uint32_t ml = l >> 5, mr = r >> 5;
    mic = MICRO && mr - ml < v.micro_span;
    const uint32_t a = mic ? ml : div31(l, v.dv);
    const uint32_t b = mic ? mr : div31(r, v.dv);
    const int lev = ilog2(b - a + 1u);
    uint32_t x = a, y = b + 1u - (1u << lev);
    if (MICRO && mic) {
        // lev >= 1: the query spans at least two micro-blocks. The two
        // windows overlap, so 1-byte offsets often share an aligned 8-byte
        // word (one load), and both windows often point at the same best
        // micro-block (one minimum load).
        const uint64_t row = static_cast<uint64_t>(lev - 1) * v.nmicro;
        if (v.moff_bytes == 1u && ((row + x) >> 3) == ((row + y) >> 3)) {
            const uint64_t w = ld_moff_word(v, row + x, pol);
            x += static_cast<uint32_t>(w >> (8 * ((row + x) & 7))) & 0xffu;
            y += static_cast<uint32_t>(w >> (8 * ((row + y) & 7))) & 0xffu;
            if constexpr (STATS) s.c[kStatTable] += 1u;
        } else {
            x += ld_moff(v, row + x, pol);
            y += ld_moff(v, row + y, pol);
            if constexpr (STATS) s.c[kStatTable] += 2u;
        }
        const Entry e1 = ld_entry_keep(v.mst, x, v.nmicro, pol);
        Entry e2 = e1;
        if (x != y) e2 = ld_entry_keep(v.mst, y, v.nmicro, pol);
        if constexpr (STATS) s.c[kStatTable] += x != y ? 2u : 1u;
        return better(e1, e2);
    }
    const Entry *t = v.st + static_cast<uint64_t>(lev) * v.nb;
    const uint64_t size = static_cast<uint64_t>(v.levels - lev) * v.nb;
    const Entry e1 = ld_entry_keep(t, x, size, pol);
    const Entry e2 = ld_entry_keep(t, y, size, pol);
    if constexpr (STATS) s.c[kStatTable] += 2u;
    return better(e1, e2);
}

// One step of the queued form over `cnt` queries from `base` on (cnt <=
// THREADS * QPT): thread t handles base + t + k * THREADS, already loaded
// into qq. FULL: cnt == THREADS * QPT, so no query needs a bounds check.
// MICRO: the index has the sub-block level (then every query inside one
// block spans few enough micro-blocks for the micro table, and only the
// block table serves longer ones). LIGHT: a light index (no per-element
// entries). Queries left open join the warp's queue, whose length `count`
// carries from step to step; `id0` is the step's first query in the CTA's
// numbering. The caller drains the queue.
template <bool ALIGNED, bool MICRO, bool LIGHT, uint32_t MODE, int THREADS, int QPT, bool STATS,
          bool FULL>
__device__ __forceinline__ void answer_step_queued(const V1View &v, const QueryOut &o,
                                                   int64_t base, uint32_t cnt, uint32_t id0,
                                                   const int2 (&qq)[QPT], QStats &s,
                                                   MissQueue<QPT> &mq, uint32_t &count) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t pol = l2_keep_policy();
    float *const vs = o.val ? o.val + base : nullptr;
    int32_t *const is = o.idx ? o.idx + base : nullptr;
    Entry res[QPT];
    bool ok[QPT], scan[QPT], mic[QPT];
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const uint32_t j = threadIdx.x + k * THREADS;
        const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
        ok[k] = (FULL || j < cnt) && qq[k].x >= 0 && l <= r && r < v.n;
        scan[k] = MICRO && (l >> 5) == (r >> 5);
        mic[k] = false;
        res[k] = kEntryNone;
        if (ok[k] && !scan[k]) res[k] = superset_probe<MICRO, STATS>(v, l, r, pol, s, mic[k]);
    }
    bool miss[QPT];
    bool any_miss = false;
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const uint32_t j = threadIdx.x + k * THREADS;
        const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
        miss[k] = false;
        if (!ok[k]) {
            if (FULL || j < cnt) {
                put_invalid(o, base + j);
                if constexpr (STATS) s.c[kStatInvalid] += 1u;
            }
            continue;
        }
        // a query inside one micro-block still holds kEntryNone here, whose
        // index lies outside [l, r]
        miss[k] = entry_idx(res[k]) - l > r - l;
        any_miss |= miss[k];
        if constexpr (STATS) {
            if (MICRO && scan[k]) {
                s.c[kStatMicroScan] += 1u;
                s.c[kStatSectors] += range_sectors(v, l, r);
            } else {
                s.c[kStatFirst] += miss[k] ? 0u : 1u;
            }
        }
        // the probe's answer is stored even for a query it leaves open: the
        // drain (same warp, after __syncwarp) or the warp scan (same thread)
        // overwrites it, and whole-warp stores keep the output lines whole
        if (vs) __stcs(reinterpret_cast<unsigned int *>(vs) + j, decode_bits<MODE>(res[k]));
        if (is) __stcs(is + j, static_cast<int32_t>(entry_idx(res[k])));
    }
    if (!__any_sync(0xffffffffu, any_miss)) return;
    bool wscan[QPT];
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
        wscan[k] = false;
        if (!MICRO && miss[k]) {
            const uint32_t lB = div31(l, v.dv);
            if (lB == div31(r, v.dv)) {
                // one block without the sub-block level: an edge entry when the
                // query touches the block's edge, else the warp scans it
                const uint32_t bstart = lB * v.bs;
                const uint32_t bend = min(bstart + v.bs, v.n) - 1u;
                if (r != bend && l != bstart) {
                    miss[k] = false;
                    wscan[k] = true;
                }
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, miss[k]);
        if (miss[k]) {
            const uint32_t e = count + __popc(mask & ((1u << lane) - 1u));
            mq.l[e] = l | (entry_idx(res[k]) < l ? kMissLeft : 0u);
            mq.r[e] = r;
            mq.id[e] = id0 + threadIdx.x + k * THREADS;
        }
        count += __popc(mask);
    }
    if constexpr (!MICRO) {
#pragma unroll
        for (int k = 0; k < QPT; ++k) {
            unsigned mask = __ballot_sync(0xffffffffu, wscan[k]);
            while (mask) {
                const int src = __ffs(mask) - 1;
                mask &= mask - 1u;
                const uint32_t ls = __shfl_sync(0xffffffffu, static_cast<uint32_t>(qq[k].x), src);
                const uint32_t rs = __shfl_sync(0xffffffffu, static_cast<uint32_t>(qq[k].y), src);
                const Entry e = warp_scan_range<ALIGNED>(v, ls, rs, static_cast<int>(lane), MODE);
                if (static_cast<int>(lane) == src) {
                    put_result(o, base + threadIdx.x + k * THREADS, e, MODE);
                    if constexpr (STATS) {
                        s.c[kStatWarpScan] += 1u;
                        s.c[kStatSectors] += range_sectors(v, ls, rs);
                    }
                }
            }
        }
    }
}

// Adds a thread's counters to the launch's device counters (one atomic per
// warp and counter).
__device__ __forceinline__ void flush_stats(const QStats &s, unsigned long long *out) {
#pragma unroll
    for (int c = 0; c < kStatCount; ++c) {
        unsigned long long x = s.c[c];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) x += __shfl_down_sync(0xffffffffu, x, d);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(out + c, x);
    }
}

// Answer queries [q0, q1) of one array with the whole CTA (THREADS
// threads) in the queued form, QPT queries per thread per step; `mq` is the
// calling warp's queue, empty on entry and on return. LIGHT: a light index.
template <bool ALIGNED, bool MICRO, bool LIGHT, uint32_t MODE, int THREADS, int QPT>
__device__ __forceinline__ void answer_range_queued(const V1View &v, const QueryOut &o,
                                                    int64_t q0, int64_t q1, MissQueue<QPT> &mq) {
    constexpr int64_t step = static_cast<int64_t>(THREADS) * QPT;
    const StepMap map{q0, step};
    QStats s;
    uint32_t waiting = 0, id0 = 0;
    for (int64_t base = q0; base < q1; base += step, id0 += step) {
        int2 qq[QPT];
        load_queries<QPT>(o, base, q1, qq);
        if (base + step <= q1)
            answer_step_queued<ALIGNED, MICRO, LIGHT, MODE, THREADS, QPT, false, true>(
                v, o, base, static_cast<uint32_t>(step), id0, qq, s, mq, waiting);
        else
            answer_step_queued<ALIGNED, MICRO, LIGHT, MODE, THREADS, QPT, false, false>(
                v, o, base, static_cast<uint32_t>(q1 - base), id0, qq, s, mq, waiting);
        // one site for the drain: its code is large, and every copy of it
        // costs instruction fetches
        while (waiting >= (base + step >= q1 ? 1u : 32u))
            drain_misses<ALIGNED, MICRO, LIGHT, MODE, false, THREADS, QPT>(v, o, map, mq, waiting,
                                                                           l2_keep_policy(), s);
    }
}

}  // namespace rmq
