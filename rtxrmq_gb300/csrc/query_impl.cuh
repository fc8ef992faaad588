// query_impl.cuh -- the CTA-level query body shared by the plain query kernel
// (query.cu) and the persistent batch kernel (batch.cu).
//
// It replaces RTX_blocks' ray programs (src/rtx_kernels.cu:85-193 for
// values, 350-465 for indices). The reference fires up to three rays per
// query: one through the fully covered blocks lB+1..rB-1, one through the
// left partial block and one through the right partial block, and keeps the
// closest hit. Here the same decomposition is answered from arrays:
//   left partial block   -> a line of values and the micro-blocks after it
//   right partial block  -> a line of values and the micro-blocks before it
//   full blocks between  -> two sparse-table entries (L2-resident)
// (suf[l] and pre[r] for the partial blocks of an index without the sub-block
// level), and it is needed only for the few queries a cheaper test does not
// settle: every query first probes a small L2-resident table over all the
// units it touches (blocks lB..rB, or the 32-element micro-blocks
// l/32..r/32), and when the leftmost best of that superset lies inside [l, r]
// it is the answer without a look at the values. A query inside one
// micro-block is settled from that 128-byte line, copied to shared memory by
// 8 lanes; without the sub-block level a query inside one block that
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
#include "lines.cuh"
#include "tables_impl.cuh"

namespace rmq {

// One built array: values A[off .. off + n) of the buffer A (loads never go
// past A[limit - 1]); structure arrays are array-relative. A batched array
// that starts off a 128-byte boundary is built from that boundary on, with
// `lead` elements before its first that no query reaches (LEAD): positions
// here count from the boundary, queries and answers from the array's first
// element.
struct V1View {
    const float *A;
    int64_t off;
    int64_t limit;
    uint32_t n;
    uint32_t lead;  // elements before the array's first (LEAD launches)
    uint32_t bs;
    uint32_t nb;
    Div31 dv;
    const Entry *st;
    // block table of larger blocks (2^k elements, cdiv the multiplier of their
    // Div31), for queries whose end micro-blocks are coarse_from or more apart
    const Entry *cst;
    uint32_t cnb, clevels, cdiv;
    uint32_t coarse_from;  // 2^32 - 1: none
    // table index: 32-element micro-blocks (local index / 32) and the micro
    // table over their minima (tables_impl.cuh); blocks hold whole
    // micro-blocks. Null when the index has none: per-element entries then
    // (same-block queries use the warp-cooperative scan)
    const Entry *mst;      // micro-block minima
    const void *mask;
    bool wide;             // 64-bit masks, else 32-bit
    const void *moff;
    uint32_t moff_bytes;
    uint32_t nmicro;
    const Entry *pre;
    const Entry *suf;
    uint32_t kmode;     // KeyMode: element type and minimum / maximum
    uint32_t levels;    // sparse-table levels (st holds levels * nb entries)
    uint32_t mlevels;   // micro-table levels (moff holds moff_rows(mlevels) rows of nmicro)
    bool light;         // counting launches: how the end parts are counted
    // a query whose end micro-blocks ml < mr have mr - ml < micro_span is probed
    // through the micro table (at most 2^mlevels - 1; 0: no micro level)
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

// Mask of micro-block j, its low 32 bits, and offset i of the micro table's
// rows. Width is the same for every query of an index, so the branches on it
// do not diverge. The low word serves windows of up to 32 micro-blocks of
// either width, with 32-bit shifts (n = 1e8, lr = -3, with the queue's one
// drain site: 0.795 and 0.771 ms).
__device__ __forceinline__ uint32_t ld_mask_low(const V1View &v, uint32_t j, uint64_t pol) {
    if (!rmq_chk(j < v.nmicro)) return 1u;
    const uint32_t *at = static_cast<const uint32_t *>(v.mask) + (static_cast<uint64_t>(j) << (v.wide ? 1 : 0));
    uint32_t r;
    asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(r) : "l"(at), "l"(pol));
    return r;
}
__device__ __forceinline__ uint64_t ld_mask(const V1View &v, uint32_t j, uint64_t pol) {
    if (!rmq_chk(j < v.nmicro)) return 1u;
    if (v.wide) {
        unsigned long long r;
        asm volatile("ld.global.L2::cache_hint.u64 %0, [%1], %2;"
                     : "=l"(r) : "l"(static_cast<const uint64_t *>(v.mask) + j), "l"(pol));
        return r;
    }
    uint32_t r;
    asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;"
                 : "=r"(r) : "l"(static_cast<const uint32_t *>(v.mask) + j), "l"(pol));
    return r;
}
__device__ __forceinline__ uint32_t ld_moff(const V1View &v, uint64_t i, uint64_t pol) {
    if (!rmq_chk(i < static_cast<uint64_t>(moff_rows(v.mlevels, v.wide)) * v.nmicro)) return 0u;
    uint32_t r;
    if (v.moff_bytes == 1u)
        asm volatile("ld.global.L2::cache_hint.u8 %0, [%1], %2;"
                     : "=r"(r) : "l"(static_cast<const uint8_t *>(v.moff) + i), "l"(pol));
    else
        asm volatile("ld.global.L2::cache_hint.u16 %0, [%1], %2;"
                     : "=r"(r) : "l"(static_cast<const uint16_t *>(v.moff) + i), "l"(pol));
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

__device__ __forceinline__ void put_result(const QueryOut &o, int64_t i, Entry e, uint32_t mode,
                                           uint32_t lead = 0u) {
    put_bits_idx(o, i, o.val ? entry_bits(e, mode) : 0u, entry_idx(e) - lead);
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

// Queries base + threadIdx.x + k * blockDim.x (k < QPT) of [.., q1), loaded
// ahead of use (the query stream may come from host memory over the host
// link, so a caller can issue the next step's loads before answering the
// current step). A query past q1 is an invalid one.
template <int QPT>
__device__ __forceinline__ void load_queries(const QueryOut &o, int64_t base, int64_t q1,
                                             int2 (&qq)[QPT]) {
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const int64_t i = base + threadIdx.x + static_cast<int64_t>(k) * blockDim.x;
        qq[k] = make_int2(-1, -1);
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
// better(part, best of units a+1..b) when the latter falls at or before r
// (`part` is the best of [l, end of a]), and the three-part decomposition of
// the reference (left partial, units between, right partial) only when it
// does not. The parts, the random HBM lookups, are read only on those two
// fallbacks.

// Query counters of a measurement launch (rmq_query_stats); the normal
// kernels compile them out.
enum QStat : int {
    kStatFirst = 0,   // settled by the superset probe
    kStatSecond,      // settled by a second probe and one end part, or by one mask (tied_entry)
    kStatFull,        // three-part decomposition: two end parts and a middle probe
    kStatMicroScan,   // inside one micro-block: its line of values is scanned
    kStatBlockEdge,   // one block, no sub-block level: pre / suf at a block edge
    kStatWarpScan,    // one block, no sub-block level: warp-cooperative scan
    kStatEntries,     // end parts read (pre / suf entries, or lines of values)
    kStatTable,       // small-table words read (sparse table, masks, offsets and minima)
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

// Leftmost best of micro-blocks a..b (a <= b, b - a + 1 < 2^mlevels): from
// the mask of a for up to 32 (64) of them, else the better of the two windows
// of 2^k that cover them (the lowest such k from the masks' highest bits, then
// offset rows).
template <bool STATS>
__device__ __forceinline__ Entry micro_probe(const V1View &v, uint32_t a, uint32_t b, uint64_t pol,
                                             QStats &s) {
    const uint32_t w = b - a + 1u;
    if (w <= (v.wide ? 64u : 32u)) {
        uint32_t x = a;
        if (w > 32u)
            x += 63u - __clzll(ld_mask(v, a, pol) & (~0ull >> (64u - w)));
        else if (w > 1u)
            x += 31u - __clz(ld_mask_low(v, a, pol) & (0xffffffffu >> (32u - w)));
        if constexpr (STATS) s.c[kStatTable] += w > 1u ? 2u : 1u;
        return ld_entry_keep(v.mst, x, v.nmicro, pol);
    }
    const uint32_t lev = ilog2(w);
    uint32_t x = a, y = b + 1u - (1u << lev);
    const uint32_t row0 = mask_levels(v.wide);
    if (lev < row0) {
        const uint64_t mx = ld_mask(v, x, pol), my = ld_mask(v, y, pol);
        x += 63u - __clzll(mx);
        y += 63u - __clzll(my);
    } else {
        const uint64_t row = static_cast<uint64_t>(lev - row0) * v.nmicro;
        const uint32_t ox = ld_moff(v, row + x, pol), oy = ld_moff(v, row + y, pol);
        x += ox;
        y += oy;
    }
    const Entry ex = ld_entry_keep(v.mst, x, v.nmicro, pol);
    Entry ey = ex;
    if (y != x) ey = ld_entry_keep(v.mst, y, v.nmicro, pol);
    if constexpr (STATS) s.c[kStatTable] += y != x ? 4u : 3u;
    return better(ex, ey);
}

// Without the sub-block level: suf[l] (best of A[l .. end of l's block]),
// pre[r] (best of A[start of r's block .. r]).
template <bool STATS>
__device__ __forceinline__ Entry left_entry(const V1View &v, uint32_t l, QStats &s) {
    if constexpr (STATS) s.c[kStatEntries] += 1u;
    return ld_entry(v.suf, l, v.n);
}
template <bool STATS>
__device__ __forceinline__ Entry right_entry(const V1View &v, uint32_t r, QStats &s) {
    if constexpr (STATS) s.c[kStatEntries] += 1u;
    return ld_entry(v.pre, r, v.n);
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
// A query inside one micro-block, and the end part of a query whose probe did
// not settle it, is the best of part of one 32-element line. Scanned by the
// lane that owns the query straight from memory, a load instruction touches
// up to 32 different 128-byte lines, one L1 tag lookup each, for up to 9
// instructions. Here the warp first copies the lines of its requests into
// shared memory, 8 lanes per line and 16 bytes each (one tag lookup per line,
// all copies in flight together, no registers held), and the probes of the
// same drain run while they arrive; then every lane reduces lines without
// bank conflicts (chunks XOR-swizzled by the line's slot).

// Lines a warp stages at a time: 16 (2 KB per warp, two lanes per line). 32
// need fewer instructions but twice the shared memory, taken from the L1 that
// block tables live in (n = 1e8, 2^26 queries, uniform lengths, bs 2^15:
// 0.33 ms with 16, 0.57 with 32; ranges of 32: 1.60 and 1.81).
constexpr int kStageLines = 16;

// Starts copying the chunks holding a set bit of the requests of lanes
// h .. h + kStageLines - 1 into the warp's stage. Bytes past the end of the
// buffer are not read.
template <bool ALIGNED>
__device__ __forceinline__ void stage_lines(const V1View &v, uint32_t line, uint32_t bits,
                                            uint32_t stage, uint32_t h) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, grp = lane >> 3;
    // whole chunks by 16-byte copies when every requested line lies inside
    // the buffer and on a 16-byte boundary
    const int64_t end = v.off + static_cast<int64_t>(line) * 32 + 32;
    const bool whole = ALIGNED && (v.off & 3) == 0 &&
                       !__any_sync(0xffffffffu, bits != 0u && end > v.limit);
    const float *const base = v.A + v.off + 4 * sub;
    if (whole) {
        // slot 4 t + grp: its swizzle depends on t's parity alone
        const uint32_t d0 = staged_line(stage, grp) ^ (sub << 4);
        const uint32_t d1 = staged_line(stage, 4u + grp) ^ (sub << 4);
        // through L1 (.ca): of a small array thousands of warps want the same
        // few lines, which queue up at the L2 (n = 1335, 2^25 ranges of 20: 0.92
        // ms, 1.78 with .cg; n = 1e8, lr=-3: 0.798 and 0.787)
#pragma unroll
        for (uint32_t t = 0; t < kStageLines / 4; ++t) {
            const uint32_t ln = __shfl_sync(0xffffffffu, line, h + 4u * t + grp);
            const uint32_t bt = __shfl_sync(0xffffffffu, bits, h + 4u * t + grp);
            const float *src = base + static_cast<size_t>(ln) * 32;
            const uint32_t dst = ((t & 1u) ? d1 : d0) + (t / 2u) * 1024u;
            if ((bt >> (4u * sub)) & 15u && rmq_chk(v.off + static_cast<int64_t>(ln) * 32 + 32 <= v.limit))
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
        }
    } else {
#pragma unroll 1
        for (uint32_t t = 0; t < kStageLines / 4; ++t) {
            const uint32_t slot = 4u * t + grp;
            const uint32_t ln = __shfl_sync(0xffffffffu, line, h + slot);
            const uint32_t nib = (__shfl_sync(0xffffffffu, bits, h + slot) >> (4u * sub)) & 15u;
            const uint32_t dst = staged_line(stage, slot) ^ (sub << 4);
            const float *src = base + static_cast<size_t>(ln) * 32;
            const int64_t g = v.off + static_cast<int64_t>(ln) * 32 + 4 * sub;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if ((nib >> k) & 1u && rmq_chk(g >= 0 && g + k < v.limit))
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                                 :: "r"(dst + 4u * k), "l"(src + k) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// What a request's lane knows of its line before it forms the entry: the bits
// of the best element and its position, or that every element of the request
// has the largest key (no number, or the fill), when the first of them is it.
struct LineBest {
    uint32_t bits, pos;
    bool last;
};

// Waits for the staged lines and gives lanes h .. h + kStageLines - 1 the best
// of their requests (leftmost; meaningless without a set bit). Two lanes
// reduce a line, four consecutive chunks each; they meet on the value, and a
// request's key is formed once, by its own lane. The set bits of a request
// are consecutive.
template <uint32_t MODE>
__device__ __forceinline__ void reduce_lines(uint32_t bits, uint32_t stage, uint32_t h, LineBest &out) {
    using B = Best<MODE>;
    static_assert(kStageLines == 16, "two lanes per line");
    const uint32_t lane = threadIdx.x & 31u;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    const uint32_t slot = lane >> 1, c0 = (lane & 1u) * 4u;
    const uint32_t mine = (__shfl_sync(0xffffffffu, bits, h + slot) >> (4u * c0)) & 0xffffu;
    const uint32_t base = staged_line(stage, slot) ^ (c0 << 4);
    // the elements outside the request in its first and last chunk are
    // overwritten with the fill, so that only whole chunks are selected below
    const uint32_t first = mine ? __ffs(mine) - 1u : 0u, end = 31u - __clz(mine | 1u);
    const uint32_t fill = B::bits(B::fill());
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) {
        if (k < (first & 3u))
            asm volatile("st.shared.u32 [%0], %1;" :: "r"((base ^ ((first >> 2) << 4)) + 4u * k), "r"(fill) : "memory");
        if (3u - k > (end & 3u))
            asm volatile("st.shared.u32 [%0], %1;" :: "r"((base ^ ((end >> 2) << 4)) + 12u - 4u * k), "r"(fill) : "memory");
    }
    typename B::T m[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint4 f = lds_chunk(base ^ (c << 4));
        m[c] = B::best(B::best(B::best(B::of(f.x), B::of(f.y)), B::of(f.z)), B::of(f.w));
        m[c] = mine & (15u << (4 * c)) ? m[c] : B::fill();
    }
    typename B::T mm = B::best(B::best(m[0], m[1]), B::best(m[2], m[3]));
    const typename B::T both = B::best(mm, B::of(__shfl_xor_sync(0xffffffffu, B::bits(mm), 1)));
    // the half that holds the best (the left one when both do), in it the
    // first chunk and the first element
    const uint32_t holds = __ballot_sync(0xffffffffu, mm == both);
    const uint32_t cs = m[0] == mm ? 0u : m[1] == mm ? 1u : m[2] == mm ? 2u : 3u;
    uint32_t wb;
    const uint32_t pos = 4u * (c0 + cs) + first_in_chunk<MODE>(lds_chunk(base ^ (cs << 4)), mm, wb);
    const uint32_t me = (lane - h) & 15u;
    const uint32_t from = 2u * me + ((holds >> (2u * me)) & 1u ^ 1u);
    const uint32_t rb = __shfl_sync(0xffffffffu, wb, from), rp = __shfl_sync(0xffffffffu, pos, from);
    const uint32_t rl = __shfl_sync(0xffffffffu, !(both == both) || both == B::fill() ? 1u : 0u, from);
    if (lane - h < kStageLines) out = LineBest{rb, rp, rl != 0u};
    __syncwarp();  // the stage may be written again
}

template <uint32_t MODE>
__device__ __forceinline__ Entry line_entry(const LineBest &x, uint32_t line, uint32_t bits) {
    if (bits == 0u) return kEntryNone;
    const uint32_t key = x.last ? 0xffffffffu : key_of(x.bits, MODE);
    const uint32_t lo = x.last ? (__ffs(bits) - 1u) << 1 : (x.pos << 1) | negzero_of(x.bits, MODE);
    return (static_cast<uint64_t>(key) << 32) | ((line << 6) + lo);
}

// Bits lo .. hi (inclusive, 0 <= lo <= hi <= 31)
__device__ __forceinline__ uint32_t bit_range(uint32_t lo, uint32_t hi) {
    return (0xffffffffu >> (31u - hi)) & (0xffffffffu << lo);
}

// Table index: of the query's part in its end unit on one side, [l, end of
// l's unit] (left) or [start of r's unit, r] (right), what lies outside the
// line of its end: for a block, the best of the block's whole micro-blocks on
// that side. The side is a value, not a branch, so that lanes settling left
// and right parts run the same code.
template <bool STATS>
__device__ __forceinline__ Entry end_rest(const V1View &v, bool micro, bool left, uint32_t a,
                                          uint32_t b, uint32_t l, uint32_t r, uint64_t pol,
                                          QStats &s) {
    if constexpr (STATS) {
        if (v.light)
            s.c[kStatSectors] += range_sectors(v, left ? l : (r & ~31u), left ? l | 31u : r);
        else
            s.c[kStatEntries] += 1u;
    }
    if (micro) return kEntryNone;
    // block a is full when a < b: its last micro-block ends inside the array
    const uint32_t pb = v.bs >> 5;
    const uint32_t ml = l >> 5, me = (a + 1u) * pb - 1u;
    const uint32_t mr = r >> 5, ms = b * pb;
    const bool has = left ? ml < me : ms < mr;
    if (!has) return kEntryNone;
    return micro_probe<STATS>(v, left ? ml + 1u : ms, left ? me : mr - 1u, pol, s);
}

// Without the sub-block level: settles one query whose superset best lay
// outside [l, r], or inside one block at an edge, from the per-element
// entries: the query's part in the end block on that side and a narrower
// probe, loaded together, then only if needed the other end's part and the
// middle blocks.
template <bool STATS>
__device__ __forceinline__ Entry finish_entries(const V1View &v, bool left, uint32_t l, uint32_t r,
                                                uint64_t pol, QStats &s) {
    const uint32_t a = div31(l, v.dv), b = div31(r, v.dv);
    if (a == b) {
        if constexpr (STATS) s.c[kStatBlockEdge] += 1u;
        const uint32_t bend = min(a * v.bs + v.bs, v.n) - 1u;
        return r == bend ? left_entry<STATS>(v, l, s) : right_entry<STATS>(v, r, s);
    }
    // the narrower probe first: its loads are in flight while the part's
    // entry is loaded
    const Entry e2 = st_probe<STATS>(v, left ? a + 1u : a, left ? b : b - 1u, pol, s);
    const Entry e1 = left ? left_entry<STATS>(v, l, s) : right_entry<STATS>(v, r, s);
    const uint32_t m2 = entry_idx(e2);
    if (left ? m2 <= r : m2 >= l) {
        if constexpr (STATS) s.c[kStatSecond] += 1u;
        return better(e1, e2);
    }
    if constexpr (STATS) s.c[kStatFull] += 1u;
    const Entry mid = (b - a >= 2u) ? st_probe<STATS>(v, a + 1u, b - 1u, pol, s) : kEntryNone;
    const Entry other = left ? right_entry<STATS>(v, r, s) : left_entry<STATS>(v, l, s);
    return better(better(e1, other), mid);
}

// Ties. Where the least value of a range repeats all over the array, its first
// place in l's block nearly always lies before l, and every query of the block
// tables is open. The best of the micro-blocks from l's on that one mask
// covers answers such a query when it has the value that the probe found and
// lies at or after l; no end part is read. A warp looks for it when many of its 64 queries are open:
// of distinct values few are, and none of those is answered this way (n = 2^27,
// values of 256, 2^26 ranges of 2^16: 2.70 ms, so 0.94; n = 4.5e7, 2^23 ranges of
// uniform length: 0.33 and 0.14).
constexpr uint32_t kManyOpen = 16;
template <bool STATS>
__device__ __forceinline__ Entry tied_entry(const V1View &v, uint32_t l, uint64_t pol, QStats &s) {
    if constexpr (STATS) s.c[kStatTable] += 2u;
    return ld_entry_keep(v.mst, (l >> 5) + 63u - __clzll(ld_mask(v, l >> 5, pol)), v.nmicro, pol);
}

// Leftmost best of l .. r inside one micro-block and within kShortChunks
// 16-byte chunks, by the lane alone. More chunks cost more L1 lookups than
// the warp's staged copy of the line does (one). 2^25 ranges of 8 in an array
// of 3e5: 0.99 ms all staged, 1.06 with two chunks, 0.74 with three.
constexpr uint32_t kShortChunks = 3;
template <bool ALIGNED, uint32_t MODE>
__device__ __forceinline__ Entry short_range(const V1View &v, uint32_t l, uint32_t r) {
    const uint32_t c = l & ~3u;
    const int64_t g = v.off + c;
    uint32_t w[4 * kShortChunks];
    if (ALIGNED && (v.off & 3) == 0 && g + 4 * kShortChunks <= v.limit) {
#pragma unroll
        for (uint32_t k = 0; k < kShortChunks; ++k) {
            // past r the first chunk again: no further line
            const uint4 x = ld_elem4(v, c + 4u * k <= r ? g + 4 * k : g);
            w[4 * k] = x.x, w[4 * k + 1] = x.y, w[4 * k + 2] = x.z, w[4 * k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (uint32_t k = 0; k < 4 * kShortChunks; ++k)
            w[k] = c + k >= l && c + k <= r ? ld_elem(v, g + k) : 0u;
    }
    using B = Best<MODE>;
    typename B::T best = B::fill();
#pragma unroll
    for (uint32_t k = 0; k < 4 * kShortChunks; ++k)
        if (c + k >= l && c + k <= r) best = B::best(best, B::of(w[k]));
    // the first element holding it; l when none does or only the fill
    uint32_t pos = l, wb = 0u;
#pragma unroll
    for (int k = 4 * kShortChunks - 1; k >= 0; --k)
        if (c + k >= l && c + k <= r && B::of(w[k]) == best) pos = c + k, wb = w[k];
    const bool last = !(best == best) || best == B::fill();
    return (static_cast<uint64_t>(last ? 0xffffffffu : key_of(wb, MODE)) << 32) |
           ((last ? l : pos) << 1) | (last ? 0u : negzero_of(wb, MODE));
}

// One warp's queue (up to 31 waiting queries plus the 32 that one query slot
// of a step can add, 16 bytes each) and its line stage. What they take from
// the L1 matters, the block table's upper levels live there: 3 KB per warp
// are 100 KB per SM, with 256 bytes more the next carve-out is 132 KB (n =
// 1e8, uniform lengths, bs 2^14: 0.36 and 0.45 ms). `id` numbers the queries
// of the CTA in the order it takes them: step * step size + place in the
// step.
template <bool MICRO, bool WHOLE = false>
struct MissQueue {
    static constexpr int kCap = 64;
    uint4 stage[MICRO ? kStageLines * 8 : 1];  // on a 128-byte boundary (staged_line)
    uint32_t l[kCap];    // kMissLeft set: the probe's best lay left of l
    uint32_t r[kCap];    // kSecond set: back for its other end
    uint32_t id[kCap];   // below 2^30
    uint32_t key[MICRO ? kCap : 1];
};
template <>
struct MissQueue<true, true> : MissQueue<true, false> {
    Entry done[kCap];  // answers of the step's queued queries
};
static_assert(sizeof(MissQueue<true>) % 128 == 0 && sizeof(MissQueue<true, true>) % 128 == 0,
              "the stages of all warps lie on 128-byte boundaries");
constexpr uint32_t kMissLeft = 0x80000000u;  // above every index
// A query back for its other end has the best of the end that is settled in
// its entry: its key, its index in place of that end's position (it lies in
// the same unit), its -0.0 flag, and which table's units are meant.
constexpr uint32_t kSecond = 0x80000000u;
constexpr uint32_t kPartNegzero = 0x80000000u, kPartMicro = 0x40000000u;  // in id

// The queries a CTA takes: steps of `chunk` consecutive ones, `stride` apart.
struct StepMap {
    int64_t first;
    int64_t stride;
    __device__ __forceinline__ int64_t query(uint32_t id, uint32_t chunk) const {
        return first + static_cast<int64_t>(id / chunk) * stride + id % chunk;
    }
};

// Settles the last min(count, 32) queued queries, one per lane; the whole
// warp calls it (count is warp-uniform). With the sub-block level, a query
// inside one micro-block is one line of values. A query whose probe's best
// lay outside needs the units without the end unit that held it (e2) and its
// part in that end unit; e2 settles it when it lies inside [l, r]. Else,
// rarely, it joins the queue again, for the units between both ends and its
// part at the other end: few lanes in a warp need that, so doing it at once
// would cost every drain a second pass.
template <bool ALIGNED, bool MICRO, uint32_t MODE, bool STATS, bool LEAD, int THREADS, int QPT,
          bool WHOLE>
__device__ __forceinline__ void drain_misses(const V1View &v, const QueryOut &o,
                                             const StepMap &map, MissQueue<MICRO, WHOLE> &mq,
                                             uint32_t &count, uint64_t pol, QStats &s) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t take = count < 32u ? count : 32u;
    __syncwarp();
    count -= take;
    const uint32_t e = count + lane;
    const bool act = lane < take;
    const uint32_t lq = act ? mq.l[e] : 0u, rq = act ? mq.r[e] : 0u;
    const uint32_t iq = act ? mq.id[e] : 0u;
    const uint32_t l = lq & ~kMissLeft, r = rq & ~kSecond;
    const uint32_t id = iq & ~(kPartNegzero | kPartMicro);
    const bool left = (lq & kMissLeft) != 0u;
    Entry res = kEntryNone;
    bool again = false, micro = false;
    if constexpr (!MICRO) {
        if (act) res = finish_entries<STATS>(v, left, l, r, pol, s);
    } else {
        const uint32_t stage = static_cast<uint32_t>(__cvta_generic_to_shared(mq.stage));
        const bool second = (rq & kSecond) != 0u;
        const bool side = left != second;  // the end whose line is wanted
        const bool scan = !second && (l >> 5) == (r >> 5);
        const uint32_t line = (side ? l : r) >> 5;
        // the left end's unit lies before the right end's, so its line is whole
        uint32_t bits = scan ? bit_range(l & 31u, r & 31u)
                        : side ? 0xffffffffu << (l & 31u) : 0xffffffffu >> (31u - (r & 31u));
        if (!act) bits = 0u;
        stage_lines<ALIGNED>(v, line, bits, stage, 0u);
        // the probes run while the lines arrive
        if (act && !scan) {
            micro = second ? (iq & kPartMicro) != 0u : (r >> 5) - (l >> 5) < v.micro_span;
            const uint32_t a = micro ? (l >> 5) : div31_ge2(l, v.dv);
            const uint32_t b = micro ? (r >> 5) : div31_ge2(r, v.dv);
            const uint32_t lo = a + (left || second), hi = b - (!left || second);
            Entry e2 = kEntryNone;
            if (lo <= hi)
                e2 = micro ? micro_probe<STATS>(v, lo, hi, pol, s) : st_probe<STATS>(v, lo, hi, pol, s);
            res = end_rest<STATS>(v, micro, side, a, b, l, r, pol, s);
            const uint32_t m2 = entry_idx(e2);
            again = !second && (left ? m2 > r : m2 < l);
            if (!again) res = better(res, e2);
            if (second)
                res = better(res, (static_cast<uint64_t>(mq.key[e]) << 32) | ((left ? l : r) << 1) | (iq >> 31));
            if constexpr (STATS)
                if (!second) s.c[again ? kStatFull : kStatSecond] += 1u;
        }
        LineBest best;
        reduce_lines<MODE>(bits, stage, 0u, best);
        if (take > kStageLines) {
            stage_lines<ALIGNED>(v, line, bits, stage, kStageLines);
            reduce_lines<MODE>(bits, stage, kStageLines, best);
        }
        res = better(res, line_entry<MODE>(best, line, bits));
    }
    if (act && !again) {
        if constexpr (WHOLE)
            mq.done[id] = res;
        else
            put_result(o, map.query(id, THREADS * QPT), res, MODE, LEAD ? v.lead : 0u);
    }
    if constexpr (MICRO) {
        const unsigned mask = __ballot_sync(0xffffffffu, again);
        if (again) {
            const uint32_t w = count + __popc(mask & ((1u << lane) - 1u));
            const uint32_t at = entry_idx(res);
            mq.l[w] = left ? at | kMissLeft : l;
            mq.r[w] = (left ? r : at) | kSecond;
            mq.id[w] = id | (static_cast<uint32_t>(res) << 31) | (micro ? kPartMicro : 0u);
            mq.key[w] = static_cast<uint32_t>(res >> 32);
        }
        count += __popc(mask);
    }
    __syncwarp();
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
// it, else through a block table (two entries, one straight sequence), with
// COARSE that of the larger blocks for long queries. What the larger blocks
// leave open is drained with the smaller ones. For shorter ranges they leave
// too much open, also with a second probe before the queue (n = 1e7, lr=-2,
// blocks of 2048 and 1024: 0.67 ms so, 0.54 by the smaller ones at once).
template <bool MICRO, bool COARSE, bool STATS>
__device__ __forceinline__ Entry superset_probe(const V1View &v, uint32_t l, uint32_t r,
                                                uint64_t pol, QStats &s) {
    const uint32_t ml = l >> 5, mr = r >> 5;
    if (MICRO && mr - ml < v.micro_span) return micro_probe<STATS>(v, ml, mr, pol, s);
    const bool coarse = COARSE && mr - ml >= v.coarse_from;
    const uint32_t m = coarse ? v.cdiv : v.dv.m, sh = coarse ? 0u : v.dv.shift, nb = coarse ? v.cnb : v.nb;
    const uint32_t a = MICRO ? __umulhi(l, m) >> sh : div31(l, v.dv);
    const uint32_t b = MICRO ? __umulhi(r, m) >> sh : div31(r, v.dv);
    const int lev = ilog2(b - a + 1u);
    const Entry *t = (coarse ? v.cst : v.st) + static_cast<uint64_t>(lev) * nb;
    const uint64_t size = static_cast<uint64_t>((coarse ? v.clevels : v.levels) - lev) * nb;
    const Entry e1 = ld_entry_keep(t, a, size, pol);
    const Entry e2 = ld_entry_keep(t, b + 1u - (1u << lev), size, pol);
    if constexpr (STATS) s.c[kStatTable] += 2u;
    return better(e1, e2);
}

// One step of the queued form over `cnt` queries from `base` on (cnt <=
// THREADS * QPT): thread t handles base + t + k * THREADS, already loaded
// into qq (invalid from base + cnt on, so that only the rare path of invalid
// queries compares with cnt).
// MICRO: the index has the sub-block level (then every query inside one
// block spans few enough micro-blocks for the micro table, and only the
// block table serves longer ones). Queries left open join the warp's queue, whose length `count`
// carries from step to step (`last` empties it); `id0` is the step's first
// query in the CTA's numbering. SHORT: the lanes settle the shortest ranges
// themselves.
// WHOLE: the results go to host memory, where a store of part of a line travels
// the link by itself. Every query of the step is settled before any is stored (the
// queue is empty between steps, numbers are places in the warp's 64), and each slot
// is stored once, by the whole warp. The drains are less full, which the link hides
// (n = 1e6, 2^23 queries, 0.44 ms at the link's rate: ranges of 8 1.57 ms by the
// device-memory form, 0.47 so; ranges of 40 1.30 and 0.46; uniform lengths 0.44 both).
// In device memory L2 puts the parts together, and drains are worth more.
template <bool ALIGNED, bool MICRO, uint32_t MODE, int THREADS, int QPT, bool STATS, bool LEAD,
          bool SHORT, bool WHOLE = false>
__device__ __forceinline__ void answer_step_queued(const V1View &v, const QueryOut &o,
                                                   const StepMap &map, int64_t base, uint32_t cnt,
                                                   uint32_t id0, bool last,
                                                   const int2 (&in)[QPT], QStats &s,
                                                   MissQueue<MICRO, WHOLE> &mq, uint32_t &count) {
    static_assert(!WHOLE || (MICRO && SHORT && !STATS && !LEAD), "plain queries of a table index");
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t pol = l2_keep_policy();
    float *const vs = o.val ? o.val + base : nullptr;
    int32_t *const is = o.idx ? o.idx + base : nullptr;
    Entry res[QPT];
    bool ok[QPT], scan[QPT];
    const uint32_t lead = LEAD ? v.lead : 0u;
    int2 qq[QPT];
#pragma unroll
    for (int k = 0; k < QPT; ++k)  // unsigned: an end past 2^31 - 1 stays past n
        qq[k] = make_int2(static_cast<int>(in[k].x + lead), static_cast<int>(in[k].y + lead));
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
        ok[k] = in[k].x >= 0 && l <= r && r < v.n;
        scan[k] = MICRO && (l >> 5) == (r >> 5);
        res[k] = kEntryNone;
        if (ok[k] && !scan[k]) res[k] = superset_probe<MICRO, MICRO && SHORT, STATS>(v, l, r, pol, s);
    }
    bool miss[QPT];
    bool any_scan = false;
#pragma unroll
    for (int k = 0; k < QPT; ++k) {
        const uint32_t j = threadIdx.x + k * THREADS;
        const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
        miss[k] = false;
        if (!ok[k]) {
            if (j < cnt) {
                put_invalid(o, base + j);
                if constexpr (STATS) s.c[kStatInvalid] += 1u;
            }
            continue;
        }
        // a query inside one micro-block still holds kEntryNone here, whose
        // index lies outside [l, r]
        miss[k] = entry_idx(res[k]) - l > r - l;
        any_scan |= scan[k];
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
        // overwrites it, and whole-warp stores keep the output lines whole. A
        // query inside one micro-block has none
        if (WHOLE || (MICRO && scan[k])) continue;
        if (vs) __stcs(reinterpret_cast<unsigned int *>(vs) + j, decode_bits<MODE>(res[k]));
        if (is) __stcs(is + j, static_cast<int32_t>(entry_idx(res[k]) - lead));
    }
    if constexpr (!MICRO) {
#pragma unroll
        for (int k = 0; k < QPT; ++k) {
            // one block without the sub-block level: an edge entry when the
            // query touches the block's edge, else the warp scans it
            bool wscan = false;
            if (miss[k]) {
                const uint32_t l = static_cast<uint32_t>(qq[k].x), r = static_cast<uint32_t>(qq[k].y);
                const uint32_t lB = div31(l, v.dv);
                const uint32_t bstart = lB * v.bs;
                const uint32_t bend = min(bstart + v.bs, v.n) - 1u;
                wscan = lB == div31(r, v.dv) && r != bend && l != bstart;
                if (wscan) miss[k] = false;
            }
            unsigned mask = __ballot_sync(0xffffffffu, wscan);
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
    // what is open joins the queue, up to 32 queries at a time: both slots
    // together when they fit (about always: a few lanes in a hundred miss), else
    // one after the other. One site for the drain, whose code is large: before
    // each, and after the last step until the queue is empty (n = 1e8, lr = -2,
    // 2^26 queries: 0.586 and 0.565 ms slot by slot and so)
    static_assert(QPT == 2, "two slots");
    const uint32_t below = (1u << lane) - 1u;
    uint32_t m0 = __ballot_sync(0xffffffffu, miss[0]), m1 = __ballot_sync(0xffffffffu, miss[1]);
    if (!WHOLE && (m0 | m1) == 0u && !last) return;
    bool tiny[2] = {false, false};
    if (MICRO && SHORT && __any_sync(0xffffffffu, any_scan))
#pragma unroll
        for (int k = 0; k < 2; ++k)
            tiny[k] = scan[k] && miss[k] &&
                      (static_cast<uint32_t>(qq[k].y) >> 2) - (static_cast<uint32_t>(qq[k].x) >> 2) < kShortChunks;
    if (MICRO && SHORT && __any_sync(0xffffffffu, tiny[0] || tiny[1])) {
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            const uint32_t l = static_cast<uint32_t>(k ? qq[1].x : qq[0].x);
            const uint32_t r = static_cast<uint32_t>(k ? qq[1].y : qq[0].y);
            if (k ? tiny[1] : tiny[0]) {
                const Entry x = short_range<ALIGNED, MODE>(v, l, r);
                if constexpr (WHOLE) {
                    if (k) res[1] = x;
                    else res[0] = x;
                } else {
                    put_result(o, base + threadIdx.x + k * THREADS, x, MODE, lead);
                }
            }
        }
        miss[0] = miss[0] && !tiny[0];
        miss[1] = miss[1] && !tiny[1];
        m0 = __ballot_sync(0xffffffffu, miss[0]);
        m1 = __ballot_sync(0xffffffffu, miss[1]);
    }
    if (MICRO && __popc(m0) + __popc(m1) >= kManyOpen &&
        __any_sync(0xffffffffu, miss[0] && static_cast<uint32_t>((qq[0].y >> 5) - (qq[0].x >> 5)) >= v.micro_span)) {
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            const uint32_t l = static_cast<uint32_t>(k ? qq[1].x : qq[0].x);
            const uint32_t r = static_cast<uint32_t>(k ? qq[1].y : qq[0].y);
            const Entry e = k ? res[1] : res[0];
            if ((k ? miss[1] : miss[0]) && entry_idx(e) < l && (r >> 5) - (l >> 5) >= v.micro_span) {
                const Entry x = tied_entry<STATS>(v, l, pol, s);
                if ((x >> 32) == (e >> 32) && entry_idx(x) >= l) {
                    if constexpr (WHOLE) {
                        if (k) res[1] = x;
                        else res[0] = x;
                    } else {
                        put_result(o, base + threadIdx.x + k * THREADS, x, MODE, lead);
                    }
                    if (k) miss[1] = false;
                    else miss[0] = false;
                    if constexpr (STATS) s.c[kStatSecond] += 1u;
                }
            }
        }
        m0 = __ballot_sync(0xffffffffu, miss[0]);
        m1 = __ballot_sync(0xffffffffu, miss[1]);
    }
    const uint32_t n0 = __popc(m0), n1 = __popc(m1);
    if constexpr (WHOLE) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!miss[k]) continue;
            const uint32_t l = static_cast<uint32_t>(qq[k].x);
            const uint32_t e = k ? n0 + __popc(m1 & below) : __popc(m0 & below);
            mq.l[e] = l | (entry_idx(res[k]) < l ? kMissLeft : 0u);
            mq.r[e] = static_cast<uint32_t>(qq[k].y);
            mq.id[e] = lane + 32u * k;
        }
        count = n0 + n1;
#pragma unroll 1
        while (count > 0u)
            drain_misses<ALIGNED, MICRO, MODE, STATS, LEAD, THREADS, QPT>(v, o, map, mq, count, pol, s);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t j = threadIdx.x + k * THREADS;
            const Entry x = miss[k] ? mq.done[lane + 32u * k] : res[k];
            if (ok[k] && vs) __stcs(reinterpret_cast<unsigned int *>(vs) + j, decode_bits<MODE>(x));
            if (ok[k] && is) __stcs(is + j, static_cast<int32_t>(entry_idx(x)));
        }
        __syncwarp();  // the next step's drains write the answers again
        return;
    }
    const bool both = n0 + n1 <= 32u;
#pragma unroll 1
    for (uint32_t k = both ? 1u : 0u; k < 2u + (last ? 1u : 0u); ++k) {
        const uint32_t drain_at = k == 2u ? 1u : 32u;
#pragma unroll 1
        while (count >= drain_at)
            drain_misses<ALIGNED, MICRO, MODE, STATS, LEAD, THREADS, QPT>(v, o, map, mq, count, pol, s);
        if (k == 2u) break;
        const uint32_t first = both || k == 0u ? n0 : 0u;
        if (miss[0] && (both || k == 0u)) {
            const uint32_t l = static_cast<uint32_t>(qq[0].x), e = count + __popc(m0 & below);
            mq.l[e] = l | (entry_idx(res[0]) < l ? kMissLeft : 0u);
            mq.r[e] = static_cast<uint32_t>(qq[0].y);
            mq.id[e] = id0 + threadIdx.x;
        }
        if (miss[1] && k == 1u) {
            const uint32_t l = static_cast<uint32_t>(qq[1].x), e = count + first + __popc(m1 & below);
            mq.l[e] = l | (entry_idx(res[1]) < l ? kMissLeft : 0u);
            mq.r[e] = static_cast<uint32_t>(qq[1].y);
            mq.id[e] = id0 + threadIdx.x + THREADS;
        }
        count += first + (k == 1u ? n1 : 0u);
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
// calling warp's queue, empty on entry and on return.
template <bool ALIGNED, bool MICRO, uint32_t MODE, bool LEAD, int THREADS, int QPT>
__device__ __forceinline__ void answer_range_queued(const V1View &v, const QueryOut &o,
                                                    int64_t q0, int64_t q1, MissQueue<MICRO> &mq) {
    constexpr int64_t step = static_cast<int64_t>(THREADS) * QPT;
    const StepMap map{q0, step};
    QStats s;
    uint32_t waiting = 0, id0 = 0;
    int2 qq[QPT];
    load_queries<QPT>(o, q0, q1, qq);
    for (int64_t base = q0; base < q1; base += step, id0 += step) {
        int2 nxt[QPT];
        load_queries<QPT>(o, base + step, q1, nxt);  // in flight while this step is answered
        answer_step_queued<ALIGNED, MICRO, MODE, THREADS, QPT, false, LEAD, false>(
            v, o, map, base, static_cast<uint32_t>(min(step, q1 - base)), id0, base + step >= q1, qq,
            s, mq, waiting);
#pragma unroll
        for (int k = 0; k < QPT; ++k) qq[k] = nxt[k];
    }
}

}  // namespace rmq
