// tables_impl.cuh -- the micro table: for every window of consecutive
// 32-element micro-blocks a query can ask for, where its best one is.
//
//   mask[j]    bit d set when micro-block j + d is a strict new best of j ..
//              j + d (bit 0 always). The leftmost best of j .. j + w - 1 is j
//              + (highest set bit below w): one load answers every window of
//              up to 32 micro-blocks (64 where the table is small,
//              wide_masks), and the word's highest bit is the best of the
//              whole window.
//   moff       one row per level k = 6 .. (7 ..): the offset from j of the
//              leftmost best of the window of 2^k micro-blocks at j.
//
// Two windows of level k cover 2^k .. 2^(k+1) - 1 micro-blocks. The masks
// take the place of five or six rows of offsets, of which a query read two
// entries. What bounds short queries is L1 tag lookups, one per scattered
// load: two of them now (mask, minimum) for ranges of up to 1000 (2000)
// elements, three to four before.
#pragma once

#include "common.cuh"

namespace rmq {

// 64-bit masks while they and the minima (16 bytes per micro-block) take at
// most 60 MB: each die's half of the L2 holds a copy of what its SMs read, so
// more than that is read from DRAM. n = 1e8, 2^26 queries, bs 2048, ranges of
// 2^10: 0.62 ms with 64 bits, 0.72 with 32; n = 2^27, ranges of 32: 1.96 and
// 1.76.
RMQ_HD bool wide_masks(uint32_t nmicro) { return nmicro <= (60u << 20) / 16u; }

// Levels that need no offset row.
RMQ_HD uint32_t mask_levels(bool wide) { return wide ? 7u : 6u; }

// Rows of offsets of a micro table of `mlevels` levels.
RMQ_HD uint32_t moff_rows(uint32_t mlevels, bool wide) {
    return mlevels > mask_levels(wide) ? mlevels - mask_levels(wide) : 0u;
}

// Micro-blocks past a tile's last position that its windows reach (at least
// the masks' 63).
RMQ_HD uint32_t table_halo(uint32_t mlevels) {
    return mlevels > 7u ? (1u << (mlevels - 1)) - 1u : 63u;
}

#ifdef __CUDACC__

// One micro table in global memory.
struct MicroTable {
    const Entry *mst;   // [nmicro] micro-block minima
    void *mask;         // [nmicro], 64 or 32 bits wide
    void *moff;         // [moff_rows][nmicro], moff_bytes wide
    uint32_t moff_bytes;
    uint32_t nmicro;
    uint32_t mlevels;
};

// Shared memory of a tile of `entries` minima (its positions and halo, an
// even number): two buffers of composites, the keys alone padded for 16-byte
// reads past the last one, and the 32-bit half masks.
constexpr uint32_t kKeyPad = 32;
RMQ_HD constexpr uint32_t key_words(uint32_t entries) { return (entries + 3) / 4 * 4 + kKeyPad; }
constexpr size_t table_smem(uint32_t entries) {
    return 2 * sizeof(Entry) * static_cast<size_t>(entries) +
           2 * sizeof(uint32_t) * static_cast<size_t>(key_words(entries));
}

// Masks of the windows of 32 at positions i0 .. i0 + 3 from their keys. Every key
// is read once into registers (9 16-byte reads without bank conflicts); per
// position and distance a compare and two predicated moves. ALU-bound, about
// 100 instructions per micro-block of 32 elements.
__device__ __forceinline__ void mask4(const uint32_t *keys, uint32_t i0, uint32_t (&m)[4]) {
    uint32_t k[36];
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const uint4 f = *reinterpret_cast<const uint4 *>(keys + i0 + 4 * c);
        k[4 * c] = f.x;
        k[4 * c + 1] = f.y;
        k[4 * c + 2] = f.z;
        k[4 * c + 3] = f.w;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        uint32_t run = k[p], bits = 1u;
#pragma unroll
        for (int d = 1; d < 32; ++d)
            if (k[p + d] < run) {
                run = k[p + d];
                bits |= 1u << d;
            }
        m[p] = bits;
    }
}

// Levels k0 .. of one tile in rows of O. `src` holds the best of every window
// of level k0 - 1 that lies in the loaded range; each level writes the other
// buffer, one barrier per level.
template <class O, int THREADS>
__device__ __forceinline__ void tile_rows(const MicroTable &T, uint32_t t0, uint32_t count,
                                          uint32_t e, Entry *src, Entry *dst, uint32_t k0) {
    O *off = static_cast<O *>(T.moff);
    for (uint32_t k = k0; k < T.mlevels && (1u << k) <= e; ++k) {
        const uint32_t half = 1u << (k - 1);
        const uint32_t valid = e - (1u << k) + 1;  // windows inside the loaded range
        O *__restrict__ row = off + static_cast<size_t>(k - k0) * T.nmicro + t0;
        for (uint32_t i = threadIdx.x; i < valid; i += THREADS) {
            const Entry m = better(src[i], src[i + half]);
            dst[i] = m;
            if (i < count && rmq_chk(t0 + i < T.nmicro))
                row[i] = static_cast<O>((entry_idx(m) >> 5) - (t0 + i));
        }
        __syncthreads();
        Entry *t = src;
        src = dst;
        dst = t;
    }
}

// Masks and offset rows at positions [t0, t0 + count) from the minima a[0 ..
// e) of micro-blocks [t0, t0 + e) in shared memory. b: a second buffer of as
// many entries; keys, half: key_words(e) words each, keys[i] the key of a[i]
// and the largest key from e on. The CTA calls it after a barrier; it ends
// with the buffers still in use by other threads.
template <int THREADS>
__device__ __forceinline__ void table_tile(const MicroTable &T, uint32_t t0, uint32_t count,
                                           uint32_t e, Entry *a, Entry *b, const uint32_t *keys,
                                           uint32_t *half) {
    const bool wide = wide_masks(T.nmicro);
    const uint32_t k0 = mask_levels(wide), span = 1u << (k0 - 1u);
    const bool rows = T.mlevels > k0 && e >= 2u * span;
    // the rows' first level needs the best of every mask's window that lies in
    // the loaded range, also past the tile's own positions; a 64-bit mask
    // needs the half mask 32 further on
    const uint32_t npos = rows ? max(count, e - span + 1u) : count;
    const uint32_t nhalf = wide ? min(npos + 32u, e) : npos;
    for (uint32_t i0 = 4u * threadIdx.x; i0 < nhalf; i0 += 4u * THREADS) {
        uint32_t m[4];
        mask4(keys, i0, m);
        *reinterpret_cast<uint4 *>(half + i0) = make_uint4(m[0], m[1], m[2], m[3]);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < npos; i += THREADS) {
        const uint32_t lo = half[i];
        uint32_t d = 31u - __clz(lo);
        const bool mine = i < count && rmq_chk(t0 + i < T.nmicro);
        if (wide) {
            // the second half's new bests (their keys fall strictly) from the
            // first that beats the first half's best on
            uint32_t hi = i + 32u < e ? half[i + 32u] : 0u;
            const uint32_t best = keys[i + d];
            while (hi && keys[i + 31u + __ffs(hi)] >= best) hi &= hi - 1u;
            if (mine) static_cast<uint64_t *>(T.mask)[t0 + i] = (static_cast<uint64_t>(hi) << 32) | lo;
            if (hi) d = 63u - __clz(hi);
        } else if (mine) {
            static_cast<uint32_t *>(T.mask)[t0 + i] = lo;
        }
        if (rows) b[i] = a[min(i + d, e - 1u)];
    }
    if (!rows) return;
    __syncthreads();
    if (T.moff_bytes == 1u)
        tile_rows<uint8_t, THREADS>(T, t0, count, e, b, a, k0);
    else
        tile_rows<uint16_t, THREADS>(T, t0, count, e, b, a, k0);
}

// The keys of a[0 .. e) and the padding behind them.
template <int THREADS>
__device__ __forceinline__ void tile_keys(const Entry *a, uint32_t e, uint32_t *keys) {
    for (uint32_t i = threadIdx.x; i < key_words(e); i += THREADS)
        keys[i] = i < e ? static_cast<uint32_t>(a[i] >> 32) : 0xffffffffu;
}

// A tile whose minima are read from global memory (tile positions [t0, t0 +
// count), smem: table_smem of count + halo rounded up to an even number,
// 16-byte aligned).
template <int THREADS>
__device__ __forceinline__ void table_tile_global(const MicroTable &T, uint32_t t0, uint32_t count,
                                                  unsigned char *smem) {
    const uint32_t e = min(count + table_halo(T.mlevels), T.nmicro - t0);
    const uint32_t cap = (count + table_halo(T.mlevels) + 1u) & ~1u;
    Entry *a = reinterpret_cast<Entry *>(smem);
    Entry *b = a + cap;
    uint32_t *keys = reinterpret_cast<uint32_t *>(b + cap);
    for (uint32_t i = threadIdx.x; i < e; i += THREADS)
        a[i] = rmq_chk(t0 + i < T.nmicro) ? T.mst[t0 + i] : kEntryNone;
    __syncthreads();
    tile_keys<THREADS>(a, e, keys);
    __syncthreads();
    table_tile<THREADS>(T, t0, count, e, a, b, keys, keys + key_words(cap));
    __syncthreads();  // a further tile overwrites the buffers
}

#endif  // __CUDACC__

}  // namespace rmq
