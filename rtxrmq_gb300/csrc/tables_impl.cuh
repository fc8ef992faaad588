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
// entries. What bounds short queries is scattered loads that miss the L1 (its
// requests to the L2 are busy 78% of the time at lr = -3): two of them now (mask,
// minimum) for ranges of up to 1000 (2000) elements, three to four before.
#pragma once

#include "common.cuh"
#include "lines.cuh"
#include "minima_impl.cuh"

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

// One step of a record mask: bit d of `bits` when k beats `run`, which
// becomes the smaller of both. Three instructions; the compiler's form of the
// same takes four to five.
template <int D>
__device__ __forceinline__ void record_step(uint32_t k, uint32_t &run, uint32_t &bits) {
    asm("{\n\t.reg .pred p;\n\t"
        "setp.lt.u32 p, %2, %0;\n\t"
        "min.u32 %0, %0, %2;\n\t"
        "@p or.b32 %1, %1, %3;\n\t}"
        : "+r"(run), "+r"(bits) : "r"(k), "n"(1u << D));
}
template <int D>
__device__ __forceinline__ void record_steps(const uint32_t *k, uint32_t &run, uint32_t &bits) {
    if constexpr (D < 32) {
        record_step<D>(k[D], run, bits);
        record_steps<D + 1>(k, run, bits);
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

// The offset rows of positions [t0, t0 + count) from the masks and minima in
// global memory (written by an earlier launch or phase), for tables with rows
// up to windows of 512 and 1024 (split_rows). smem: two buffers of count +
// halo entries.
template <int THREADS>
__device__ __forceinline__ void rows_tile_global(const MicroTable &T, uint32_t t0, uint32_t count,
                                                 unsigned char *smem) {
    const bool wide = wide_masks(T.nmicro);
    const uint32_t k0 = mask_levels(wide), span = 1u << (k0 - 1u);
    const uint32_t e = min(count + table_halo(T.mlevels), T.nmicro - t0);
    if (e < 2u * span) return;  // no window of the first row starts here
    Entry *a = reinterpret_cast<Entry *>(smem);
    Entry *b = a + ((count + table_halo(T.mlevels) + 1u) & ~1u);
    for (uint32_t i = threadIdx.x; i + span <= e; i += THREADS) {
        const uint32_t j = t0 + i;
        const uint32_t d = wide ? 63u - __clzll(static_cast<const uint64_t *>(T.mask)[j])
                                : 31u - __clz(static_cast<const uint32_t *>(T.mask)[j]);
        if (rmq_chk(j + d < T.nmicro)) b[i] = T.mst[j + d];
    }
    __syncthreads();
    if (T.moff_bytes == 1u)
        tile_rows<uint8_t, THREADS>(T, t0, count, e, b, a, k0);
    else
        tile_rows<uint16_t, THREADS>(T, t0, count, e, b, a, k0);
    __syncthreads();
}

// Whether rows are made apart from the masks: windows of 512 and 1024 reach
// further than the fused builder's ring.
RMQ_HD bool split_rows(uint32_t mlevels) { return mlevels >= 10u; }

// ---- minima and micro table in one pass over the values ---------------------
//
// A CTA takes a run of consecutive micro-blocks, from its right end to its
// left, in units of 256: copies of the next unit's values are in flight while
// the masks of the current one are made, and the minima to its right that its
// windows reach are still in shared memory (a ring of 512 positions, indexed
// by micro-block mod 512) from the unit before. So the values are read once
// plus 63 to 255 micro-blocks per run, and the masks' arithmetic (about 200
// instructions per micro-block) hides behind the stream. As two launches,
// minima and then tables, 10^8 values took 63 + 38 us.
constexpr uint32_t kUnit = 256;         // micro-blocks per unit = threads
constexpr uint32_t kRing = 512;
constexpr uint32_t kMirror = 64;        // ring positions 0 .. 63 again behind its end
struct TableSmem {
    uint4 stage[kUnit * 8];             // the unit's values, 4 KB per warp
    Entry a[kRing + kMirror];           // minima
    Entry c[kRing];                     // best of the whole mask's window
    uint32_t key[kRing + kMirror];
    uint32_t half[kRing + kMirror];     // masks of windows of 32, 0 past the array
    Entry warp[kUnit / 32];             // each warp's best
};

// Whether the run also reduces its blocks' minima: blocks of pb micro-blocks
// tile a unit. (Read again from the micro-block minima, they cost the ragged
// benchmark 0.44 GB and a grid barrier.)
RMQ_HD bool fused_blocks(uint32_t pb) { return pb <= kUnit && (pb & (pb - 1u)) == 0u; }

// Micro-blocks [lo, hi) (multiples of kUnit, or hi the array's last) of the
// array whose element 0 is value `base`; the CTA of kUnit threads. With `T`'s
// rows only when they are not split, the block minima only when they are fused.
template <bool ALIGNED, uint32_t MODE>
__device__ __forceinline__ void build_run(const float *__restrict__ A, int64_t limit, int64_t base,
                                          uint32_t n, uint32_t lead, Entry *mst, const MicroTable &T,
                                          uint32_t lo, uint32_t hi, Entry *bmin, uint32_t pb,
                                          TableSmem &sm) {
    const uint32_t t = threadIdx.x, warp = t >> 5;
    const uint32_t stage = static_cast<uint32_t>(__cvta_generic_to_shared(sm.stage)) + 4096u * warp;
    const bool wide = wide_masks(T.nmicro);
    const uint32_t k0 = mask_levels(wide), span = 1u << (k0 - 1u);
    const bool rows = T.mlevels > k0 && !split_rows(T.mlevels);
    const uint32_t reach = rows ? (1u << (T.mlevels - 1u)) - 1u : 63u;
    const bool blocks = fused_blocks(pb);
    LineStep step;
    auto issue = [&](uint32_t s, uint32_t cnt) {
        const uint32_t w0 = 32u * warp;
        step = LineStep{base, n, lead, s + w0, cnt > w0 ? min(kStepLines, cnt - w0) : 0u, mst};
        if (step.cnt) copy_step<ALIGNED>(A, limit, step, stage);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // first what lies right of the run (no output), then its units
    uint32_t s = hi, cnt = min(reach, T.nmicro - hi);
    bool out = false;
    issue(s, cnt);
    for (uint32_t i = t; i < kRing + kMirror; i += kUnit) {
        sm.a[i] = kEntryNone;
        sm.key[i] = 0xffffffffu;
        sm.half[i] = 0u;
        if (i < kRing) sm.c[i] = kEntryNone;
    }
    for (;;) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const Entry m = reduce_step<MODE>(step, stage);
        const uint32_t j = s + t, r = j & (kRing - 1u);
        const bool have = t < cnt;
        __syncthreads();  // the slots written next were the last unit's right neighbours
        if (have) {
            const uint32_t key = static_cast<uint32_t>(m >> 32);
            sm.a[r] = m;
            sm.key[r] = key;
            if (r < kMirror) {
                sm.a[r + kRing] = m;
                sm.key[r + kRing] = key;
            }
            if (out && rmq_chk(j < T.nmicro)) mst[j] = m;
        }
        if (blocks) {
            // the best of min(pb, 32) lanes; of more, the warps' bests below
            Entry best = have ? m : kEntryNone;
            if (pb >= 32u) {
                const uint32_t k = __reduce_min_sync(0xffffffffu, static_cast<uint32_t>(best >> 32));
                const uint32_t l = __reduce_min_sync(
                    0xffffffffu, static_cast<uint32_t>(best >> 32) == k ? static_cast<uint32_t>(best) : 0xffffffffu);
                if ((t & 31u) == 0u) sm.warp[warp] = (static_cast<uint64_t>(k) << 32) | l;
            } else {
                for (uint32_t o = pb >> 1; o > 0u; o >>= 1) best = better(best, __shfl_xor_sync(0xffffffffu, best, o));
                if (out && have && (t & (pb - 1u)) == 0u) bmin[j / pb] = best;
            }
        }
        __syncthreads();
        if (blocks && out && pb >= 32u && t < kUnit / pb && t * pb < cnt) {
            Entry best = sm.warp[t * (pb / 32u)];
            for (uint32_t i = 1; i < pb / 32u; ++i) best = better(best, sm.warp[t * (pb / 32u) + i]);
            bmin[s / pb + t] = best;
        }
        const uint32_t next = out ? s - kUnit : (hi - 1u) / kUnit * kUnit;
        const bool more = out ? s > lo : true;
        if (more) issue(next, min(hi - next, kUnit));

        uint32_t bits = 1u;
        {
            uint32_t run = sm.key[r];
            const uint32_t *k = sm.key + r;
            record_steps<1>(k, run, bits);
        }
        if (have) {
            sm.half[r] = bits;
            if (r < kMirror) sm.half[r + kRing] = bits;
        }
        __syncthreads();
        uint32_t d = 31u - __clz(bits);
        uint32_t top = 0u;
        if (wide) {
            // the second half's new bests (their keys fall strictly) from the
            // first that beats the first half's best on: none when its last
            // does not, else by bisection (a loop over the bests to drop costs
            // a warp its longest one, twice as much)
            top = sm.half[r + 32u];
            const uint32_t best = sm.key[r + d];
            const uint32_t *k2 = sm.key + r + 32u;
            if (top != 0u && k2[31u - __clz(top)] >= best) top = 0u;
            uint32_t from = 0u;
#pragma unroll
            for (uint32_t w = 16u; w > 0u; w >>= 1) {
                const uint32_t sub = (top >> from) & ((1u << w) - 1u);
                if (sub == 0u || k2[from + 31u - __clz(sub)] >= best) from += w;
            }
            top &= 0xffffffffu << from;
            if (top) d = 63u - __clz(top);
        }
        const bool store = out && have && rmq_chk(j < T.nmicro);
        if (store) {
            if (wide)
                static_cast<uint64_t *>(T.mask)[j] = (static_cast<uint64_t>(top) << 32) | bits;
            else
                static_cast<uint32_t *>(T.mask)[j] = bits;
        }
        if (rows) {
            if (have) sm.c[r] = sm.a[r + d];
            __syncthreads();
            if (store) {
                Entry acc = sm.c[r];
                for (uint32_t k = k0; k < T.mlevels; ++k) {
                    const uint32_t parts = 1u << (k - k0);
                    for (uint32_t i = parts; i < 2u * parts; ++i)
                        acc = better(acc, sm.c[(r + i * span) & (kRing - 1u)]);
                    if (j + (1u << k) <= T.nmicro) {
                        const size_t at = static_cast<size_t>(k - k0) * T.nmicro + j;
                        const uint32_t off = (entry_idx(acc) >> 5) - j;
                        if (T.moff_bytes == 1u)
                            static_cast<uint8_t *>(T.moff)[at] = static_cast<uint8_t>(off);
                        else
                            static_cast<uint16_t *>(T.moff)[at] = static_cast<uint16_t>(off);
                    }
                }
            }
        }
        if (!more) break;
        s = next;
        cnt = min(hi - next, kUnit);
        out = true;
    }
    __syncthreads();  // a further run clears the ring
}

// Minima of blocks [b0, b1) of `pb` micro-blocks each, from the micro-block
// minima: a thread per block for small blocks, a warp per block otherwise.
template <int THREADS>
__device__ __forceinline__ void block_minima(const Entry *mst, uint32_t nmicro, uint32_t pb,
                                             uint32_t b0, uint32_t b1, uint32_t nb, Entry *bmin) {
    if (pb <= 16u) {
        for (uint32_t b = b0 + threadIdx.x; b < b1; b += THREADS) {
            Entry m = kEntryNone;
            const uint32_t j1 = min(b * pb + pb, nmicro);
            for (uint32_t j = b * pb; j < j1; ++j) m = better(m, mst[j]);
            if (rmq_chk(b < nb)) bmin[b] = m;
        }
        return;
    }
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t b = b0 + (threadIdx.x >> 5); b < b1; b += THREADS / 32) {
        Entry m = kEntryNone;
        const uint32_t j1 = min(b * pb + pb, nmicro);
        for (uint32_t j = b * pb + lane; j < j1; j += 32u) m = better(m, mst[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = better(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0u && rmq_chk(b < nb)) bmin[b] = m;
    }
}

// Levels k0 + 1 .. k0 + g (g <= kLevelGroup) of a block table st[levels][nb]
// at positions [first, first + count), from level k0 (`src`): a level's entry is
// the best of 2^g entries of level k0, 2^k0 apart, so several levels need no
// synchronisation between them. The last one also goes to `top`, if any.
// COARSE: a second table C is written as well, and windows that reach past the
// last block are entries too, of what there is.
constexpr uint32_t kLevelGroup = 3;

// A second block table st[levels][nb] over blocks 2^shift times as large: row
// k holds every 2^shift-th entry of row k + shift.
struct CoarseTable {
    Entry *st = nullptr;
    uint32_t nb = 0, levels = 0, shift = 1;
};
template <int THREADS, bool COARSE = false>
__device__ __forceinline__ void level_group(const Entry *src, Entry *st, uint32_t nb, uint32_t k0,
                                            uint32_t g, uint32_t first, uint32_t count, Entry *top,
                                            uint32_t levels = 0u, const CoarseTable C = CoarseTable()) {
    for (uint32_t j = first + threadIdx.x; j < first + count; j += THREADS) {
        Entry x[1 << kLevelGroup];
#pragma unroll
        for (uint32_t i = 0; i < (1u << kLevelGroup); ++i) {
            const uint64_t at = j + (static_cast<uint64_t>(i) << k0);
            x[i] = i < (1u << g) && at < nb ? src[at] : kEntryNone;
        }
#pragma unroll
        for (uint32_t t = 1; t <= kLevelGroup; ++t) {
#pragma unroll
            for (uint32_t i = 0; i < (1u << (kLevelGroup - t)); ++i)
                x[i] = better(x[2 * i], x[2 * i + 1]);
            if constexpr (COARSE) {
                if (t <= g && k0 + t < levels) st[static_cast<size_t>(k0 + t) * nb + j] = x[0];
                const uint32_t c = k0 + t - C.shift;  // wraps below its levels
                if (t <= g && c < C.levels && (j & ((1u << C.shift) - 1u)) == 0u)
                    C.st[static_cast<size_t>(c) * C.nb + (j >> C.shift)] = x[0];
            } else if (t <= g && j + (1ull << (k0 + t)) <= nb) {
                st[static_cast<size_t>(k0 + t) * nb + j] = x[0];
                if (top && t == g) top[j] = x[0];
            }
        }
    }
}

// Every level of a block table st[levels][nb] from its block minima, by one
// CTA: a group of levels per step between two buffers of nb entries in shared
// memory (nb = 3052, 12 levels: 11 us with a step per level).
template <int THREADS>
__device__ __forceinline__ void all_levels(Entry *st, uint32_t nb, uint32_t levels, Entry *buf) {
    Entry *src = buf, *dst = buf + nb;
    for (uint32_t i = threadIdx.x; i < nb; i += THREADS) src[i] = st[i];
    __syncthreads();
    for (uint32_t k = 0; k + 1u < levels; k += kLevelGroup) {
        level_group<THREADS>(src, st, nb, k, min(kLevelGroup, levels - 1u - k), 0u, nb, dst);
        __syncthreads();
        Entry *t = src;
        src = dst;
        dst = t;
    }
    __syncthreads();  // a further table overwrites the buffers
}

#endif  // __CUDACC__

}  // namespace rmq
