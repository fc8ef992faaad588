// minima_impl.cuh -- the minimum of every 32-element micro-block, the one pass
// over the values that a table index needs.
//
// A warp takes 32 consecutive micro-blocks (4 KB) per step: it copies them
// into its own shared memory (cp.async, 16 bytes per lane, coalesced) and
// then every lane reduces one whole line. No exchange between lanes and no
// barrier: about 75 instructions per line, where 8 lanes per micro-block with
// shuffles took about 300, and the bytes in flight do not sit in registers.
// Bound by HBM.
#pragma once

#include "common.cuh"
#include "lines.cuh"

namespace rmq {

// Micro-blocks of one warp step.
constexpr uint32_t kStepLines = 32;

#ifdef __CUDACC__

// One warp step: micro-blocks j0 .. j0 + cnt - 1 (cnt <= 32) of the array
// whose element 0 is value `base` of the buffer, n elements of which the
// first `lead` do not count.
struct LineStep {
    int64_t base;
    uint32_t n, lead;
    uint32_t j0, cnt;
    Entry *mst;
};

// Starts copying a step's lines; nothing past value limit - 1 is read.
// ALIGNED: base is a 16-byte boundary (element base of a 16-byte aligned
// buffer, base a multiple of 4).
template <bool ALIGNED>
__device__ __forceinline__ void copy_step(const float *__restrict__ A, int64_t limit,
                                          const LineStep &s, uint32_t stage) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, grp = lane >> 3;
    const int64_t g0 = s.base + static_cast<int64_t>(s.j0) * 32;
    if (ALIGNED) {
        const uint32_t d0 = staged_line(stage, grp) ^ (sub << 4);
        const uint32_t d1 = staged_line(stage, 4u + grp) ^ (sub << 4);
        const float *src = A + g0 + 4 * lane;
        if (s.cnt == kStepLines && g0 + 32 * static_cast<int64_t>(kStepLines) <= limit) {
#pragma unroll
            for (uint32_t t = 0; t < kStepLines / 4; ++t)
                if (rmq_chk(g0 >= 0))
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                 :: "r"(((t & 1u) ? d1 : d0) + (t / 2u) * 1024u), "l"(src + 128 * t) : "memory");
        } else {
#pragma unroll 1
            for (uint32_t t = 0; 4u * t < s.cnt; ++t) {
                const int64_t room = limit - (g0 + 4 * lane + 128 * static_cast<int64_t>(t));
                if (4u * t + grp < s.cnt && room > 0) {
                    const uint32_t bytes = room >= 4 ? 16u : 4u * static_cast<uint32_t>(room);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                 :: "r"(((t & 1u) ? d1 : d0) + (t / 2u) * 1024u), "l"(src + 128 * t), "r"(bytes) : "memory");
                }
            }
        }
    } else {
#pragma unroll 4
        for (uint32_t r = 0; r < s.cnt; ++r) {
            const int64_t g = g0 + 32 * static_cast<int64_t>(r) + lane;
            const uint32_t dst = (staged_line(stage, r) ^ ((lane >> 2) << 4)) + 4u * (lane & 3u);
            if (g < limit && rmq_chk(g >= 0))
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst), "l"(A + g) : "memory");
        }
    }
}

// The minimum of line `lane` of a staged step.
template <uint32_t MODE>
__device__ __forceinline__ Entry reduce_step(const LineStep &s, uint32_t stage) {
    using B = Best<MODE>;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t base = staged_line(stage, lane);
    const uint32_t j = s.j0 + lane;
    const uint32_t first = j == 0u ? s.lead : 0u;
    // elements before the array's first and past its last one become the
    // fill, which never beats an element (rare: an array's end lines)
    if (lane < s.cnt && (first != 0u || 32u * j + 32u > s.n)) {
        const uint32_t valid = s.n - 32u * j;
        for (uint32_t e = 0; e < 32u; ++e)
            if (e < first || e >= valid)
                asm volatile("st.shared.u32 [%0], %1;"
                             :: "r"((base ^ ((e >> 2) << 4)) + 4u * (e & 3u)), "r"(B::bits(B::fill())) : "memory");
    }
    typename B::T m[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const uint4 f = lds_chunk(base ^ (c << 4));
        m[c] = B::best(B::best(B::best(B::of(f.x), B::of(f.y)), B::of(f.z)), B::of(f.w));
    }
    const typename B::T mm = B::best(B::best(B::best(m[0], m[1]), B::best(m[2], m[3])),
                                     B::best(B::best(m[4], m[5]), B::best(m[6], m[7])));
    uint32_t cs = 7u;
#pragma unroll
    for (int c = 6; c >= 0; --c) cs = m[c] == mm ? c : cs;
    uint32_t wb;
    const uint32_t pos = first_in_chunk<MODE>(lds_chunk(base ^ (cs << 4)), mm, wb);
    // no number, or nothing above the fill: every element has the largest
    // key, and the first of them is the best
    const bool last = !(mm == mm) || mm == B::fill();
    const uint32_t key = last ? 0xffffffffu : key_of(wb, MODE);
    const uint32_t lo = ((32u * j + (last ? first : 4u * cs + pos)) << 1) | (last ? 0u : negzero_of(wb, MODE));
    return (static_cast<uint64_t>(key) << 32) | lo;
}

#endif  // __CUDACC__

}  // namespace rmq
