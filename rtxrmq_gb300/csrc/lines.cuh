// lines.cuh -- 32-element lines of values in shared memory: what the query
// kernels (end parts of open queries) and the builders (micro-block minima)
// share. A staged line is 128 bytes whose 16-byte chunks are XOR-swizzled by
// the line's slot, so that 8 lanes writing one line and 32 lanes reading the
// same chunk of 32 lines both go without bank conflicts.
#pragma once

#include "common.cuh"

namespace rmq {

#ifdef __CUDACC__

// What a key mode compares: IEEE minimum / maximum, which skips NaN (ordered
// last) and equates the zeros, or signed minimum / maximum. `fill` stands for
// an element outside the request: it never beats one inside.
template <uint32_t MODE>
struct Best {
    using T = float;
    static __device__ __forceinline__ T of(uint32_t b) { return __uint_as_float(b); }
    static __device__ __forceinline__ uint32_t bits(T x) { return __float_as_uint(x); }
    static __device__ __forceinline__ T fill() { return __uint_as_float(0x7fc00000u); }
    static __device__ __forceinline__ T best(T a, T b) { return MODE == kFloatMin ? fminf(a, b) : fmaxf(a, b); }
};
template <>
struct Best<kIntMin> {
    using T = int32_t;
    static __device__ __forceinline__ T of(uint32_t b) { return static_cast<int32_t>(b); }
    static __device__ __forceinline__ uint32_t bits(T x) { return static_cast<uint32_t>(x); }
    static __device__ __forceinline__ T fill() { return 0x7fffffff; }
    static __device__ __forceinline__ T best(T a, T b) { return min(a, b); }
};
template <>
struct Best<kIntMax> {
    using T = int32_t;
    static __device__ __forceinline__ T of(uint32_t b) { return static_cast<int32_t>(b); }
    static __device__ __forceinline__ uint32_t bits(T x) { return static_cast<uint32_t>(x); }
    static __device__ __forceinline__ T fill() { return -0x7fffffff - 1; }
    static __device__ __forceinline__ T best(T a, T b) { return max(a, b); }
};

// Shared-memory address of chunk 0 of a staged line; chunk c is at ^ (c << 4).
__device__ __forceinline__ uint32_t staged_line(uint32_t stage, uint32_t slot) {
    return stage + slot * 128u + ((slot & 7u) << 4);
}
__device__ __forceinline__ uint4 lds_chunk(uint32_t addr) {
    uint4 f;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(f.x), "=r"(f.y), "=r"(f.z), "=r"(f.w) : "r"(addr));
    return f;
}

// First of the four elements of a chunk that equals `best`, which one of them
// does (or any, when none does: 3), and its bits.
template <uint32_t MODE>
__device__ __forceinline__ uint32_t first_in_chunk(const uint4 &f, typename Best<MODE>::T best,
                                                   uint32_t &bits) {
    using B = Best<MODE>;
    uint32_t pos = 3u;
    bits = f.w;
    if (B::of(f.z) == best) pos = 2u, bits = f.z;
    if (B::of(f.y) == best) pos = 1u, bits = f.y;
    if (B::of(f.x) == best) pos = 0u, bits = f.x;
    return pos;
}

#endif  // __CUDACC__

}  // namespace rmq
