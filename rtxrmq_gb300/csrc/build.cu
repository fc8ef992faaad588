// build.cu -- construction of the block-decomposition index for one array.
//
// The reference builds, for RTX_blocks, one triangle per element plus one
// per block minimum and hands them to the OptiX BVH builder
// (src/device_tools.cuh:139-169, 243-253, src/rtx.h:3-22, 39-99). GB300 has
// no RT cores, so the search structure is rebuilt as arrays a query indexes
// directly: in-block prefix / suffix minima (build_impl.cuh) and a sparse
// table over the block minima:
//   st[k][j] = leftmost minimum of blocks j .. j + 2^k - 1 (k = 0: block minima)
#include "build_impl.cuh"
#include "engine.h"
#include "tables_impl.cuh"

// CTAs per SM the unit kernel is compiled for (a register bound).
#ifndef RMQ_BUILD_MINB
#define RMQ_BUILD_MINB 4
#endif

namespace rmq {
namespace {

template <bool ALIGNED, uint32_t MODE>
__global__ void __launch_bounds__(kBuildThreads, RMQ_BUILD_MINB)
build_units_kernel(UnitJob J, uint32_t nunits) {
    __shared__ Entry stage[kStageEntries];
    __shared__ uint64_t s_warp[kWarpSlots];
    __shared__ uint32_t s_flag[2 * kBuildWarps];
    for (uint32_t u = blockIdx.x; u < nunits; u += gridDim.x)
        build_unit<ALIGNED, MODE>(J, u, stage, s_warp, s_flag);
}

template <bool ALIGNED>
void launch_units(const UnitJob &J, uint32_t nunits, uint32_t grid, cudaStream_t s) {
    switch (J.kmode) {
    case kFloatMax: build_units_kernel<ALIGNED, kFloatMax><<<grid, kBuildThreads, 0, s>>>(J, nunits); break;
    case kIntMin: build_units_kernel<ALIGNED, kIntMin><<<grid, kBuildThreads, 0, s>>>(J, nunits); break;
    case kIntMax: build_units_kernel<ALIGNED, kIntMax><<<grid, kBuildThreads, 0, s>>>(J, nunits); break;
    default: build_units_kernel<ALIGNED, kFloatMin><<<grid, kBuildThreads, 0, s>>>(J, nunits); break;
    }
}

__global__ void st_level_kernel(Entry *st, uint32_t nb, uint32_t k) {
    const Entry *prev = st + static_cast<size_t>(k - 1) * nb;
    Entry *cur = st + static_cast<size_t>(k) * nb;
    const uint32_t half = 1u << (k - 1);
    const uint32_t cnt = nb - (1u << k) + 1;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < cnt;
         j += gridDim.x * blockDim.x)
        if (rmq_chk(j + half < nb)) cur[j] = better(prev[j], prev[j + half]);
}

constexpr int kTableThreads = 256;

// The micro table (masks and offset rows) from the micro-block minima, one
// tile of consecutive positions per CTA.
__global__ void __launch_bounds__(kTableThreads)
table_kernel(MicroTable T, uint32_t tile) {
    extern __shared__ __align__(16) unsigned char s_tile[];
    const uint32_t t0 = blockIdx.x * tile;
    table_tile_global<kTableThreads>(T, t0, min(tile, T.nmicro - t0), s_tile);
}

// One pass over the values: the minimum of every 32-element
// micro-block (level 0 of the micro table) and, folded in with a 64-bit
// atomic minimum, of every block (level 0 of the block table, filled with
// all-ones before; bs a multiple of 32, so every micro-block lies in one
// block). A warp takes 16 consecutive micro-blocks per step: four 512-byte
// rows, each lane 4 consecutive elements of every row, all four loads in
// flight before any reduction; 8 lanes reduce one micro-block. When the 16
// micro-blocks lie in one block (bs a multiple of 512, or away from block
// edges) the warp folds them into that block with a single atomic.

template <uint32_t MODE>
__global__ void __launch_bounds__(256)
micro_min_kernel(const float *__restrict__ A, uint32_t n, uint32_t nmicro, uint32_t per_block,
                 Entry *mst0, Entry *bmin, bool aligned) {
    static_assert(kMicroElems == kMicro, "micro-block size");
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t sub = lane & 7u;
    const uint32_t grp = lane >> 3;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t nblocks = (nmicro + per_block - 1) / per_block;
    for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
         w * kMicroPerWarp < nmicro; w += warps) {
        const uint32_t j0 = w * kMicroPerWarp;
        Entry m[4];  // micro-block j0 + 4i + grp, on all 8 lanes of the group
        if (aligned && (j0 + kMicroPerWarp) * kMicro <= n)
            micro_min_warp<MODE, true>(A, n, j0, nmicro, mst0, 0u, m);
        else
            micro_min_warp<MODE, false>(A, n, j0, nmicro, mst0, 0u, m);
        const uint32_t jl = min(j0 + kMicroPerWarp, nmicro) - 1u;
        if (j0 / per_block == jl / per_block) {
            // one block: micro-blocks past nmicro hold kEntryNone, the identity
            Entry v = better(better(m[0], m[1]), better(m[2], m[3]));
            v = better(v, __shfl_xor_sync(0xffffffffu, v, 8));
            v = better(v, __shfl_xor_sync(0xffffffffu, v, 16));
            const uint32_t blk = j0 / per_block;
            if (lane == 0u && rmq_chk(blk < nblocks))
                atomicMin(reinterpret_cast<unsigned long long *>(bmin + blk),
                          static_cast<unsigned long long>(v));
        } else if (sub == 0u) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t j = j0 + 4u * i + grp;
                const uint32_t blk = j / per_block;
                if (j < nmicro && rmq_chk(blk < nblocks))
                    atomicMin(reinterpret_cast<unsigned long long *>(bmin + blk),
                              static_cast<unsigned long long>(m[i]));
            }
        }
    }
}

std::atomic<int> g_units_per_sm[2];

cudaError_t launch_levels(Entry *st, uint32_t nb, uint32_t levels, const DeviceInfo &dev,
                          cudaStream_t s) {
    for (uint32_t k = 1; k < levels; ++k) {
        const uint32_t cnt = nb - (1u << k) + 1;
        uint32_t g = (cnt + 255) / 256;
        const uint32_t cap = static_cast<uint32_t>(dev.sms) * 8u;
        if (g > cap) g = cap;
        st_level_kernel<<<g, 256, 0, s>>>(st, nb, k);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

// Positions per table tile: 1024, 2048 where the halo is about as long (rows
// up to level 9 and 10), 256 while a tile per SM is not to be had.
uint32_t table_tile_size(const BuildPlan &p, const DeviceInfo &dev) {
    if (p.mlevels >= 10) return 2048u;
    return p.nmicro >= 1024u * static_cast<uint32_t>(dev.sms) ? 1024u : 256u;
}

cudaError_t launch_table(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s) {
    MicroTable T;
    T.mst = p.mst;
    T.mask = p.mask;
    T.moff = p.moff;
    T.moff_bytes = p.moff_bytes;
    T.nmicro = p.nmicro;
    T.mlevels = p.mlevels;
    const uint32_t tile = table_tile_size(p, dev);
    const size_t smem = table_smem((tile + table_halo(p.mlevels) + 1u) & ~1u);
    static std::atomic<bool> ready{false};
    if (!ready.load(std::memory_order_relaxed)) {
        // the largest tile: 2048 positions and a halo of 1023
        const cudaError_t err = cudaFuncSetAttribute(
            table_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
            static_cast<int>(table_smem(2048u + 1024u)));
        if (err != cudaSuccess) return err;
        ready.store(true, std::memory_order_relaxed);
    }
    table_kernel<<<(p.nmicro + tile - 1) / tile, kTableThreads, smem, s>>>(T, tile);
    return cudaGetLastError();
}

}  // namespace

uint32_t st_levels(uint32_t nb) { return nb ? static_cast<uint32_t>(ilog2(nb)) + 1u : 0u; }

namespace {
size_t a256(size_t x) { return (x + 255) / 256 * 256; }
struct Offsets {
    size_t pre, suf, st, mst, mask, moff, counter, total;
};
Offsets offsets_of(const BuildPlan &p) {
    Offsets o;
    const size_t nent = p.micro ? 0 : a256(sizeof(Entry) * static_cast<size_t>(p.n));
    o.pre = 0;
    o.suf = nent;
    o.st = 2 * nent;
    o.mst = o.st + a256(sizeof(Entry) * static_cast<size_t>(p.nb) * p.levels);
    o.mask = o.mst + a256(sizeof(Entry) * static_cast<size_t>(p.nmicro));
    o.moff = o.mask + a256((wide_masks(p.nmicro) ? 8 : 4) * static_cast<size_t>(p.nmicro));
    o.counter = o.moff + a256(static_cast<size_t>(p.moff_bytes) * p.nmicro * moff_rows(p.mlevels, wide_masks(p.nmicro)));
    o.total = o.counter + 256;
    return o;
}
}  // namespace

size_t plan_index(BuildPlan &p, bool no_micro) {
    p.micro = !no_micro;
    p.tbs = p.micro ? table_block(p.bs) : p.bs;
    p.nb = (p.n + p.tbs - 1) / p.tbs;
    p.levels = st_levels(p.nb);
    p.mlevels = p.micro ? micro_levels(p.tbs) : 0u;
    p.nmicro = p.micro ? (p.n + kMicro - 1) / kMicro : 0u;
    p.moff_bytes = p.micro ? micro_offset_bytes(p.mlevels) : 0u;
    p.aligned = reinterpret_cast<uintptr_t>(p.A) % 16 == 0;
    return offsets_of(p).total;
}

unsigned long long *place_index(BuildPlan &p, void *base_v) {
    char *base = static_cast<char *>(base_v);
    const Offsets o = offsets_of(p);
    p.pre = p.micro ? nullptr : reinterpret_cast<Entry *>(base + o.pre);
    p.suf = p.micro ? nullptr : reinterpret_cast<Entry *>(base + o.suf);
    p.st = reinterpret_cast<Entry *>(base + o.st);
    p.mst = p.micro ? reinterpret_cast<Entry *>(base + o.mst) : nullptr;
    p.mask = p.micro ? static_cast<void *>(base + o.mask) : nullptr;
    p.moff = p.micro ? static_cast<void *>(base + o.moff) : nullptr;
    return reinterpret_cast<unsigned long long *>(base + o.counter);
}

size_t layout_v5(uint32_t n, uint32_t bs, bool light, bool no_micro, LayoutV5 *out) {
    out->nb = (n + bs - 1) / bs;
    out->levels = st_levels(out->nb);
    out->mlevels = no_micro ? 0u : micro_levels(bs);
    out->nmicro = out->mlevels ? (n + kMicro - 1) / kMicro : 0u;
    const size_t nent = light ? 0 : a256(sizeof(Entry) * static_cast<size_t>(n));
    size_t total = 2 * nent + a256(sizeof(Entry) * static_cast<size_t>(out->nb) * out->levels) + 256;
    if (out->mlevels)
        total += a256(sizeof(Entry) * static_cast<size_t>(out->nmicro)) + 2 * nent +
                 a256(static_cast<size_t>(micro_offset_bytes(out->mlevels)) * out->nmicro *
                      (out->mlevels - 1));
    return total;
}

// The micro table works on 32-element micro-blocks aligned in the array,
// whatever the block size. A query first probes it over every micro-block it
// touches (a superset of [l, r]; two windows of 2^k micro-blocks cover up to
// 2^(k+1) - 1 of them), so it holds windows long enough for any query inside
// one block: a block touches bs/32 micro-blocks when blocks start on
// micro-block boundaries (bs a multiple of 32, as in every table index), at
// most floor((bs + 30) / 32) + 1 otherwise.
uint32_t micro_levels(uint32_t bs) {
    if (bs < 2 * kMicro) return 0;
    const uint32_t touched = (bs % kMicro == 0) ? bs / kMicro : (bs + kMicro - 2) / kMicro + 1;
    return st_levels(touched);
}

static cudaError_t launch_build_tables(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s) {
    cudaError_t err = cudaMemsetAsync(p.st, 0xff, sizeof(Entry) * static_cast<size_t>(p.nb), s);
    if (err != cudaSuccess) return err;
    // 8 warps per CTA, kMicroPerWarp micro-blocks per warp step
    uint32_t g = (p.nmicro + 8 * kMicroPerWarp - 1) / (8 * kMicroPerWarp);
    const uint32_t cap = static_cast<uint32_t>(dev.sms) * 8u;
    if (g > cap) g = cap;
    const uint32_t per_block = p.tbs / kMicro;
    switch (p.kmode) {
    case kFloatMax:
        micro_min_kernel<kFloatMax><<<g, 256, 0, s>>>(p.A, p.n, p.nmicro, per_block, p.mst, p.st,
                                                      p.aligned);
        break;
    case kIntMin:
        micro_min_kernel<kIntMin><<<g, 256, 0, s>>>(p.A, p.n, p.nmicro, per_block, p.mst, p.st,
                                                    p.aligned);
        break;
    case kIntMax:
        micro_min_kernel<kIntMax><<<g, 256, 0, s>>>(p.A, p.n, p.nmicro, per_block, p.mst, p.st,
                                                    p.aligned);
        break;
    default:
        micro_min_kernel<kFloatMin><<<g, 256, 0, s>>>(p.A, p.n, p.nmicro, per_block, p.mst, p.st,
                                                      p.aligned);
        break;
    }
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    err = launch_levels(p.st, p.nb, p.levels, dev, s);
    if (err != cudaSuccess) return err;
    return launch_table(p, dev, s);
}

cudaError_t launch_build_entries(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s) {
    UnitJob J;
    J.A = p.A;
    J.off = 0;
    J.limit = p.n;
    J.n = p.n;
    J.bs = p.bs;
    const uint32_t nb = (p.n + p.bs - 1) / p.bs;
    J.U = make_unit_layout(p.bs, nb);
    J.dv = make_div31(p.bs);
    J.pre = p.pre;
    J.suf = p.suf;
    J.bmin = p.st;
    J.kmode = p.kmode;
    J.nb = nb;
    const uint32_t nunits = unit_count(nb, J.U);

    // every key mode compiles to the same resources; the float-min
    // instantiation stands for all four
    int per_sm;
    cudaError_t err =
        p.aligned ? occupancy_cached(build_units_kernel<true, kFloatMin>, kBuildThreads,
                                     g_units_per_sm[1], per_sm)
                  : occupancy_cached(build_units_kernel<false, kFloatMin>, kBuildThreads,
                                     g_units_per_sm[0], per_sm);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    uint32_t grid = static_cast<uint32_t>(dev.sms) * static_cast<uint32_t>(per_sm);
    if (grid > nunits) grid = nunits;
    if (p.aligned)
        launch_units<true>(J, nunits, grid, s);
    else
        launch_units<false>(J, nunits, grid, s);
    return cudaGetLastError();
}

cudaError_t launch_build(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s) {
    if (p.n == 0) return cudaSuccess;
    if (p.micro) return launch_build_tables(p, dev, s);
    const cudaError_t err = launch_build_entries(p, dev, s);
    if (err != cudaSuccess) return err;
    return launch_levels(p.st, p.nb, p.levels, dev, s);
}

RMQ_VIOLATIONS_READER(violations_build)

}  // namespace rmq
