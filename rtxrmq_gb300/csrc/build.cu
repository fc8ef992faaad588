// build.cu -- construction of the block-decomposition index for one array.
//
// The reference builds, for RTX_blocks, one triangle per element plus one
// per block minimum and hands them to the OptiX BVH builder
// (src/device_tools.cuh:139-169, 243-253, src/rtx.h:3-22, 39-99). GB300 has
// no RT cores, so the search structure is rebuilt as arrays a query indexes
// directly: micro-block minima and the micro table over them
// (tables_impl.cuh) and sparse tables over block minima:
//   st[k][j] = leftmost minimum of blocks j .. j + 2^k - 1 (k = 0: block minima)
// Without the sub-block level: in-block prefix / suffix minima per element
// (build_impl.cuh) and one sparse table.
#include "build_impl.cuh"
#include "engine.h"
#include "minima_impl.cuh"
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

// Micro-block minima and the micro table (build_run): a run of `units` units
// of micro-blocks per CTA.
#ifndef RMQ_TABLE_MINB
#define RMQ_TABLE_MINB 4
#endif
template <bool ALIGNED, uint32_t MODE>
__global__ void __launch_bounds__(kUnit, RMQ_TABLE_MINB)
table_kernel(const float *__restrict__ A, int64_t limit, int64_t base, uint32_t n, uint32_t lead,
             Entry *mst, MicroTable T, uint32_t units, Entry *bmin, uint32_t pb) {
    extern __shared__ __align__(1024) unsigned char s_table[];
    const uint32_t lo = blockIdx.x * units * kUnit;
    build_run<ALIGNED, MODE>(A, limit, base, n, lead, mst, T, lo, min(lo + units * kUnit, T.nmicro),
                             bmin, pb, *reinterpret_cast<TableSmem *>(s_table));
}

// Tables in blocks of bs (arrays of a batch, rmq_query_stats; an index's own
// blocks leave nothing): what the runs left out, from the micro-block minima, the offset
// rows of split_rows, one tile of kRowTile positions per CTA, and in the CTAs
// before them the block minima of blocks that do not tile a unit, a thread
// per block of up to 16 micro-blocks, else a warp. One launch: the block
// minima are few and slow (n = 1e8, bs 2^15: 11 us beside the rows' 26).
constexpr uint32_t kRowTile = 2048;
constexpr int kRestThreads = 512;
__global__ void __launch_bounds__(kRestThreads)
rest_kernel(MicroTable T, uint32_t pb, Entry *bmin, uint32_t nb, uint32_t per_cta, uint32_t block_ctas) {
    extern __shared__ __align__(16) unsigned char s_tile[];
    if (blockIdx.x < block_ctas) {
        const uint32_t b0 = blockIdx.x * per_cta;
        block_minima<kRestThreads>(T.mst, T.nmicro, pb, b0, min(b0 + per_cta, nb), nb, bmin);
    } else {
        const uint32_t t0 = (blockIdx.x - block_ctas) * kRowTile;
        rows_tile_global<kRestThreads>(T, t0, min(kRowTile, T.nmicro - t0), s_tile);
    }
}

constexpr int kLevelThreads = 1024;
constexpr uint32_t kSmallTable = 4096;
__global__ void __launch_bounds__(kLevelThreads)
small_levels_kernel(Entry *st, uint32_t nb, uint32_t levels) {
    extern __shared__ Entry s_level[];
    all_levels<kLevelThreads>(st, nb, levels, s_level);
}

// Levels k0 + 1 .. k0 + g of a larger block table, and of the table C of larger
// blocks.
template <bool COARSE>
__global__ void __launch_bounds__(256)
level_group_kernel(Entry *st, uint32_t nb, uint32_t levels, uint32_t k0, uint32_t g, CoarseTable C) {
    const uint32_t first = blockIdx.x * 256u;
    level_group<256, COARSE>(st + static_cast<size_t>(k0) * nb, st, nb, k0, g, first,
                             min(256u, nb - first), nullptr, levels, C);
}

std::atomic<int> g_units_per_sm[2];

cudaError_t launch_levels(Entry *st, uint32_t nb, uint32_t levels, const CoarseTable &C, cudaStream_t s) {
    if (levels <= 1) return cudaSuccess;
    if (nb <= kSmallTable && !C.st) {
        const size_t smem = 2 * sizeof(Entry) * nb;
        if (smem > kDefaultSmem) {
            // belongs to the current device, so it is set at each launch (0.2 us)
            const cudaError_t err = cudaFuncSetAttribute(
                small_levels_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (err != cudaSuccess) return err;
        }
        small_levels_kernel<<<1, kLevelThreads, smem, s>>>(st, nb, levels);
        return cudaGetLastError();
    }
    const uint32_t all = C.st && C.levels + C.shift > levels ? C.levels + C.shift : levels;
    for (uint32_t k = 0; k + 1 < all; k += kLevelGroup) {
        const uint32_t g = all - 1 - k < kLevelGroup ? all - 1 - k : kLevelGroup;
        if (C.st)
            level_group_kernel<true><<<(nb + 255) / 256, 256, 0, s>>>(st, nb, levels, k, g, C);
        else
            level_group_kernel<false><<<(nb + 255) / 256, 256, 0, s>>>(st, nb, levels, k, g, C);
        const cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

template <bool ALIGNED, uint32_t MODE>
cudaError_t launch_runs_t(const BuildPlan &p, const MicroTable &T, const DeviceInfo &dev,
                          cudaStream_t s) {
    static std::atomic<int> per_sm_cache{0};
    auto kern = table_kernel<ALIGNED, MODE>;
    static_assert(sizeof(TableSmem) <= kDefaultSmem, "no attribute needed");
    int per_sm;
    const cudaError_t err = occupancy_cached(kern, kUnit, per_sm_cache, per_sm, sizeof(TableSmem));
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    const uint32_t cap = static_cast<uint32_t>(dev.sms) * static_cast<uint32_t>(per_sm);
    const uint32_t all = (p.nmicro + kUnit - 1) / kUnit, units = (all + cap - 1) / cap;
    kern<<<(all + units - 1) / units, kUnit, sizeof(TableSmem), s>>>(
        p.A, p.limit, p.off, p.n, p.lead, p.mst, T, units, p.st, p.tbs / kMicro);
    return cudaGetLastError();
}

template <bool ALIGNED>
cudaError_t launch_runs(const BuildPlan &p, const MicroTable &T, const DeviceInfo &dev,
                        cudaStream_t s) {
    switch (p.kmode) {
    case kFloatMax: return launch_runs_t<ALIGNED, kFloatMax>(p, T, dev, s);
    case kIntMin: return launch_runs_t<ALIGNED, kIntMin>(p, T, dev, s);
    case kIntMax: return launch_runs_t<ALIGNED, kIntMax>(p, T, dev, s);
    default: return launch_runs_t<ALIGNED, kFloatMin>(p, T, dev, s);
    }
}

cudaError_t launch_build_tables(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s) {
    MicroTable T;
    T.mst = p.mst;
    T.mask = p.mask;
    T.moff = p.moff;
    T.moff_bytes = p.moff_bytes;
    T.nmicro = p.nmicro;
    T.mlevels = p.mlevels;
    cudaError_t err = p.aligned ? launch_runs<true>(p, T, dev, s) : launch_runs<false>(p, T, dev, s);
    if (err != cudaSuccess) return err;
    const uint32_t pb = p.tbs / kMicro;
    const uint32_t per_cta = pb <= 16u ? kRestThreads : kRestThreads / 32;
    const uint32_t block_ctas = fused_blocks(pb) ? 0u : (p.nb + per_cta - 1) / per_cta;
    const uint32_t row_ctas = split_rows(p.mlevels) ? (p.nmicro + kRowTile - 1) / kRowTile : 0u;
    if (block_ctas + row_ctas > 0u) {
        const size_t smem = row_ctas ? 2 * sizeof(Entry) * ((kRowTile + table_halo(p.mlevels) + 1u) & ~1u) : 0;
        // the longest halo: 1023
        static_assert(2 * sizeof(Entry) * (kRowTile + 1024u) <= kDefaultSmem, "no attribute needed");
        rest_kernel<<<block_ctas + row_ctas, kRestThreads, smem, s>>>(T, pb, p.st, p.nb, per_cta, block_ctas);
        err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    CoarseTable C;
    if (p.cbs) C = CoarseTable{p.cst, p.cnb, p.clevels, static_cast<uint32_t>(ilog2(p.cbs / p.tbs))};
    return launch_levels(p.st, p.nb, p.levels, C, s);
}

}  // namespace

namespace {
size_t a256(size_t x) { return (x + 255) / 256 * 256; }
struct Offsets {
    size_t pre, suf, st, cst, mst, mask, moff, counter, total;
};
Offsets offsets_of(const BuildPlan &p) {
    Offsets o;
    const size_t nent = p.micro ? 0 : a256(sizeof(Entry) * static_cast<size_t>(p.n));
    o.pre = 0;
    o.suf = nent;
    o.st = 2 * nent;
    o.cst = o.st + a256(sizeof(Entry) * static_cast<size_t>(p.nb) * p.levels);
    o.mst = o.cst + a256(sizeof(Entry) * static_cast<size_t>(p.cnb) * p.clevels);
    o.mask = o.mst + a256(sizeof(Entry) * static_cast<size_t>(p.nmicro));
    o.moff = o.mask + a256((wide_masks(p.nmicro) ? 8 : 4) * static_cast<size_t>(p.nmicro));
    o.counter = o.moff + a256(static_cast<size_t>(p.moff_bytes) * p.nmicro * moff_rows(p.mlevels, wide_masks(p.nmicro)));
    o.total = o.counter + 256;
    return o;
}
}  // namespace

size_t plan_index(BuildPlan &p, bool no_micro, bool asked) {
    p.off = 0;
    p.limit = p.n;
    p.lead = 0;
    p.micro = !no_micro;
    IndexShape shape = index_shape(p.n);
    if (asked) {
        const TableShape t = table_shape(p.n, p.bs);
        shape = IndexShape{t.tbs, t.mlevels, (1u << t.mlevels) - 1u, 0u};
    }
    p.tbs = p.micro ? shape.tbs : p.bs;
    p.nb = (p.n + p.tbs - 1) / p.tbs;
    p.levels = st_levels(p.nb);
    p.cbs = p.micro ? shape.cbs : 0u;
    p.cnb = p.cbs ? (p.n + p.cbs - 1) / p.cbs : 0u;
    p.clevels = st_levels(p.cnb);
    p.mlevels = p.micro ? shape.mlevels : 0u;
    p.micro_span = p.micro ? shape.micro_span : 0u;
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
    p.cst = p.cbs ? reinterpret_cast<Entry *>(base + o.cst) : nullptr;
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
    return launch_levels(p.st, p.nb, p.levels, CoarseTable(), s);
}

RMQ_VIOLATIONS_READER(violations_build)

}  // namespace rmq
