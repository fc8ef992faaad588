// batch_impl.cuh -- the persistent batch kernel, instantiated by batch.cu
// (16-byte aligned values) and batch_unaligned.cu.
//
// Persistent kernel, phases separated by grid-wide barriers of a cooperative
// launch (all CTAs are co-resident, guaranteed by the launch):
//   A  run items (array, first unit, units): micro-block minima and micro
//      table, the plain builder's CTA body (build_run, tables_impl.cuh);
//   B  table items (array, kind | level, first, count), one step per barrier:
//      the block minima and the rows not made in the runs at step 1, the block
//      table's levels after them;
//   C  query items (array, first query, count), query_impl.cuh's queued form.
// Work lists are built on the host once per plan, so a run allocates nothing
// and can be captured in a CUDA graph. A launch of phase C alone needs no
// barrier: it is an ordinary launch of a kernel of its own.
//
// Launches of one plan may overlap, at their ends, when they are on different
// streams. So a launch shares no state with the next but the index: the two
// counters from which a building launch's CTAs take items are its own (a pair
// out of kCounterPairs), and a query launch has none.
//
// An array is built from the 128-byte boundary (32 values) at or before its
// first element on: its micro-blocks are whole 128-byte lines whatever its
// offset, so rows stored back to back take 16-byte copies too.
#pragma once

#include <cooperative_groups.h>

#include "engine.h"
#include "query_impl.cuh"
#include "tables_impl.cuh"

// CTAs per SM the persistent batch kernel is compiled for (a register bound).
#ifndef RMQ_BATCH_MINB
#define RMQ_BATCH_MINB 4
#endif

namespace rmq {

constexpr int kBatchThreads = kUnit;  // phase A runs the table builder
constexpr int kBatchQPT = 2;
// default tile schedule: queries per query item (at most, see kRunUnits), table
// entries per level item (a plan can set both per size bucket,
// rmq_batch_create_ex)
constexpr uint32_t kQueryChunk = 4096;
constexpr uint32_t kLevelChunk = 4096;
constexpr int kMaxSteps = 16;
// units (of 256 micro-blocks) per run item, at most: 1 MB of values, so that
// the 63 to 255 micro-blocks a run reads beyond its end stay below a few
// percent (ragged benchmark's build: 1.25 ms with 8 units, 1.20 with 16, 1.18
// with 32; with 64 1.17, but a few arrays of 2e7 leave SMs idle: 0.14 and 0.23
// ms). Fewer where a plan has not that many for every CTA, and the same for
// the queries of an item where the tile does not set them (29 arrays of up to
// 2.6e5 values, 26 thousand queries: 101 us with the most, 43 so; 100 of up to
// 1e6, 1 million queries: 160 and 66).
constexpr uint32_t kRunUnits = 32;
constexpr uint32_t kLeastQueryChunk = 512;  // one step of a CTA
constexpr int32_t kMostQueryChunk = 1 << 29;
// positions per item of rows made apart, and the largest block table that one
// item takes through all its levels: both fit the run's shared memory
constexpr uint32_t kBatchRowTile = 1024;
constexpr uint32_t kOneItemTable = 2048;

// kinds of table items (bits 16.. of the item's second word; bits 0..15 hold
// the level)
enum : uint32_t {
    kItemBlockMinima = 0,  // block minima from the micro-block minima
    kItemRows = 1,         // offset rows (split_rows)
    kItemTable = 2,        // every level of a small block table
    kItemLevels = 3,       // levels k + 1 .. k + kLevelGroup of a larger one
};

struct BatchArray {
    int64_t off;    // the 128-byte boundary its index starts at (values)
    int64_t qoff;   // first query
    int64_t st;     // workspace entry offset of the block table
    int64_t mst;    // ... of the micro-block minima
    int64_t mask;   // ... of the micro table's masks
    int64_t moff;   // ... of its offset rows
    uint32_t n;     // elements from off on
    uint32_t lead;  // of which the first `lead` are not the array's
    uint32_t bs, nb, levels;
    uint32_t nmicro, mlevels, moff_bytes;
    Div31 dv;
};

struct BatchParams {
    const float *A;
    int64_t limit;
    const int2 *Q;
    float *val;
    int32_t *idx;
    unsigned long long *invalid;
    Entry *ws;
    const BatchArray *arrays;
    const uint4 *runs;
    int32_t nruns;
    const uint4 *tables;
    int32_t steps;        // table steps run: 1 .. steps - 1
    int32_t step_start[kMaxSteps + 1];
    const uint4 *qitems;
    int32_t nqitems;
    int64_t total_q;      // one past the last query any array owns
    uint32_t *next;       // the launch's work counters: runs, query items (0 when it starts)
    bool queries;         // batch_kernel: phase C too
};

// Pairs of work counters of a plan: launches take them in turn, captured ones
// from a half of their own. A building launch fills the GPU and its CTAs wait for
// one another, so no more than two can overlap. Captured launches keep their
// pair for every replay.
constexpr uint32_t kCounterPairs = 64;

// Dynamic shared memory of a CTA: the run's buffers in phase A, buffers of
// two halves in phase B, the warps' miss queues in phase C.
constexpr size_t kBatchSmem = sizeof(TableSmem);
static_assert(kBatchSmem <= kDefaultSmem, "no attribute needed");
static_assert(2 * sizeof(Entry) * (kBatchRowTile + 1024) <= kBatchSmem, "row tiles fit");
static_assert(2 * sizeof(Entry) * kOneItemTable <= kBatchSmem, "small tables fit");
static_assert(sizeof(MissQueue<true>) * (kBatchThreads / 32) <= kBatchSmem, "miss queues fit");

// The instantiation for (aligned, key mode): of batch_kernel and its CTAs per SM,
// or without `build` of batch_query_kernel.
cudaError_t batch_kernel_aligned(uint32_t mode, bool build, const void **fn, int *per_sm);
cudaError_t batch_kernel_unaligned(uint32_t mode, bool build, const void **fn, int *per_sm);

namespace {

namespace cg = cooperative_groups;

template <uint32_t MODE>
__device__ __forceinline__ V1View batch_view(const BatchParams &P, const BatchArray &a) {
    V1View v;
    v.A = P.A;
    v.off = a.off;
    v.limit = P.limit;
    v.n = a.n;
    v.lead = a.lead;
    v.bs = a.bs;
    v.nb = a.nb;
    v.dv = a.dv;
    v.st = P.ws + a.st;
    v.coarse_from = 0xffffffffu;
    v.mst = P.ws + a.mst;
    v.mask = P.ws + a.mask;
    v.wide = wide_masks(a.nmicro);
    v.moff = P.ws + a.moff;
    v.moff_bytes = a.moff_bytes;
    v.nmicro = a.nmicro;
    v.pre = nullptr;
    v.suf = nullptr;
    v.kmode = MODE;
    v.levels = a.levels;
    v.mlevels = a.mlevels;
    v.micro_span = (1u << a.mlevels) - 1u;
    v.light = true;
    return v;
}

__device__ __forceinline__ MicroTable batch_table(const BatchParams &P, const BatchArray &a) {
    MicroTable T;
    T.mst = P.ws + a.mst;
    T.mask = P.ws + a.mask;
    T.moff = P.ws + a.moff;
    T.moff_bytes = a.moff_bytes;
    T.nmicro = a.nmicro;
    T.mlevels = a.mlevels;
    return T;
}

// The next item of a work list for this CTA: items go to CTAs as they come
// free (their costs differ by more than ten times). Called by the whole CTA;
// a barrier on either side of the shared word.
__device__ __forceinline__ int32_t next_item(uint32_t *counter, int32_t *s_item) {
    __syncthreads();
    if (threadIdx.x == 0) *s_item = static_cast<int32_t>(atomicAdd(counter, 1u));
    __syncthreads();
    return *s_item;
}

// Phase B: table steps 1 .. steps - 1, a grid barrier after each.
__device__ __forceinline__ void table_steps(const BatchParams &P, cg::grid_group &grid,
                                            unsigned char *smem) {
    for (int s = 1; s < P.steps; ++s) {
        for (int32_t it = P.step_start[s] + blockIdx.x; it < P.step_start[s + 1]; it += gridDim.x) {
            const uint4 w = P.tables[it];
            const BatchArray &a = P.arrays[w.x];
            const uint32_t kind = w.y >> 16, k = w.y & 0xffffu;
            Entry *st = P.ws + a.st;
            if (kind == kItemBlockMinima)
                block_minima<kBatchThreads>(P.ws + a.mst, a.nmicro, a.bs / 32u, w.z, w.z + w.w, a.nb, st);
            else if (kind == kItemRows)
                rows_tile_global<kBatchThreads>(batch_table(P, a), w.z, w.w, smem);
            else if (kind == kItemTable)
                all_levels<kBatchThreads>(st, a.nb, a.levels, reinterpret_cast<Entry *>(smem));
            else
                level_group<kBatchThreads>(st + static_cast<size_t>(k) * a.nb, st, a.nb, k,
                                           min(kLevelGroup, a.levels - 1u - k), w.z, w.w, nullptr);
        }
        grid.sync();
    }
}

// Phase C, one query item by the CTA, in the queued form.
template <bool ALIGNED, uint32_t MODE>
__device__ __forceinline__ void query_item(const BatchParams &P, int32_t it, MissQueue<true> &mq) {
    const uint4 w = P.qitems[it];
    const BatchArray a = P.arrays[w.x];
    const V1View v = batch_view<MODE>(P, a);
    QueryOut o;
    o.Q = P.Q + a.qoff;
    o.val = P.val ? P.val + a.qoff : nullptr;
    o.idx = P.idx ? P.idx + a.qoff : nullptr;
    o.invalid = P.invalid;
    o.span = P.total_q - a.qoff;
    answer_range_queued<ALIGNED, true, MODE, true, kBatchThreads, kBatchQPT>(
        v, o, w.y, static_cast<int64_t>(w.y) + w.z, mq);
}

template <bool ALIGNED, uint32_t MODE>
__global__ void __launch_bounds__(kBatchThreads, RMQ_BATCH_MINB) batch_kernel(BatchParams P) {
    extern __shared__ __align__(1024) unsigned char s_batch[];
    __shared__ int32_t s_item;
    cg::grid_group grid = cg::this_grid();
    // each counter is cleared in the phase that does not use it
    if (blockIdx.x == 0 && threadIdx.x == 0) P.next[1] = 0u;
    for (int32_t it; (it = next_item(P.next, &s_item)) < P.nruns;) {
        const uint4 w = P.runs[it];
        const BatchArray &a = P.arrays[w.x];
        const uint32_t lo = w.y * kUnit;
        build_run<ALIGNED, MODE>(P.A, P.limit, a.off, a.n, a.lead, P.ws + a.mst, batch_table(P, a), lo,
                                 min(lo + w.z * kUnit, a.nmicro), P.ws + a.st, a.bs / 32u,
                                 *reinterpret_cast<TableSmem *>(s_batch));
    }
    grid.sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) P.next[0] = 0u;
    table_steps(P, grid, s_batch);
    MissQueue<true> &mq = reinterpret_cast<MissQueue<true> *>(s_batch)[threadIdx.x >> 5];
    for (int32_t it; P.queries && (it = next_item(P.next + 1, &s_item)) < P.nqitems;)
        query_item<ALIGNED, MODE>(P, it, mq);
}

// Phase C alone (rmq_batch_query): a CTA per item.
template <bool ALIGNED, uint32_t MODE>
__global__ void __launch_bounds__(kBatchThreads, RMQ_BATCH_MINB) batch_query_kernel(BatchParams P) {
    __shared__ __align__(1024) MissQueue<true> s_mq[kBatchThreads / 32];
    query_item<ALIGNED, MODE>(P, static_cast<int32_t>(blockIdx.x), s_mq[threadIdx.x >> 5]);
}

std::atomic<int> g_batch_per_sm[4];  // per key mode, of this unit's alignment

template <bool ALIGNED, uint32_t MODE>
cudaError_t pick_batch(bool build, const void **fn, int *per_sm) {
    if (!build) {
        *fn = reinterpret_cast<const void *>(batch_query_kernel<ALIGNED, MODE>);
        return cudaSuccess;
    }
    auto kern = batch_kernel<ALIGNED, MODE>;
    *fn = reinterpret_cast<const void *>(kern);
    return occupancy_cached(kern, kBatchThreads, g_batch_per_sm[MODE], *per_sm, kBatchSmem);
}

template <bool ALIGNED>
cudaError_t batch_kernel_t(uint32_t mode, bool build, const void **fn, int *per_sm) {
    switch (mode) {
    case kFloatMax: return pick_batch<ALIGNED, kFloatMax>(build, fn, per_sm);
    case kIntMin: return pick_batch<ALIGNED, kIntMin>(build, fn, per_sm);
    case kIntMax: return pick_batch<ALIGNED, kIntMax>(build, fn, per_sm);
    default: return pick_batch<ALIGNED, kFloatMin>(build, fn, per_sm);
    }
}

}  // namespace
}  // namespace rmq
