// query_kernel.cuh -- the plain query kernel and its launch, instantiated by
// query.cu (plain indexes), query_lead.cu (arrays of a batch that start off a
// 128-byte boundary) and query_host.cu (results in host memory).
#pragma once

#include "engine.h"
#include "query_impl.cuh"

namespace rmq {
namespace {

constexpr int kThreads = 256;
#ifndef RMQ_QUERY_QPT
#define RMQ_QUERY_QPT 2  // queries per thread per step (independent lookups in flight)
#endif
constexpr int kQPT = RMQ_QUERY_QPT;
#ifndef RMQ_QUERY_MINB
#define RMQ_QUERY_MINB 4  // CTAs per SM the query kernel is compiled for (a register bound)
#endif

// Queries base + t + k * kThreads (k < kQPT) of a full step, no bounds checks.
__device__ __forceinline__ void load_full(const QueryOut &o, int64_t base, int2 (&qq)[kQPT]) {
    const int2 *Qs = o.Q + base;
#pragma unroll
    for (int k = 0; k < kQPT; ++k) qq[k] = __ldcs(Qs + threadIdx.x + k * kThreads);
}

// Grid-stride over steps of 256 * kQPT queries (answer_step_queued); the
// next step's queries are loaded before the current step is answered, so
// their latency (host memory over the host link when called through
// rmq_query_host) overlaps the current step's lookups. Specialised on the
// key mode and on whether the index has the sub-block level. STATS: the
// measurement instantiation (rmq_query_stats), which also counts how each
// query was settled and what it read into stats[kStatCount]. WHOLE: results in
// host memory (answer_step_queued).
template <bool ALIGNED, bool MICRO, uint32_t MODE, bool STATS, bool LEAD, bool WHOLE>
__global__ void __launch_bounds__(kThreads, RMQ_QUERY_MINB)
query_kernel(V1View v, QueryOut o, int64_t q, unsigned long long *stats) {
    __shared__ __align__(128) MissQueue<MICRO, WHOLE> s_mq[kThreads / 32];
    constexpr int64_t chunk = static_cast<int64_t>(kThreads) * kQPT;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * chunk;
    int64_t c0 = static_cast<int64_t>(blockIdx.x) * chunk;
    if (c0 >= q) return;
    const int64_t last_full = q - chunk;  // steps starting at or before it are full
    QStats s;
    if constexpr (STATS)
        for (int c = 0; c < kStatCount; ++c) s.c[c] = 0u;
    MissQueue<MICRO, WHOLE> &mq = s_mq[threadIdx.x >> 5];
    uint32_t waiting = 0;  // the warp's queue length (warp-uniform)
    int2 cur[kQPT];
    if (c0 <= last_full)
        load_full(o, c0, cur);
    else
        load_queries<kQPT>(o, c0, q, cur);
    const StepMap map{c0, stride};
    for (uint32_t id0 = 0; c0 < q; c0 += stride, id0 += static_cast<uint32_t>(chunk)) {
        const int64_t c1 = c0 + stride;
        int2 nxt[kQPT];
        if (c1 <= last_full)
            load_full(o, c1, nxt);
        else if (c1 < q)
            load_queries<kQPT>(o, c1, q, nxt);
        answer_step_queued<ALIGNED, MICRO, MODE, kThreads, kQPT, STATS, LEAD, true, WHOLE>(
            v, o, map, c0, static_cast<uint32_t>(min(chunk, q - c0)), id0, c1 >= q, cur, s, mq, waiting);
#pragma unroll
        for (int k = 0; k < kQPT; ++k) cur[k] = nxt[k];
    }
    if constexpr (STATS) flush_stats(s, stats);
}

template <typename K>
cudaError_t occupancy(K kernel, std::atomic<int> *cache, int *per_sm) {
    const cudaError_t err = occupancy_cached(kernel, kThreads, *cache, *per_sm);
    if (*per_sm < 1) *per_sm = 1;
    return err;
}

// `bytes` of shared memory per SM (the runtime's 1 KB per CTA included) as a
// percentage of the largest carve-out, 228 KB. Rounded down: a hint above one
// of the supported sizes takes the next one.
int carveout_percent(size_t bytes) { return static_cast<int>(bytes * 100 / (228 * 1024)); }

uint32_t grid_size(int64_t q, int64_t per_block, int per_sm, const DeviceInfo &dev) {
    const int64_t need = (q + per_block - 1) / per_block;
    const int64_t cap = static_cast<int64_t>(dev.sms) * per_sm;
    return static_cast<uint32_t>(need < cap ? need : cap);
}

template <bool ALIGNED, bool MICRO, uint32_t MODE, bool STATS, bool LEAD, bool WHOLE>
cudaError_t launch_query_t(const V1View &v, const QueryOut &o, int64_t q,
                           unsigned long long *stats, const DeviceInfo &dev, cudaStream_t s) {
    static std::atomic<int> per_sm_cache[kMaxDevices] = {};  // the carve-out is set per device
    auto kern = query_kernel<ALIGNED, MICRO, MODE, STATS, LEAD, WHOLE>;
    int per_sm = per_sm_cache[dev.device].load(std::memory_order_relaxed);
    if (per_sm == 0) {
        cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, 0);
        if (err != cudaSuccess) return err;
        if (per_sm < 1) per_sm = 1;
        // Shared memory no larger than the resident CTAs' queues need: the
        // rest stays L1, where the block table's upper levels hit. The
        // default split gives 100 KB for the 41 KB used (lr=-2, bs 4096,
        // n = 1e8: 0.52 ms, with this 0.48).
        err = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   carveout_percent(per_sm * (sizeof(MissQueue<MICRO, WHOLE>) * (kThreads / 32) + 1024)));
        if (err != cudaSuccess) return err;
        per_sm_cache[dev.device].store(per_sm, std::memory_order_relaxed);
    }
    kern<<<grid_size(q, kThreads * kQPT, per_sm, dev), kThreads, 0, s>>>(v, o, q, stats);
    return cudaGetLastError();
}

template <bool ALIGNED, bool MICRO, bool STATS, bool LEAD, bool WHOLE = false>
cudaError_t launch_query_m(const V1View &v, const QueryOut &o, int64_t q,
                           unsigned long long *stats, const DeviceInfo &dev, cudaStream_t s) {
    switch (v.kmode) {
    case kFloatMax: return launch_query_t<ALIGNED, MICRO, kFloatMax, STATS, LEAD, WHOLE>(v, o, q, stats, dev, s);
    case kIntMin: return launch_query_t<ALIGNED, MICRO, kIntMin, STATS, LEAD, WHOLE>(v, o, q, stats, dev, s);
    case kIntMax: return launch_query_t<ALIGNED, MICRO, kIntMax, STATS, LEAD, WHOLE>(v, o, q, stats, dev, s);
    default: return launch_query_t<ALIGNED, MICRO, kFloatMin, STATS, LEAD, WHOLE>(v, o, q, stats, dev, s);
    }
}

}  // namespace
}  // namespace rmq
