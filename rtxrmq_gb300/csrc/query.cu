// query.cu -- plain query kernels.
//
// query_kernel: one CTA answers 256 * QPT consecutive queries at a time with
// the queued body of query_impl.cuh (RTX_blocks' three-ray decomposition,
// src/rtx_kernels.cu:85-193 and 350-465, needed only for the queries a
// probe of the small tables over a superset of [l, r] does not settle).
// Queries and outputs may live in device memory or in pinned host memory
// mapped into the device address space: on a Grace-Blackwell node the kernel
// then streams them over NVLink-C2C while its random lookups hit HBM.
//
// scan_kernel is the GPU brute force of alg 2 / 102
// (src/cuda_methods.cuh:3-66): one thread per query, strict `<` from A[l].
#include "query_kernel.cuh"

namespace rmq {
namespace {

// Random-access ceiling of the un-pruned query on this index
// (rmq_probe_gather): query_kernel's grid, query stream and output stores,
// but per query only the two random 8-byte lookups suf[l] and pre[r] (no
// block decision, no table probe, no scan). Its answers are not range minima.
__global__ void __launch_bounds__(kThreads)
gather_kernel(V1View v, QueryOut o, int64_t q) {
    const int64_t chunk = static_cast<int64_t>(kThreads) * kQPT;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * chunk;
    for (int64_t c0 = static_cast<int64_t>(blockIdx.x) * chunk; c0 < q; c0 += stride) {
        int2 qq[kQPT];
        load_queries<kQPT>(o, c0, c0 + chunk < q ? c0 + chunk : q, qq);
        Entry e[kQPT];
#pragma unroll
        for (int k = 0; k < kQPT; ++k) {
            // clamped into the array: the probe never reads out of bounds
            const uint32_t l = min(static_cast<uint32_t>(max(qq[k].x, 0)), v.n - 1u);
            const uint32_t r = min(static_cast<uint32_t>(max(qq[k].y, 0)), v.n - 1u);
            e[k] = better(v.suf[l], v.pre[r]);
        }
#pragma unroll
        for (int k = 0; k < kQPT; ++k) {
            const int64_t i = c0 + threadIdx.x + static_cast<int64_t>(k) * kThreads;
            if (i < q) put_result(o, i, e[k], v.kmode);
        }
    }
}

// 64-bit finaliser of SplitMix64 (Steele, Lea, Flood, OOPSLA 2014).
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// Random-access rate of this GPU, independent of any index layout
// (rmq_probe_random): query_kernel's grid, query stream and output stores,
// and per query two 8-byte loads at positions hashed from (i, l, r),
// uniform over buf[0 .. words).
__global__ void __launch_bounds__(kThreads)
random_gather_kernel(const unsigned long long *__restrict__ buf, uint64_t words, QueryOut o,
                     int64_t q) {
    const int64_t chunk = static_cast<int64_t>(kThreads) * kQPT;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * chunk;
    for (int64_t c0 = static_cast<int64_t>(blockIdx.x) * chunk; c0 < q; c0 += stride) {
        int2 qq[kQPT];
        load_queries<kQPT>(o, c0, c0 + chunk < q ? c0 + chunk : q, qq);
        Entry e[kQPT];
#pragma unroll
        for (int k = 0; k < kQPT; ++k) {
            const int64_t i = c0 + threadIdx.x + static_cast<int64_t>(k) * kThreads;
            const uint64_t h1 = mix64((static_cast<uint64_t>(i) << 32) ^ static_cast<uint32_t>(qq[k].x));
            const uint64_t h2 = mix64(h1 ^ static_cast<uint32_t>(qq[k].y));
            const uint64_t p1 = __umul64hi(h1, words), p2 = __umul64hi(h2, words);
            e[k] = better(__ldg(buf + p1), __ldg(buf + p2));
        }
#pragma unroll
        for (int k = 0; k < kQPT; ++k) {
            const int64_t i = c0 + threadIdx.x + static_cast<int64_t>(k) * kThreads;
            if (i < q) put_bits_idx(o, i, static_cast<uint32_t>(e[k] >> 32), static_cast<uint32_t>(e[k]));
        }
    }
}

__global__ void __launch_bounds__(kThreads)
scan_kernel(const float *__restrict__ A, uint32_t n, QueryOut o, int64_t q) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kThreads;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; i < q;
         i += stride) {
        const int2 qq = o.Q[i];
        if (qq.x < 0 || qq.x > qq.y || static_cast<uint32_t>(qq.y) >= n) {
            put_invalid(o, i);
            continue;
        }
        float m = A[qq.x];
        uint32_t mi = static_cast<uint32_t>(qq.x);
        for (uint32_t j = static_cast<uint32_t>(qq.x); j <= static_cast<uint32_t>(qq.y); ++j) {
            const float x = A[j];
            if (x < m) {
                m = x;
                mi = j;
            }
        }
        put_bits_idx(o, i, __float_as_uint(m), mi);
    }
}

std::atomic<int> g_gather_per_sm{0};
std::atomic<int> g_random_per_sm{0};
std::atomic<int> g_scan_per_sm{0};

}  // namespace

V1View view_of(const BuildPlan &p) {
    V1View v;
    v.A = p.A;
    v.off = p.off;
    v.limit = p.limit;
    v.n = p.n;
    v.lead = p.lead;
    v.bs = p.tbs;
    v.nb = p.nb;
    v.dv = make_div31(p.tbs);
    v.st = p.st;
    v.cst = p.cst;
    v.cnb = p.cnb;
    v.clevels = p.clevels;
    v.cdiv = p.cbs ? make_div31(p.cbs).m : 0u;
    v.coarse_from = p.cbs ? kCoarseFrom * (p.cbs / kMicro) : 0xffffffffu;
    v.mst = p.mst;
    v.mask = p.mask;
    v.wide = wide_masks(p.nmicro);
    v.moff = p.moff;
    v.moff_bytes = p.moff_bytes;
    v.nmicro = p.nmicro;
    v.pre = p.pre;
    v.suf = p.suf;
    v.kmode = p.kmode;
    v.levels = p.levels;
    v.mlevels = p.mlevels;
    v.micro_span = p.micro_span;
    v.light = p.light;
    return v;
}

template <bool STATS>
cudaError_t launch_query_s(const BuildPlan &p, const V1View &v, const QueryOut &o, int64_t q,
                           unsigned long long *stats, const DeviceInfo &dev, cudaStream_t s) {
    if (p.aligned)
        return p.micro ? launch_query_m<true, true, STATS, false>(v, o, q, stats, dev, s)
                       : launch_query_m<true, false, STATS, false>(v, o, q, stats, dev, s);
    return p.micro ? launch_query_m<false, true, STATS, false>(v, o, q, stats, dev, s)
                   : launch_query_m<false, false, STATS, false>(v, o, q, stats, dev, s);
}

// Arrays with a lead (query_lead.cu).
cudaError_t launch_query_lead(const BuildPlan &p, const V1View &v, const QueryOut &o, int64_t q,
                              const DeviceInfo &dev, cudaStream_t s);

// Results in host memory (query_host.cu).
cudaError_t launch_query_host(const BuildPlan &p, const V1View &v, const QueryOut &o, int64_t q,
                              const DeviceInfo &dev, cudaStream_t s);

cudaError_t launch_query(const BuildPlan &p, const QueryArgs &a, const DeviceInfo &dev,
                         cudaStream_t s) {
    if (a.q <= 0) return cudaSuccess;
    const V1View v = view_of(p);
    QueryOut o;
    o.Q = a.Q;
    o.val = a.val;
    o.idx = a.idx;
    o.invalid = a.invalid;
    o.span = a.q;
    if (p.lead != 0u) return launch_query_lead(p, v, o, a.q, dev, s);
    if (a.host && p.micro) return launch_query_host(p, v, o, a.q, dev, s);
    if (a.stats) return launch_query_s<true>(p, v, o, a.q, a.stats, dev, s);
    return launch_query_s<false>(p, v, o, a.q, nullptr, dev, s);
}

cudaError_t launch_probe_random(const unsigned long long *buf, uint64_t words, const QueryArgs &a,
                                const DeviceInfo &dev, cudaStream_t s) {
    if (a.q <= 0) return cudaSuccess;
    QueryOut o;
    o.Q = a.Q;
    o.val = a.val;
    o.idx = a.idx;
    o.invalid = nullptr;
    o.span = a.q;
    int per_sm;
    cudaError_t err = occupancy(random_gather_kernel, &g_random_per_sm, &per_sm);
    if (err != cudaSuccess) return err;
    random_gather_kernel<<<grid_size(a.q, kThreads * kQPT, per_sm, dev), kThreads, 0, s>>>(
        buf, words, o, a.q);
    return cudaGetLastError();
}

cudaError_t launch_probe_gather(const BuildPlan &p, const QueryArgs &a, const DeviceInfo &dev,
                                cudaStream_t s) {
    if (a.q <= 0) return cudaSuccess;
    const V1View v = view_of(p);
    QueryOut o;
    o.Q = a.Q;
    o.val = a.val;
    o.idx = a.idx;
    o.invalid = nullptr;
    o.span = a.q;
    int per_sm;
    cudaError_t err = occupancy(gather_kernel, &g_gather_per_sm, &per_sm);
    if (err != cudaSuccess) return err;
    gather_kernel<<<grid_size(a.q, kThreads * kQPT, per_sm, dev), kThreads, 0, s>>>(v, o, a.q);
    return cudaGetLastError();
}

cudaError_t launch_query_scan(const float *A, uint32_t n, const QueryArgs &a,
                              const DeviceInfo &dev, cudaStream_t s) {
    if (a.q <= 0) return cudaSuccess;
    int per_sm;
    cudaError_t err = occupancy(scan_kernel, &g_scan_per_sm, &per_sm);
    if (err != cudaSuccess) return err;
    QueryOut o;
    o.Q = a.Q;
    o.val = a.val;
    o.idx = a.idx;
    o.invalid = a.invalid;
    o.span = a.q;
    scan_kernel<<<grid_size(a.q, kThreads, per_sm, dev), kThreads, 0, s>>>(A, n, o, a.q);
    return cudaGetLastError();
}

RMQ_VIOLATIONS_READER(violations_query)

}  // namespace rmq
