// engine.h -- internal interface between the C ABI (api.cu) and the kernel
// translation units. Nothing here is exported.
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <cstdint>
#include <cuda_runtime.h>

#include <nvtx3/nvToolsExt.h>

#include "common.cuh"
#include "tables_impl.cuh"

namespace rmq {

// Records a message for rmq_last_error_string() and returns `code`.
int set_error(int code, const char *fmt, ...);
// Converts a CUDA error into RMQ_ECUDA (RMQ_ENOMEM for an allocation
// failure) with the call site in the message.
int cuda_fail(cudaError_t err, const char *what);

// Device properties the launchers need, cached per device.
struct DeviceInfo {
    int device;
    int sms;
    size_t l2_bytes;
};
int device_info(DeviceInfo *out);

// NVTX range over one C-ABI call (named after it), visible to profilers
// and tracers; nearly free when none is attached.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// Every device allocation of the library goes through here. Memory that the
// pool below keeps counts as free: when there is no other, it is given back
// and the allocation tried again. Fault injection for tests: with
// RTXRMQ_FAIL_ALLOC=1 in the environment it fails as an out-of-memory would,
// without touching the device.
cudaError_t dev_malloc(void **p, size_t bytes);

// Id of the calling thread's current context, 0 when there is none or the
// driver cannot tell.
unsigned long long current_context_id();

// Device memory of an index, in stream order: from a pool of the library (one
// per device and context) that keeps at most kPoolKeep bytes of freed memory;
// the rest goes back to the device at the next synchronisation, all of it by
// pool_trim(). *pool_context is the context whose pool it came from. Larger
// requests, and requests while `s` is capturing, take cudaMalloc (0). cudaMalloc
// + cudaFree cost 0.2 ms a call, cudaFree waits for the device: a build + query
// of 10^5 values took 0.24 ms.
constexpr size_t kPoolKeep = size_t(256) << 20;
cudaError_t pool_malloc(void **p, size_t bytes, int device, cudaStream_t s,
                        unsigned long long *pool_context);
cudaError_t pool_trim(int device);

// Dynamic shared memory that a launch may ask for without
// cudaFuncAttributeMaxDynamicSharedMemorySize. Function attributes belong to a
// device: what one device was told does not hold on the next.
constexpr size_t kDefaultSmem = 48 * 1024;
constexpr int kMaxDevices = 64;  // device_info refuses higher ordinals

// Resident CTAs per SM of `kernel` at `threads` threads and `dynamic_smem`
// bytes of dynamic shared memory, computed once per cache slot; concurrent
// first callers compute and store the same value.
template <class K>
cudaError_t occupancy_cached(K kernel, int threads, std::atomic<int> &cache, int &per_sm,
                             size_t dynamic_smem = 0) {
    int v = cache.load(std::memory_order_relaxed);
    if (v == 0) {
        const cudaError_t err =
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, threads, dynamic_smem);
        if (err != cudaSuccess) return err;
        cache.store(v, std::memory_order_relaxed);
    }
    per_sm = v;
    return cudaSuccess;
}

// Checked builds: out-of-range accesses caught per translation unit.
unsigned long long violations_build();
unsigned long long violations_query();
unsigned long long violations_batch();
unsigned long long violations_query_lead();
unsigned long long violations_query_host();
unsigned long long violations_batch_unaligned();
unsigned long long violations_persist();

// ---- plain index (build.cu) ----
struct BuildPlan {
    const float *A;   // buffer; element i of the array is A[off + i]
    int64_t off;      // table index only; 0 but for an array of a batch
    int64_t limit;    // one past the buffer's last value
    uint32_t lead;    // elements before the array's first (of n), 0 but in a batch
    uint32_t n;
    uint32_t bs;      // block size asked for
    bool aligned;
    uint32_t kmode;   // KeyMode: float32 / int32 elements, minimum / maximum
    // the table index (every index but RMQ_BUILD_NO_MICRO ones): minima of
    // the 32-element micro-blocks, the micro table over them (masks and
    // offset rows, tables_impl.cuh) and a sparse table over the minima of
    // blocks of tbs elements. Without it: pre / suf per element and the
    // sparse table over blocks of bs (tbs == bs)
    bool micro;
    bool light;       // RMQ_BUILD_LIGHT was given (reported, same structure)
    uint32_t tbs;
    uint32_t nb;      // blocks of tbs elements
    uint32_t levels;
    Entry *st;        // [levels * nb], level 0 = block minima
    // block table of larger blocks for longer ranges (cbs 0: none)
    uint32_t cbs, cnb, clevels;
    Entry *cst;       // [clevels * cnb]
    uint32_t nmicro;  // ceil(n / 32)
    uint32_t mlevels;
    uint32_t moff_bytes;
    // queries whose end micro-blocks are fewer than this apart go through the
    // micro table
    uint32_t micro_span;
    Entry *mst;       // [nmicro] micro-block minima
    void *mask;       // [nmicro] (tables_impl.cuh)
    void *moff;       // [moff_rows * nmicro]
    Entry *pre;       // [n]
    Entry *suf;       // [n]
};
constexpr uint32_t kMicro = 32;
// levels of a sparse table over nb blocks
inline uint32_t st_levels(uint32_t nb) { return nb ? static_cast<uint32_t>(ilog2(nb)) + 1u : 0u; }
// levels of a micro table that answers every query inside one block of bs
// elements (0 below 64). The micro table works on 32-element micro-blocks
// aligned in the array, whatever the block size. A query first probes it over
// every micro-block it touches (a superset of [l, r]; two windows of 2^k
// micro-blocks cover up to 2^(k+1) - 1 of them), so it holds windows long
// enough for any query inside one block: a block touches bs/32 micro-blocks
// when blocks start on micro-block boundaries (bs a multiple of 32, as in
// every table index), at most floor((bs + 30) / 32) + 1 otherwise.
inline uint32_t micro_levels(uint32_t bs) {
    if (bs < 2u * 32u) return 0;
    return st_levels(bs % 32u == 0 ? bs / 32u : (bs + 30u) / 32u + 1u);
}
// bytes of one micro-table offset for a table of `mlevels` levels: the
// largest offset is 2^(mlevels - 1) - 1
inline uint32_t micro_offset_bytes(uint32_t mlevels) {
    return mlevels <= 9 ? 1u : (mlevels <= 17 ? 2u : 4u);
}
// Shape of a table index with blocks of about bs elements (arrays of a batch;
// rmq_query_stats): the blocks of its block table (multiples of 32, so that
// blocks hold whole micro-blocks, at least 64) and the levels of its micro
// table, which answers every query inside a block.
struct TableShape {
    uint32_t tbs, mlevels;
};
// - Blocks above 2^15: the micro table would be 13 rows and more of 2-byte
//   offsets, too large for L2 and read twice per query; 4096 instead (n = 1e8,
//   2^26 queries, lr=-2, bs 195312: 0.83 ms with the rows, 0.58 with 4096).
// - Fewer than 32: a range of a few blocks is open as often as the blocks at
//   its ends are larger than it, so the blocks shrink until there are that
//   many, and windows of up to 511 micro-blocks do for blocks of no more than
//   that (rows up to level 8 are made in the run of the minima, longer ones
//   take another step); blocks of 2^14 elements hold 512 and need the next
//   level. With 128 the ragged benchmark's build takes 1.83 ms in place of 1.67
//   for its many small block tables, and its queries gain nothing.
// - The masks answer windows of up to 63 (127) micro-blocks whatever the
//   block size: 6 or 7 levels cost nothing.
constexpr uint32_t kLeastBlocks = 32;
inline TableShape table_shape(uint32_t n, uint32_t bs) {
    TableShape s;
    s.tbs = bs > (1u << 15) ? 4096u : bs <= 64u ? 64u : (bs + 31u) / 32u * 32u;
    const uint32_t least = mask_levels(wide_masks((n + kMicro - 1) / kMicro));
    s.mlevels = micro_levels(s.tbs);
    if (s.mlevels < least) s.mlevels = least;
    uint32_t few = 64u;  // a power of two, so that the run reduces their minima
    while (few <= n / kLeastBlocks / 2u) few *= 2u;
    if (few < s.tbs) {
        s.tbs = few;
        const uint32_t most = few > 511u * kMicro ? micro_levels(few) : 9u;
        if (s.mlevels > most) s.mlevels = most;
    }
    return s;
}

// Shape of the plain table index: of n alone, whatever block size is asked for.
// - Windows of up to 64 micro-blocks are answered by the micro table, from one
//   64-bit mask or two of 32. Twice as many by two masks of 64 would be, but
//   four scattered loads cost more than the block table's two, if its blocks
//   are small (n = 1e8, ranges of 3000, 2^26 queries: 0.94 ms by masks, 0.77
//   by blocks of 512). So the micro table needs no offset rows.
// - Blocks: small ones leave fewer queries open, large ones make rows that fit
//   L1. 2^13 to 2^14 of them up to 512 elements each (n = 4e6, lr=-2: 0.51 ms
//   with 512, 0.49 with 256, 0.56 with 64; n = 1e7: 0.54 with 1024, 0.52, 0.56
//   with 256).
// - From 2^13 blocks on a second table over larger ones, 2^12 to 2^13 of them,
//   for ranges of kCoarseFrom and more of those: rows of 64 KB (n = 1e8, uniform
//   lengths: 0.57 ms by blocks of 4096, 0.34 by blocks of 16384).
struct IndexShape {
    uint32_t tbs, mlevels, micro_span, cbs;
};
constexpr uint32_t kIndexBlocks = 1u << 13, kCoarseFrom = 64;
inline IndexShape index_shape(uint32_t n) {
    const bool wide = wide_masks((n + kMicro - 1) / kMicro);
    IndexShape s{64u, mask_levels(wide), wide ? 64u : 63u, 0u};
    while (s.tbs < 512u && n / (2u * s.tbs) >= kIndexBlocks) s.tbs *= 2u;
    if (n / s.tbs >= kIndexBlocks)
        for (s.cbs = 2u * s.tbs; n / s.cbs >= kIndexBlocks; s.cbs *= 2u) {}
    return s;
}

// Fill the size fields of a plan (A, n, bs and light given; the table index
// unless `no_micro`, in blocks of bs where `asked`); returns the bytes of the
// single allocation holding the index and its invalid-query counter.
size_t plan_index(BuildPlan &p, bool no_micro, bool asked = false);
// Point the plan's arrays into that allocation; returns the counter.
unsigned long long *place_index(BuildPlan &p, void *base);
cudaError_t launch_build(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s);
// Per-element prefix / suffix minima over blocks of p.bs elements into p.pre
// and p.suf, block minima into p.st[0 .. ceil(n / bs)).
cudaError_t launch_build_entries(const BuildPlan &p, const DeviceInfo &dev, cudaStream_t s);
// Size fields of index files of version 5, whose full indexes held four
// entries per element; returns the bytes of their payload.
struct LayoutV5 {
    uint32_t nb, levels, nmicro, mlevels;
};
size_t layout_v5(uint32_t n, uint32_t bs, bool light, bool no_micro, LayoutV5 *out);

// ---- handles (api.cu) ----
}  // namespace rmq
struct rmq_handle;
namespace rmq {
// The plan (with its device pointers), allocation and size of a handle.
int handle_view(const rmq_handle *h, BuildPlan *plan, void **mem, size_t *bytes);
// A new handle owning `mem` (laid out by place_index for `plan`), with its
// invalid-query counter cleared on `stream`.
int handle_adopt(BuildPlan plan, void *mem, size_t bytes, cudaStream_t stream, rmq_handle **out);

// ---- queries (query.cu) ----
struct QueryArgs {
    const int2 *Q;
    int64_t q;
    float *val;
    int32_t *idx;
    unsigned long long *invalid;  // device counter, may be null
    // measurement launches only (rmq_query_stats): kStatCount device
    // counters of how each query was settled; null for every other launch
    unsigned long long *stats = nullptr;
    bool host = false;  // val and idx, or one of them, are in host memory
};
cudaError_t launch_query(const BuildPlan &p, const QueryArgs &a, const DeviceInfo &dev,
                         cudaStream_t s);
struct V1View;
V1View view_of(const BuildPlan &p);
cudaError_t launch_probe_gather(const BuildPlan &p, const QueryArgs &a, const DeviceInfo &dev,
                                cudaStream_t s);
// Random 8-byte loads from buf[0 .. words), query_kernel's grid (rmq_probe_random).
cudaError_t launch_probe_random(const unsigned long long *buf, uint64_t words, const QueryArgs &a,
                                const DeviceInfo &dev, cudaStream_t s);
cudaError_t launch_query_scan(const float *A, uint32_t n, const QueryArgs &a,
                              const DeviceInfo &dev, cudaStream_t s);

}  // namespace rmq
