// A CUDA runtime on the host for the tests of api.cu's rules (who may use, keep
// and release which memory, when): two devices, no kernels, memory from malloc,
// every call that matters written to a log. Included by a test program together
// with api.cu; what the program does not use stays unresolved.
#pragma once
#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../include/rmq.h"
#include "engine.h"

namespace fake {
std::string log;           // calls since the last take()
int device = 0;            // current device
int capture = 0;           // a stream captures: 0 none, 1 this thread relaxed, 2 global mode
bool capturing_stream = false;  // the stream asked about captures
bool broken = false;       // the capture was invalidated
size_t left = ~size_t(0);  // bytes that cudaMalloc still has
unsigned long long context[2] = {11, 12};  // ids of the devices' contexts
std::map<void *, size_t> held;
struct Pool { int device; unsigned long long context; size_t keeps; };
std::map<void *, Pool *> pooled;
inline void note(const std::string &s) { log += s + " "; }
inline std::string take() { std::string s; s.swap(log); return s; }
inline cudaError_t unsafe(const char *) {  // potentially unsafe under a global capture
    if (capture != 2) return cudaSuccess;
    broken = true;
    return cudaErrorStreamCaptureUnsupported;
}
inline CUresult get_current(CUcontext *c) { *c = reinterpret_cast<CUcontext>(&context[device]); return CUDA_SUCCESS; }
inline CUresult get_id(CUcontext c, unsigned long long *id) { *id = *reinterpret_cast<unsigned long long *>(c); return CUDA_SUCCESS; }
}  // namespace fake

extern "C" {
const char *cudaGetErrorName(cudaError_t) { return "error"; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 100; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    *s = fake::capturing_stream ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *props) {
    fake::note("create" + std::to_string(props->location.id));
    *p = reinterpret_cast<cudaMemPool_t>(new fake::Pool{props->location.id, fake::context[props->location.id], 0});
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t) {
    const fake::Pool *f = reinterpret_cast<fake::Pool *>(pool);
    if (f->context != fake::context[f->device]) {
        fake::note("dead-pool");
        return cudaErrorInvalidValue;
    }
    if (n > fake::left) return cudaErrorMemoryAllocation;
    fake::note("pool" + std::to_string(f->device));
    fake::held[*p = std::calloc(1, n)] = n;
    fake::left -= n;
    fake::pooled[*p] = reinterpret_cast<fake::Pool *>(pool);
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t) {
    fake::Pool *f = reinterpret_cast<fake::Pool *>(pool);
    if (f->context != fake::context[f->device]) {
        fake::note("dead-pool");
        return cudaErrorInvalidValue;
    }
    fake::note("trim" + std::to_string(f->device));
    fake::left += f->keeps;
    f->keeps = 0;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    if (const cudaError_t e = fake::unsafe("cudaMalloc")) return e;
    if (n > fake::left) return cudaErrorMemoryAllocation;
    if (n > 4096) fake::note("malloc" + std::to_string(fake::device));
    fake::held[*p = std::calloc(1, n)] = n;
    fake::left -= n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {  // waits for the device, in any capture but a global one
    if (!p) return cudaSuccess;
    if (const cudaError_t e = fake::unsafe("cudaFree")) return e;
    const auto it = fake::held.find(p);
    if (it == fake::held.end()) {
        fake::note("bad-free");
        return cudaErrorInvalidValue;
    }
    fake::note((it->second > 4096 ? "free" : "wait") + std::to_string(fake::device));
    (fake::pooled.count(p) ? fake::pooled[p]->keeps : fake::left) += it->second;
    fake::pooled.erase(p);
    fake::held.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) {
    fake::note("free-async" + std::to_string(fake::device) + (s ? "s" : ""));
    fake::pooled[p]->keeps += fake::held[p];
    fake::pooled.erase(p);
    fake::held.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) {
    if (fake::capture) {
        fake::broken = true;
        return cudaErrorStreamCaptureUnsupported;
    }
    fake::note("wait" + std::to_string(fake::device));
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *st) {
    *f = std::string(name) == "cuCtxGetCurrent" ? reinterpret_cast<void *>(&fake::get_current)
                                                : reinterpret_cast<void *>(&fake::get_id);
    if (st) *st = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}

namespace rmq {
size_t plan_index(BuildPlan &p, bool no_micro, bool) {
    p.micro = !no_micro;
    return size_t(p.n) * 4;
}
unsigned long long *place_index(BuildPlan &, void *base) { return static_cast<unsigned long long *>(base); }
cudaError_t launch_build(const BuildPlan &, const DeviceInfo &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_build_entries(const BuildPlan &, const DeviceInfo &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_probe_gather(const BuildPlan &, const QueryArgs &, const DeviceInfo &, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_query(const BuildPlan &, const QueryArgs &, const DeviceInfo &, cudaStream_t) { return cudaSuccess; }
}  // namespace rmq

#define EXPECT(cond)                                                                          \
    do {                                                                                      \
        if (!(cond)) {                                                                        \
            std::printf("line %d: %s; log: %s\n", __LINE__, #cond, fake::log.c_str());         \
            return 1;                                                                         \
        }                                                                                     \
    } while (0)
