"""CPU: what a launch needs to be told about a kernel, shared memory beyond 48 KB or
a carve-out, belongs to a device. The compiled host code of the builder and of the
query launch runs against a CUDA runtime on the host that refuses a launch with more
shared memory than the current device's attribute allows: indexes of sizes around
every rule, first on one device, then on another."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <set>
#include <tuple>
#include "../../include/rmq.h"
#include "engine.h"
using namespace rmq;
namespace fake {
int device = 0;
cudaError_t last = cudaSuccess;
struct { dim3 grid, block; size_t smem; cudaStream_t s; } pending;
std::map<std::tuple<int, const void *, int>, int> attr;
std::set<std::pair<int, const void *>> launched;
int refused = 0;
}
extern "C" {
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    fake::pending = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s) {
    *g = fake::pending.grid, *b = fake::pending.block, *smem = fake::pending.smem;
    *static_cast<cudaStream_t *>(s) = fake::pending.s;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) {
    const auto at = fake::attr.find({fake::device, f, int(cudaFuncAttributeMaxDynamicSharedMemorySize)});
    if (smem > 48 * 1024 && (at == fake::attr.end() || size_t(at->second) < smem)) {
        ++fake::refused;
        return fake::last = cudaErrorInvalidValue;
    }
    fake::launched.insert({fake::device, f});
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t f, dim3 g, dim3 b, void **a, size_t smem, cudaStream_t s) {
    return cudaLaunchKernel(reinterpret_cast<const void *>(f), g, b, a, smem, s);
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    fake::attr[{fake::device, f, int(a)}] = v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = fake::last; fake::last = cudaSuccess; return e; }
}
namespace rmq {
int cuda_fail(cudaError_t, const char *) { return RMQ_ECUDA; }
}
int main() {
    for (int d : {0, 1, 5}) {
        fake::device = d;
        const DeviceInfo dev{d, 152, size_t(1) << 27};
        for (uint32_t n : {1u, 5000u, 196000u, 197000u, 250000u, 262144u, 262145u, 1000000u, 100000000u})
            for (int kind = 0; kind < 3; ++kind) {  // plain, no sub-block level, tables as asked for
                BuildPlan p;
                std::memset(&p, 0, sizeof(p));
                p.A = reinterpret_cast<const float *>(uintptr_t(1) << 30);
                p.n = n;
                p.bs = kind == 1 ? (n + 3999) / 4000 : 1u << 15;
                plan_index(p, kind == 1, kind == 2);
                place_index(p, reinterpret_cast<void *>(uintptr_t(1) << 40));
                QueryArgs a;
                a.Q = reinterpret_cast<const int2 *>(uintptr_t(1) << 41);
                a.q = 1000;
                a.val = nullptr;
                a.idx = reinterpret_cast<int32_t *>(uintptr_t(1) << 42);
                a.invalid = nullptr;
                const cudaError_t b = launch_build(p, dev, nullptr), q = launch_query(p, a, dev, nullptr);
                if (b != cudaSuccess || q != cudaSuccess || fake::refused) {
                    std::printf("device %d, n=%u, kind %d: build %d, query %d, %d launches refused\n", d, n,
                                kind, int(b), int(q), fake::refused);
                    return 1;
                }
            }
    }
    // a carve-out that one device was told of, every device that launches is told of
    int carved = 0;
    for (const auto &e : fake::attr) {
        if (std::get<2>(e.first) != int(cudaFuncAttributePreferredSharedMemoryCarveout)) continue;
        ++carved;
        for (const auto &l : fake::launched)
            if (l.second == std::get<1>(e.first) &&
                !fake::attr.count({l.first, l.second, int(cudaFuncAttributePreferredSharedMemoryCarveout)})) {
                std::printf("device %d launches without its carve-out\n", l.first);
                return 1;
            }
    }
    std::printf("ok %d\n", carved);
    return carved == 0;
}
"""


def test_second_device(native, tmp_path):
    csrc = ROOT / "rtxrmq_gb300" / "csrc"
    obj = ROOT / "rtxrmq_gb300" / "_lib" / "obj"
    src, exe = tmp_path / "attr.cpp", tmp_path / "attr"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-no-pie", f"-I{csrc}", "-I/usr/local/cuda/include", str(src),
                        str(obj / "build.cu.o"), str(obj / "query.cu.o"), "-o", str(exe), "-ldl",
                        "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
