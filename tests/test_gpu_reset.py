"""GPU: indexes before and after a reset of the device (a program of its own): the
first one after it is built in a pool of the new context, also of a size whose
block table takes more than 48 KB of shared memory; an index of before the reset
can be released; answers exact against a host scan."""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include <cuda_runtime.h>
#include "rmq.h"
#define CHECK(x) do { const int e = (x); if (e) { std::printf("line %d: %d %s\n", __LINE__, e, rmq_last_error_string()); return 1; } } while (0)
static rmq_handle_t *kept = nullptr;
static int round_of(int64_t n, bool keep) {
    std::vector<float> A(n);
    unsigned s = 1u;
    for (float &x : A) x = static_cast<float>((s = s * 1664525u + 1013904223u) >> 12);
    std::vector<int> Q;
    for (int k = 0; k < 400; ++k) {
        s = s * 1664525u + 1013904223u;
        const int l = static_cast<int>(s % static_cast<unsigned>(n));
        s = s * 1664525u + 1013904223u;
        const int r = l + static_cast<int>((s >> 4) % static_cast<unsigned>(n - l));
        Q.push_back(l);
        Q.push_back(r);
    }
    float *dA;
    int *dQ, *dI;
    CHECK(cudaMalloc(&dA, n * 4));
    CHECK(cudaMalloc(&dQ, Q.size() * 4));
    CHECK(cudaMalloc(&dI, Q.size() * 2));
    CHECK(cudaMemcpy(dA, A.data(), n * 4, cudaMemcpyHostToDevice));
    CHECK(cudaMemcpy(dQ, Q.data(), Q.size() * 4, cudaMemcpyHostToDevice));
    rmq_handle_t *h = nullptr;
    CHECK(rmq_build(dA, n, 0, nullptr, &h));
    CHECK(rmq_query(h, dQ, 400, nullptr, dI, nullptr));
    std::vector<int> I(400);
    CHECK(cudaMemcpy(I.data(), dI, 1600, cudaMemcpyDeviceToHost));
    for (int k = 0; k < 400; ++k) {
        int m = Q[2 * k];
        for (int j = m; j <= Q[2 * k + 1]; ++j) if (A[j] < A[m]) m = j;
        if (m != I[k]) { std::printf("query %d: %d, not %d\n", k, I[k], m); return 1; }
    }
    if (keep) kept = h;
    else CHECK(rmq_free_async(h, nullptr));
    return 0;
}
int main() {
    for (int reset = 0; reset < 3; ++reset) {
        for (int64_t n : {5000, 250000, 90000}) CHECK(round_of(n, false));
        CHECK(round_of(230000, true));
        CHECK(rmq_trim());
        CHECK(cudaDeviceReset());
        if (reset == 1) { CHECK(round_of(240000, false)); }
        CHECK(rmq_free(kept));
    }
    std::printf("ok\n");
    return 0;
}
"""


def test_index_after_a_device_reset(cuda, native, tmp_path):
    from rtxrmq_gb300 import build as b
    lib = b.build()
    src, exe = tmp_path / "reset.cpp", tmp_path / "reset"
    src.write_text(PROGRAM)
    home = b._cuda_home(b._nvcc())
    r = subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'include'}", f"-I{home / 'include'}", str(src),
                        "-o", str(exe), f"-L{lib.parent}", "-lrmq", f"-Wl,-rpath,{lib.parent}",
                        f"-L{home / 'lib64'}", "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
