"""CPU: the rules of api.cu about index memory, run against a CUDA runtime on the
host (fake_cuda.h): whose order a release follows, that a waiting one leaves
captures alone, that a pool ends with its context, that what it keeps counts as free,
and where tables made for one call come from."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HEAD = '#include "fake_cuda.h"\n#include "api.cu"\n'
INDEX = r"""
static float values[100000];
static rmq_handle_t *index_of(int device, rmq_stream_t s = nullptr, int64_t n = 100000) {
    fake::device = device;
    rmq_handle_t *h = nullptr;
    return rmq_build(values, n, 0, s, &h) == RMQ_OK ? h : nullptr;
}
"""


def run(tmp_path, body):
    src = tmp_path / "rules.cpp"
    src.write_text(HEAD + INDEX + "int main() {\n" + body + '    std::printf("ok\\n");\n    return 0;\n}\n')
    exe = tmp_path / "rules"
    csrc = ROOT / "rtxrmq_gb300" / "csrc"
    r = subprocess.run(["g++", "-std=c++17", "-x", "c++", f"-I{ROOT / 'tests'}", f"-I{csrc}",
                        "-I/usr/local/cuda/include", str(src), "-o", str(exe), "-ldl", "-lpthread",
                        "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_release_follows_the_index_device(tmp_path):
    """In stream order on the index's own device; on another current device the
    default stream is that device's, so the release waits for the index's."""
    run(tmp_path, r"""
    rmq_handle_t *h = index_of(0);
    EXPECT(h && fake::take() == "create0 pool0 ");
    EXPECT(rmq_free_async(h, nullptr) == RMQ_OK && fake::take() == "free-async0 ");
    h = index_of(1);
    EXPECT(h && fake::take() == "create1 pool1 ");
    fake::device = 0;
    EXPECT(rmq_free_async(h, nullptr) == RMQ_OK);
    EXPECT(fake::log == "wait1 free0 " && fake::device == 0 && fake::held.empty());
    fake::take();
    h = index_of(1);
    fake::take();
    EXPECT(rmq_free_async(h, nullptr) == RMQ_OK && fake::take() == "free-async1 ");
""")


def test_waiting_release_leaves_captures_alone(tmp_path):
    """rmq_free waits by calls that a relaxed or thread-local capture allows, as
    the release of memory from cudaMalloc does; under a global one it fails, as
    that does."""
    run(tmp_path, r"""
    rmq_handle_t *h = index_of(0), *g = index_of(0);
    fake::take();
    fake::capture = 1;
    EXPECT(rmq_free(h) == RMQ_OK && fake::take() == "wait0 free0 " && !fake::broken);
    fake::capturing_stream = true;
    EXPECT(rmq_free_async(g, nullptr) == RMQ_OK && fake::take() == "wait0 free0 " && !fake::broken);
    fake::capturing_stream = false;
    fake::capture = 0;
    h = index_of(0);
    fake::left = 0;  // not even a word for the wait
    fake::take();
    EXPECT(rmq_free(h) == RMQ_OK && fake::take() == "wait0 free0 ");
    EXPECT(fake::held.empty());
""")


def test_pool_ends_with_its_context(tmp_path):
    """A device reset ends the pool and what came from it: the next index takes a
    new pool, a handle of before releases nothing, the other device keeps its
    own."""
    run(tmp_path, r"""
    rmq_handle_t *a = index_of(0), *b = index_of(0), *c = index_of(1);
    EXPECT(fake::take() == "create0 pool0 pool0 create1 pool1 ");
    fake::device = 0;
    fake::context[0] = 21;
    EXPECT(rmq_trim() == RMQ_OK && fake::take() == "");
    rmq_handle_t *d = index_of(0);
    EXPECT(d && fake::take() == "create0 pool0 ");
    EXPECT(rmq_free(a) == RMQ_OK && rmq_free_async(b, nullptr) == RMQ_OK && fake::take() == "");
    EXPECT(rmq_free_async(d, nullptr) == RMQ_OK && fake::take() == "free-async0 ");
    EXPECT(rmq_trim() == RMQ_OK && fake::take() == "trim0 ");
    EXPECT(index_of(0) && fake::take() == "pool0 ");
    fake::device = 1;
    EXPECT(rmq_free_async(c, nullptr) == RMQ_OK && fake::take() == "free-async1 ");
""")


def test_kept_memory_counts_as_free(tmp_path):
    """Memory that the pool keeps from released indexes goes to any allocation of
    the library that finds no other, after the work before the release; injected
    failures stay failures."""
    run(tmp_path, r"""
    static int32_t queries[2], out[1];
    fake::left = 2100000;
    rmq_handle_t *a = index_of(0), *b = index_of(0);  // 400 kB each
    EXPECT(a && b && rmq_free_async(a, nullptr) == RMQ_OK);
    EXPECT(fake::left < 1600000 && fake::take() == "create0 pool0 pool0 free-async0 ");
    EXPECT(rmq_probe_gather(b, queries, 1, nullptr, out, nullptr) == RMQ_OK);  // entries of 1.6 MB
    EXPECT(fake::take() == "wait0 trim0 malloc0 ");
    EXPECT(rmq_free(b) == RMQ_OK);
    fake::take();
    setenv("RTXRMQ_FAIL_ALLOC", "1", 1);
    EXPECT(!index_of(0) && fake::take() == "");
""")


def test_counting_takes_its_tables_from_the_pool(tmp_path):
    """rmq_query_stats makes tables for the call: from the pool, and back to it in
    stream order, with no allocation that waits for the device."""
    run(tmp_path, r"""
    static int32_t queries[2];
    static int64_t counts[RMQ_QUERY_STATS_FIELDS];
    rmq_handle_t *h = index_of(0);
    fake::take();
    EXPECT(rmq_query_stats(h, queries, 1, nullptr, nullptr, counts, nullptr) == RMQ_OK);
    EXPECT(fake::take() == "pool0 free-async0 ");
    setenv("RTXRMQ_FAIL_ALLOC", "1", 1);
    EXPECT(rmq_query_stats(h, queries, 1, nullptr, nullptr, counts, nullptr) == RMQ_ENOMEM && fake::take() == "");
""")
