"""GPU: index memory from the library's pool. Indexes released in stream order
while their queries are still queued, on one stream, on several streams and
threads; streams whose lifetime is not known, and captured queries, take the
waiting release; what the pool keeps is bounded and given back by rmq_trim; a
failing allocation is reported as before. Answers exact against torch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def reference(A, Q):
    return np.array([l + int(np.argmin(A[l:r + 1])) for l, r in Q], np.int32)


def problems(cuda, seed, count, n=30_000):
    import torch

    import rtxrmq_gb300 as R
    out = []
    for k in range(count):
        A = np.random.default_rng(seed + k).random(n + 97 * k).astype(np.float32)
        Q = R.gen_queries(3000, len(A), (-1, -2, -3)[k % 3], seed + k)
        out.append((torch.from_numpy(A).to(cuda), torch.from_numpy(Q).to(cuda), reference(A, Q[:200])))
    return out


def test_release_in_stream_order(cuda, native):
    """A new index takes the memory of one whose queries have not run yet; it
    is built behind them."""
    import torch

    import rtxrmq_gb300 as R
    work = problems(cuda, 1, 12)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    for stream in (torch.cuda.current_stream(), s):
        got = []
        with torch.cuda.stream(stream):
            for _ in range(4):
                for A, Q, want in work:
                    with R.RMQIndex(A, 1024) as ix:
                        got.append((ix.query(Q)[1], want))
        torch.cuda.synchronize()
        for i, want in got:
            np.testing.assert_array_equal(i.cpu().numpy()[:200], want)


def test_release_on_several_streams_and_threads(cuda, native):
    import torch

    import rtxrmq_gb300 as R
    errors = []

    def loop(k):
        try:
            torch.cuda.set_device(cuda)
            work = problems(cuda, 100 * k, 6)
            torch.cuda.synchronize()
            s = torch.cuda.Stream()
            got = []
            with torch.cuda.stream(s):
                for _ in range(6):
                    for A, Q, want in work:
                        with R.RMQIndex(A, 256, light=k % 2 == 1) as ix:
                            got.append((ix.query(Q)[1], want))
            s.synchronize()
            for i, want in got:
                np.testing.assert_array_equal(i.cpu().numpy()[:200], want)
        except Exception as e:  # surfaced below
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors, errors


def test_other_streams_take_the_waiting_release(cuda, native):
    """A second stream, a raw handle and an external stream: the release waits
    for the device, so the index's work is done when it returns."""
    import torch

    import rtxrmq_gb300 as R
    (A, Q, want), = problems(cuda, 7, 1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    e = torch.cuda.ExternalStream(s.cuda_stream)
    for build, query in ((None, s), (s.cuda_stream, s.cuda_stream), (e, e)):
        torch.cuda.synchronize()
        ix = R.RMQIndex(A, 512, stream=build)
        torch.cuda.synchronize()
        for _ in range(50):
            v, i = ix.query(Q, stream=query)
        done = torch.cuda.Event()
        done.record(s)
        ix.close()
        assert done.query()
        np.testing.assert_array_equal(i.cpu().numpy()[:200], want)


def test_captured_query_keeps_its_index(cuda, native):
    import torch

    import rtxrmq_gb300 as R
    (A, Q, want), = problems(cuda, 9, 1)
    ix = R.RMQIndex(A, 512)
    v, i = ix.query(Q)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        ix.query(Q, out_val=v, out_idx=i)
    for _ in range(20):
        g.replay()
    done = torch.cuda.Event()
    done.record()
    ix.close()
    assert done.query()
    np.testing.assert_array_equal(i.cpu().numpy()[:200], want)


def test_bounded_and_given_back(cuda, native, monkeypatch):
    import torch

    import rtxrmq_gb300 as R
    from rtxrmq_gb300._native import RMQ_ENOMEM, check
    A = torch.rand(1 << 27, device=cuda)
    check(native.rmq_trim())
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    live = [R.RMQIndex(A, 4096) for _ in range(8)]  # 90 MB each
    for ix in live:
        ix.close()
    torch.cuda.synchronize()
    with R.RMQIndex(A, 4096):
        pass
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= (256 << 20) + (64 << 20), kept  # the bound, and what the driver rounds up
    check(native.rmq_trim())
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20
    monkeypatch.setenv("RTXRMQ_FAIL_ALLOC", "1")
    with pytest.raises(R.RMQError) as e:
        R.RMQIndex(A, 4096)
    assert e.value.code == RMQ_ENOMEM
