"""When RMQIndex.close() may release without waiting. What follows a close on the
stream that is current there (a read of the results, new tensors in the memory of
`values`) must find the index's work done or ordered before it, as it did when every
release waited for the device. The rule on the CPU, with stand-ins for streams and
the library; its effects on the GPU."""
import ctypes as C

import numpy as np
import pytest


class Calls:
    def __init__(self):
        self.seen = []

    def __getattr__(self, name):
        def call(*args):
            self.seen.append(name)
            return 0
        return call


class Stream:
    def __init__(self, handle, device=0):
        self.cuda_stream, self.device_index, self.stream_id = handle, device, 0 if handle == 0 else 2 * handle + 1


class Values:
    own = True

    def __init__(self, lib):
        self.lib = lib

    def untyped_storage(self):
        return self

    def resizable(self):
        return self.own

    def record_stream(self, s):
        self.lib.seen.append("record")


@pytest.fixture
def world(monkeypatch):
    import torch

    import rtxrmq_gb300 as R
    lib, now = Calls(), [Stream(0)]
    monkeypatch.setattr(R, "load", lambda: lib)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: now[0])
    monkeypatch.setattr(torch.cuda, "current_device", lambda: now[0].device_index)
    monkeypatch.setattr(R, "_durable", {})
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream",
                        lambda d: now[0].cuda_stream if d == now[0].device_index else 0, raising=False)

    def index(stream=None):
        ix = R.RMQIndex.__new__(R.RMQIndex)
        ix._values, ix._h = Values(lib), C.c_void_p(8)
        ix._one_stream, ix._keep = R._durable_stream(stream)
        return ix
    return lib, now, index


def test_rule(world):
    lib, now, index = world
    side = Stream(5)

    def closed(ix):
        lib.seen.clear()
        ix.close()
        return lib.seen

    in_order, waits = ["record", "rmq_free_async"], ["rmq_free"]
    assert closed(index()) == in_order
    assert closed(index(side)) == waits  # the results may be read on the current stream
    now[0] = side
    assert closed(index()) == in_order
    ix = index()
    now[0] = Stream(0)
    assert closed(ix) == waits
    now[0] = Stream(6, device=1)
    ix = index()
    now[0] = Stream(6, device=0)  # device 1 is back on its default stream
    assert closed(ix) == waits
    now[0] = Stream(0)
    ix = index()
    ix._use(side)
    assert closed(ix) == waits
    other = Stream(7)
    other.stream_id = 0x7f00  # external: its handle may be gone at the close
    now[0] = other
    assert closed(index()) == waits
    assert closed(index(other)) == waits and closed(index(7)) == waits
    now[0] = Stream(0)
    ix = index()
    ix._values.own = False  # memory of another library
    assert closed(ix) == waits
    ix = index()
    ix.query_host(np.zeros((1, 2), np.int32), np.zeros(1, np.float32))
    assert closed(ix) == waits
    assert closed(ix) == []  # once


@pytest.mark.gpu
def test_values_of_another_stream(cuda, native):
    """Values made on another stream than the index's, dropped right after the
    close: their memory is not used again while queries still read them."""
    import torch

    import rtxrmq_gb300 as R
    n = 1 << 22
    other = torch.cuda.Stream()
    want, got = [], []
    for k in range(6):
        with torch.cuda.stream(other):
            A = torch.rand(n, device=cuda)
        other.synchronize()
        Q = torch.from_numpy(R.gen_queries(200_000, n, -3, k)).to(cuda)
        want.append(A.cpu().numpy())
        ix = R.RMQIndex(A)
        torch.cuda.synchronize()
        torch.cuda._sleep(30_000_000)
        got.append((Q, *ix.query(Q)))
        ix.close()
        del A, ix
        with torch.cuda.stream(other):
            junk = [torch.full((n,), -1.0, device=cuda) for _ in range(3)]
        del junk
    torch.cuda.synchronize()
    for A, (Q, v, i) in zip(want, got):
        Q, i = Q.cpu().numpy(), i.cpu().numpy()
        np.testing.assert_array_equal(v.cpu().numpy(), A[i])
        for k in range(0, len(Q), 499):
            l, r = Q[k]
            assert i[k] == l + int(np.argmin(A[l:r + 1]))


@pytest.mark.gpu
def test_what_follows_a_close(cuda, native):
    """Closed while another stream is current, or after a query to host memory:
    the work is done when close() returns."""
    import torch

    import rtxrmq_gb300 as R
    A = torch.rand(300_000, device=cuda)
    Q = torch.from_numpy(R.gen_queries(3000, 300_000, -1, 2)).to(cuda)
    with R.RMQIndex(A) as ix:
        want = ix.query(Q)[1].cpu().numpy()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        ix = R.RMQIndex(A)
        torch.cuda._sleep(30_000_000)
        i = ix.query(Q)[1]
        done = torch.cuda.Event()
        done.record()
    ix.close()
    assert done.query()
    np.testing.assert_array_equal(i.cpu().numpy(), want)
    hQ, hI = Q.cpu().pin_memory(), torch.full((3000,), -5, dtype=torch.int32).pin_memory()
    with R.RMQIndex(A) as ix:
        torch.cuda._sleep(30_000_000)
        ix.query_host(hQ, out_idx=hI)
    np.testing.assert_array_equal(hI.numpy(), want)
    B = torch.from_dlpack(A)  # memory under another owner
    ix = R.RMQIndex(B)
    torch.cuda._sleep(30_000_000)
    ix.query(Q)
    done = torch.cuda.Event()
    done.record()
    ix.close()
    assert done.query()
