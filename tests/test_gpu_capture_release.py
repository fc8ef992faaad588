"""GPU: an index built before a capture and released while a stream captures, in
the capturing thread or in another one, in the modes that allow the release of
memory: the capture stays valid, the release waits for the index's queries, and
the graph replays."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
@pytest.mark.parametrize("how", ["close", "free"])
def test_release_during_capture(cuda, native, mode, how):
    import torch

    import rtxrmq_gb300 as R
    from rtxrmq_gb300._native import check
    A = torch.rand(50_000, device=cuda)
    Q = torch.from_numpy(R.gen_queries(4000, 50_000, -1, 3)).to(cuda)
    x = torch.ones(1000, device=cuda)
    kept, gone = R.RMQIndex(A), R.RMQIndex(A, 1024)
    v, i = kept.query(Q)
    torch.cuda.synchronize()
    s, w = torch.cuda.Stream(), torch.cuda.Stream()
    errors = []

    def release():
        try:
            torch.cuda.set_device(cuda)
            with torch.cuda.stream(w):
                torch.cuda._sleep(20_000_000)
                got = gone.query(Q, stream=w)
                done = torch.cuda.Event()
                done.record(w)
                if how == "close":
                    gone.close()  # used on two streams: waits
                else:
                    h, gone._h = gone._h, type(gone._h)()
                    check(native.rmq_free(h))
                assert done.query()
                out.append(got[1])
        except Exception as e:  # surfaced below
            errors.append(e)

    out = []
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode=mode):
        x.mul_(2.0)
        kept.query(Q, out_val=v, out_idx=i)
        if mode == "relaxed":
            h, gone._h = gone._h, type(gone._h)()
            check(native.rmq_free_async(h, s.cuda_stream) if how == "close" else native.rmq_free(h))
        else:
            t = threading.Thread(target=release)
            t.start()
            t.join(timeout=60)
        x.add_(1.0)
    assert not errors, errors
    want = i.cpu().numpy().copy()
    i.zero_()
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 7.0
    np.testing.assert_array_equal(i.cpu().numpy(), want)
    for o in out:
        np.testing.assert_array_equal(o.cpu().numpy(), want)
    kept.close()
