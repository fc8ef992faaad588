"""GPU: queries whose results go to host memory in place. A step's queries are all
settled before their results are stored, so that every line of the host buffers is
stored once and whole: ranges of every kind mixed within a warp (inside one
micro-block, open at one end or both, tied, long, invalid), partial steps, every key
mode, unaligned values, NaN and signed zeros; both outputs, either one, and one of
them in device memory. Exact against a host sparse table, bit for bit against the
results in device memory."""
import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu


def mixed(n, q, rng):
    """Ranges of all lengths in random order, a few of them invalid."""
    w = np.exp(rng.uniform(0, np.log(n + 1), q)).astype(np.int64)
    some = rng.random(q) < 0.6
    w[some] = rng.integers(1, min(n, 200) + 1, int(some.sum()))
    w = np.clip(w, 1, n)
    l = (rng.random(q) * (n - w + 1)).astype(np.int64)
    Q = np.stack([l, l + w - 1], 1)
    bad = rng.random(q) < 0.01
    Q[bad] = np.array([[5, 4], [-1, 3], [0, n]])[rng.integers(0, 3, int(bad.sum()))]
    return Q.astype(np.int32), bad


@pytest.mark.parametrize("n", [7, 1335, 262_144, 5_000_011])
@pytest.mark.parametrize("kind", ["unit", "ties", "special", "int32"])
@pytest.mark.parametrize("off,op", [(0, "min"), (1, "max"), (0, "max"), (3, "min")])
def test_results_in_host_memory(cuda, native, n, kind, off, op):
    import torch

    import rtxrmq_gb300 as R
    rng = np.random.default_rng(n + off)
    if kind == "int32":
        A = rng.integers(-2**31, 2**31 - 1, n).astype(np.int32)
        A[rng.random(n) < 0.3] = -2**31
        A[rng.random(n) < 0.3] = 2**31 - 1
    else:
        A = (rng.random(n) if kind == "unit" else rng.integers(0, 3, n)).astype(np.float32)
        if kind == "special":
            for x in (np.nan, 0.0, -0.0, np.inf, -np.inf):
                A[rng.integers(0, n, n // 9 + 1)] = x
    buf = torch.zeros(n + off, dtype=torch.from_numpy(A).dtype, device=cuda)
    buf[off:] = torch.from_numpy(A).to(cuda)
    with R.RMQIndex(buf[off:], op=op) as ix:
        for q in (1, 33, 511, 512, 513, 40_000):
            Q, bad = mixed(n, q, rng)
            dv, di = (x.cpu() for x in ix.query(torch.from_numpy(Q).to(cuda)))
            hQ = torch.from_numpy(Q).pin_memory()
            hv, hi = torch.empty_like(dv).pin_memory(), torch.empty_like(di).pin_memory()
            gv, gi = hv.to(cuda), hi.to(cuda)
            for v, i in ((hv, hi), (hv, None), (None, hi), (hv, gi), (gv, hi)):
                for x in (hv, hi, gv, gi):
                    x.fill_(77)
                ix.query_host(hQ, v, i)
                torch.cuda.synchronize()
                if v is not None:
                    np.testing.assert_array_equal(v.cpu().view(torch.int32).numpy(), dv.view(torch.int32).numpy())
                if i is not None:
                    np.testing.assert_array_equal(i.cpu().numpy(), di.numpy())
        assert (di.numpy()[bad] == -1).all()
        if kind in ("unit", "ties"):
            B = A if op == "min" else -A
            m = range_min(composites(B + 0.0), Q[~bad][:, 0], Q[~bad][:, 1])
            np.testing.assert_array_equal(di.numpy()[~bad], (m & np.uint64(0xffffffff)).astype(np.int64) >> 1)


@pytest.mark.parametrize("mode", ["1", "2", "3"])
def test_partly_staged(cuda, native, monkeypatch, mode):
    """Queries staged and results in place, results staged, both."""
    import torch

    import rtxrmq_gb300 as R
    rng = np.random.default_rng(int(mode))
    A = rng.random(300_000).astype(np.float32)
    Q, _ = mixed(len(A), 30_000, rng)
    with R.RMQIndex(torch.from_numpy(A).to(cuda)) as ix:
        dv, di = (x.cpu().numpy() for x in ix.query(torch.from_numpy(Q).to(cuda)))
        monkeypatch.setenv("RTXRMQ_HOST_MODE", mode)
        hv, hi = torch.zeros(len(Q)).pin_memory(), torch.zeros(len(Q), dtype=torch.int32).pin_memory()
        for v, i in ((hv, hi), (hv, None), (None, hi)):
            hv.fill_(7), hi.fill_(7)
            ix.query_host(torch.from_numpy(Q).pin_memory(), v, i)
            torch.cuda.synchronize()
            if v is not None:
                np.testing.assert_array_equal(hv.numpy().view(np.uint32), dv.view(np.uint32))
            if i is not None:
                np.testing.assert_array_equal(hi.numpy(), di)
