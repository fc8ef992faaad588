"""GPU: the fused table builder (runs of units of 256 micro-blocks, built from
the 128-byte boundary before an array on) at the sizes where it can go wrong:
arrays at every offset from a boundary, lengths around a unit (8192 values)
and a run (131072), block sizes without offset rows, with rows made in the run
and made apart, block tables of one item and of level groups, values off a
16-byte boundary, descending and constant values (the longest and shortest
masks). The batch, its halves and the per-array path against a host sparse
table, exact; the per-array path leaves the plan's index answering."""
import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu


def values(kind, n, rng):
    if kind == "descending":
        return np.arange(n, 0, -1).astype(np.float32)
    if kind == "constant":
        return np.full(n, 2.5, np.float32)
    return rng.integers(0, 1000, n).astype(np.float32)


@pytest.mark.parametrize("kind", ["ties", "descending", "constant"])
@pytest.mark.parametrize("bs", [64, 1024, 4096, 8192, 1 << 14, 1 << 15])
@pytest.mark.parametrize("off", [0, 1])
def test_batch_runs(cuda, native, kind, bs, off):
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    rng = np.random.default_rng(bs + off)
    lengths = [1, 31, 32, 33, 8160, 8191, 8192, 8193, 131_071, 131_072, 131_073, 300_000]
    lengths += [200 + k for k in range(32)]
    starts, at = [], 5
    for k, n in enumerate(lengths):
        starts.append(at)
        at += n + 1 + k % 7
    lengths, starts = np.array(lengths, np.int64), np.array(starts, np.int64)
    A = values(kind, at + 3, rng)
    qs = []
    for n in lengths:
        w = np.minimum(np.exp(rng.uniform(0, np.log(n + 1), 600)).astype(np.int64), n)
        w = np.maximum(w, 1)
        l = (rng.random(600) * (n - w + 1)).astype(np.int64)
        l[:20], w[:20] = 0, n           # the whole array
        l[20:40] = n - w[20:40]         # up to its last element
        qs.append(np.stack([l, l + w - 1], 1))
    Q = np.concatenate(qs)
    first = np.repeat(starts, 600)
    m = range_min(composites(A), Q[:, 0] + first, Q[:, 1] + first)
    ei = ((m & np.uint64(0xffffffff)).astype(np.int64) >> 1) - first
    ev = A[ei + first]
    big = torch.zeros(len(A) + 4, device=cuda)
    big[off:off + len(A)] = torch.from_numpy(A).to(cuda)
    dA, dQ = big[off:off + len(A)], torch.from_numpy(Q.astype(np.int32)).to(cuda)
    qstarts = np.arange(len(lengths), dtype=np.int64) * 600
    qcounts = np.full(len(lengths), 600, np.int64)
    with RMQBatch(starts, lengths, qstarts, qcounts, [bs] * 32) as b:
        outs = [b.run(dA, dQ), b.query(dA, dQ), b.run_per_array(dA, dQ), b.query(dA, dQ)]
        b.build(dA)
        outs.append(b.query(dA, dQ))
        torch.cuda.synchronize()
        assert b.invalid_count() == 0
    for k, (v, i) in enumerate(outs):
        bad = np.nonzero(i.cpu().numpy() != ei)[0]
        assert bad.size == 0, f"call {k}: {bad.size} wrong, first {tuple(Q[bad[0]])} of array {bad[0] // 600}"
        np.testing.assert_array_equal(v.cpu().numpy(), ev)


@pytest.mark.parametrize("length", [1, 10, 100])
def test_batch_ends_past_the_array(cuda, native, length):
    """Queries whose ends lie outside an array with a lead stay invalid, also
    those that wrap past 2^31 - 1 when the lead is added."""
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    top = 2**31 - 1
    Q = np.array([[0, length - 1], [0, length], [-1, 0], [-7, -7], [0, top], [top, top], [-2**31, 0],
                  [length - 1, length - 1], [1, 0]], np.int32)
    A = torch.arange(200, 0, -1, device=cuda, dtype=torch.float32)
    with RMQBatch([13], [length], [0], [len(Q)]) as b:
        v, i = b.run(A, torch.from_numpy(Q).to(cuda))
        assert list(i.cpu().numpy()) == [length - 1, -1, -1, -1, -1, -1, -1, length - 1, -1]
        assert b.invalid_count() == 7
