"""GPU: launches of one plan on several streams at a time share nothing but the
index. Two streams ask one built plan different queries, and run it on the same
values, with outputs of their own, launch after launch without waiting, also from
two threads and beside the replays of a captured run; arrays of very uneven query
counts, so that launches end raggedly and the next one starts beside the last.
Exact against a host sparse table: a query that one launch took from another
would keep the marker its output was filled with."""
import threading

import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu

ROUNDS = 24


class Plan:
    """A plan of ragged arrays, two sets of queries, their answers."""

    def __init__(self, cuda, seed=7):
        import torch

        from rtxrmq_gb300.batch import RMQBatch
        rng = np.random.default_rng(seed)
        lengths = np.concatenate([rng.integers(1, 3000, 300), [200_000, 90_000]])
        starts = np.cumsum(lengths) - lengths
        qcounts = np.concatenate([rng.integers(0, 60, 300), [60_000, 9000]])
        qstarts = np.cumsum(qcounts) - qcounts
        A = rng.integers(0, 900, int(lengths.sum())).astype(np.float32)
        first, n = np.repeat(starts, qcounts), np.repeat(lengths, qcounts)
        self.batch = RMQBatch(starts, lengths, qstarts, qcounts)
        self.values = torch.from_numpy(A).to(cuda)
        self.queries, self.want = [], []
        for _ in range(2):
            w = np.maximum(np.exp(rng.uniform(0, np.log(n + 1))).astype(np.int64), 1)
            w = np.minimum(w, n)
            l = (rng.random(len(n)) * (n - w + 1)).astype(np.int64)
            m = range_min(composites(A), l + first, l + w - 1 + first)
            self.want.append(((m & np.uint64(0xffffffff)).astype(np.int64) >> 1) - first)
            self.queries.append(torch.from_numpy(np.stack([l, l + w - 1], 1).astype(np.int32)).to(cuda))
        self.outs = [[torch.full((len(n),), -77, dtype=torch.int32, device=cuda) for _ in range(ROUNDS)]
                     for _ in range(2)]

    def launch(self, k, r, kind, stream):
        call = self.batch.run if kind == "run" else self.batch.query
        call(self.values, self.queries[k], out_idx=self.outs[k][r], values=False, stream=stream)

    def check(self):
        for k in range(2):
            for out in self.outs[k]:
                np.testing.assert_array_equal(out.cpu().numpy(), self.want[k])


@pytest.mark.parametrize("kind", ["query", "run"])
@pytest.mark.parametrize("threads", [False, True])
def test_two_streams(cuda, native, kind, threads):
    import torch
    p = Plan(cuda)
    p.batch.build(p.values)
    torch.cuda.synchronize()
    s = [torch.cuda.Stream(), torch.cuda.Stream()]
    errors = []

    def loop(k):
        try:
            torch.cuda.set_device(cuda)
            for r in range(ROUNDS):
                p.launch(k, r, kind, s[k])
        except Exception as e:  # surfaced below
            errors.append(e)

    if threads:
        ts = [threading.Thread(target=loop, args=(k,)) for k in range(2)]
        for t in ts:
            t.start()
        for t in ts:
            t.join(timeout=120)
    else:
        for r in range(ROUNDS):
            p.launch(0, r, kind, s[0])
            p.launch(1, r, kind, s[1])
    torch.cuda.synchronize()
    assert not errors, errors
    p.check()
    assert p.batch.invalid_count() == 0


def test_replays_beside_launches(cuda, native):
    import torch
    p = Plan(cuda, 9)
    p.batch.run(p.values, p.queries[0], out_idx=p.outs[0][0], values=False)
    torch.cuda.synchronize()
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for r in range(3):
            p.launch(0, r, "run", None)
        p.launch(0, 3, "query", None)
    for r in range(ROUNDS):
        with torch.cuda.stream(s):
            g.replay()
        p.launch(1, r, "run" if r % 2 else "query", t)
    for r in range(4, ROUNDS):
        p.launch(0, r, "run", s)
    torch.cuda.synchronize()
    p.check()


def test_plan_without_queries(cuda, native):
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    A = torch.rand(1000, device=cuda)
    Q = torch.empty((0, 2), dtype=torch.int32, device=cuda)
    with RMQBatch([0], [1000], [0], [0]) as b:
        b.build(A)
        v, i = b.query(A, Q)
        assert len(v) == 0 and len(i) == 0
        torch.cuda.synchronize()
