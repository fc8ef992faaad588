"""GPU: the batch plan's work items follow the plan's size, from one unit of
256 micro-blocks and one step of queries an item in a small plan to the largest
runs. Arrays that overlap in one buffer, so that few values make a large plan,
against a host sparse table: exact."""
import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("narrays", [1, 40, 160, 800])
@pytest.mark.parametrize("per_array", [3, 2000])
def test_items_of_every_size(cuda, native, narrays, per_array):
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    rng = np.random.default_rng(narrays)
    A = rng.integers(0, 50_000, 262_144 + 64).astype(np.float32)
    starts = rng.integers(0, 64, narrays)
    lengths = 262_144 - rng.integers(0, 3, narrays) * 8191
    first, n = np.repeat(starts, per_array), np.repeat(lengths, per_array)
    w = np.maximum(np.exp(rng.uniform(0, np.log(n))).astype(np.int64), 1)
    w[::per_array] = lengths  # the whole array
    l = (rng.random(len(n)) * (n - w + 1)).astype(np.int64)
    Q = np.stack([l, l + w - 1], 1)
    m = range_min(composites(A), Q[:, 0] + first, Q[:, 1] + first)
    ei = ((m & np.uint64(0xffffffff)).astype(np.int64) >> 1) - first
    dA, dQ = torch.from_numpy(A).to(cuda), torch.from_numpy(Q.astype(np.int32)).to(cuda)
    qstarts = np.arange(narrays, dtype=np.int64) * per_array
    with RMQBatch(starts, lengths, qstarts, np.full(narrays, per_array)) as b:
        v, i = b.run(dA, dQ)
        np.testing.assert_array_equal(i.cpu().numpy(), ei)
        np.testing.assert_array_equal(v.cpu().numpy(), A[ei + first])
