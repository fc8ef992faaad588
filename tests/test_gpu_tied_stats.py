"""GPU: what rmq_query_stats counts of ranges tied with the start of their block.
Values 0 and 1, ranges of several blocks that begin on a micro-block in the middle
of a block: the leftmost 0 of l's block lies before l, and the micro-blocks from l's
on begin with the answer, so that one mask settles every query and no end part is
read. Beside them ranges that the same warps settle by end parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1 << 22, (1 << 20) + 77])
@pytest.mark.parametrize("light", [False, True])
def test_tied_queries_read_no_end_part(cuda, native, n, light):
    import torch

    import rtxrmq_gb300 as R
    bs, q = 4096, 4096
    rng = np.random.default_rng(n)
    A = rng.integers(0, 2, n).astype(np.float32)
    l = rng.integers(0, n // bs - 10, q) * bs + 2048 + 32 * rng.integers(0, 32, q)
    r = l + 5 * bs + rng.integers(0, 100, q)
    Q = np.stack([l, r], 1).astype(np.int32)
    zeros = np.flatnonzero(A == 0)
    want = zeros[np.searchsorted(zeros, l)]
    dA, dQ = torch.from_numpy(A).to(cuda), torch.from_numpy(Q).to(cuda)
    v = torch.empty(q, dtype=torch.float32, device=cuda)
    i = torch.empty(q, dtype=torch.int32, device=cuda)
    with R.RMQIndex(dA, bs, light=light) as ix:
        st = ix.query_stats(dQ, out_val=v, out_idx=i)
        np.testing.assert_array_equal(i.cpu().numpy(), want)
        assert st["second_probe"] == q and st["first_probe"] == st["full"] == 0, st
        assert st["entries"] == 0 and st["scan_sectors"] == 0, st
        assert st["table_words"] == 4 * q, st  # the blocks' two, mask and minimum
