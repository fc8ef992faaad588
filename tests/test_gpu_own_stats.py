"""GPU: rmq_query_stats_ex with RMQ_STATS_OWN_TABLES counts on the tables that
rmq_query reads, whatever block size the index was asked for: the counts follow a
host model of those tables (micro-blocks for ranges of up to 64, blocks chosen by the
number of elements, larger blocks for long ranges), differ from the ones in blocks
of bs, and come with the same answers. Unknown flags are refused."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_shapes import blocks_of
from test_gpu_stats import composites, range_min, unit_minima

pytestmark = pytest.mark.gpu


def first_probes(A, Q):
    """(settled by the first probe, inside one micro-block) of an index of
    len(A) elements."""
    C_ = composites(A)
    l, r = Q[:, 0].astype(np.int64), Q[:, 1].astype(np.int64)
    b, c = blocks_of(len(A))
    d = r // 32 - l // 32
    scan, micro = d == 0, (d > 0) & (d < 64)
    coarse = (d >= 64 * (c // 32)) if c else np.zeros(len(Q), bool)
    first = 0
    for which, width in ((micro, 32), (~scan & ~micro & ~coarse, b), (~scan & ~micro & coarse, c)):
        if which.any():
            m = range_min(unit_minima(C_, width), l[which] // width, r[which] // width)
            i = (m & np.uint64(0xffffffff)).astype(np.int64) >> 1
            first += int(((i >= l[which]) & (i <= r[which])).sum())
    return first, int(scan.sum())


@pytest.mark.parametrize("n", [100_003, (1 << 20) + 9, (1 << 22) + 77, 9_000_001])
@pytest.mark.parametrize("lr", [-1, -2, -3, 8])
@pytest.mark.parametrize("light", [False, True])
def test_own_tables(cuda, native, n, lr, light):
    import torch

    import rtxrmq_gb300 as R
    q = 1 << 15
    A, Q = R.gen_values_uniform(n, 31), R.gen_queries(q, n, lr, 32)
    Q[:2] = [[3, 2], [0, n]]  # invalid
    dA, dQ = torch.from_numpy(A).to(cuda), torch.from_numpy(Q).to(cuda)
    v = torch.empty(q, dtype=torch.float32, device=cuda)
    i = torch.empty(q, dtype=torch.int32, device=cuda)
    with R.RMQIndex(dA, 1 << 15, light=light) as ix:
        st = ix.query_stats(dQ, out_val=v, out_idx=i, own=True)
        v2, i2 = ix.query(dQ)
        np.testing.assert_array_equal(i.cpu().numpy(), i2.cpu().numpy())
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), v2.cpu().numpy().view(np.uint32))
        asked = ix.query_stats(dQ)
    first, scans = first_probes(A, Q[2:])
    assert (st["first_probe"], st["micro_scan"], st["invalid"]) == (first, scans, 2), st
    assert st["first_probe"] + st["second_probe"] + st["full"] + scans + 2 == q, st
    assert st["entries"] == st["warp_scan"] == st["block_edge"] == 0, st
    # a line of at most four sectors per end part, one to two per range of 8
    ends = st["second_probe"] + 2 * st["full"]
    assert ends + scans <= st["scan_sectors"] <= 4 * ends + (2 if lr == 8 else 4) * scans, st
    if lr == -1 and n > 1 << 20:
        assert st["first_probe"] != asked["first_probe"]


def test_flags(cuda, native):
    import torch

    import rtxrmq_gb300 as R
    A = torch.rand(1000, device=cuda)
    Q = torch.tensor([[0, 999]], dtype=torch.int32, device=cuda)
    counts = (C.c_int64 * 10)()
    with R.RMQIndex(A) as ix:
        s = torch.cuda.current_stream().cuda_stream
        call = native.rmq_query_stats_ex
        assert call(ix.handle, Q.data_ptr(), 1, None, None, C.addressof(counts), 2, s) == -1
        assert call(ix.handle, Q.data_ptr(), 1, None, None, C.addressof(counts), 1, s) == 0
        assert sum(counts[:4]) == 1
    with R.RMQIndex(A, 100, micro=False) as ix:  # its tables are the ones asked for
        assert ix.query_stats(Q, own=True) == ix.query_stats(Q)
