"""GPU: the plain table index chooses its blocks by the number of elements: a
table of small blocks, from 2^13 blocks on a second one over larger blocks
for long ranges, the micro table for ranges of up to 64 micro-blocks. Ranges
at the edges of those rules (one micro-block around the micro table's window,
around the distance from which the larger blocks serve, ends on and beside
block borders, up to the last, partial block), at element counts around the
ones where a rule changes, against a host sparse table: exact, whatever block
size is asked for. The counts of rmq_query_stats belong to that block size."""
import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu


def blocks_of(n):
    """(block, larger block or 0) of the index of n elements."""
    b = 64
    while b < 512 and n // (2 * b) >= 8192:
        b *= 2
    c = 0
    if n // b >= 8192:
        c = 2 * b
        while n // c >= 8192:
            c *= 2
    return b, c


def ranges(n, rng):
    b, c = blocks_of(n)
    widths = [1, 32, 33, 31 * 32, 63 * 32, 64 * 32, 65 * 32, 127 * 32, 128 * 32, 2 * b, 5 * b]
    if c:
        widths += [k * c for k in (1, 2, 63, 64, 65, 130, 1000)]
    widths += [n // 3, n - 100, n]
    out = []
    for w in widths:
        for d in (-33, -1, 0, 1, 31):
            size = min(max(w + d, 1), n)
            for edge in (32, b, c or 1):
                l = rng.integers(0, n - size + 1, 24) // edge * edge + rng.integers(-1, 2, 24)
                out.append(np.stack([np.clip(l, 0, n - size), np.clip(l, 0, n - size) + size - 1], 1))
            out.append(np.array([[0, size - 1], [n - size, n - 1]]))
    return np.concatenate(out)


@pytest.mark.parametrize("n", [999, 8192 * 64 - 1, 8192 * 64, 8192 * 128 + 31, 8192 * 512 - 33, 8192 * 512 + 1,
                               8192 * 1024 + 65, 20_000_003])
@pytest.mark.parametrize("kind", ["ties", "normal"])
def test_index_shapes(cuda, native, n, kind):
    import torch

    import rtxrmq_gb300 as R
    rng = np.random.default_rng(n)
    A = (rng.integers(0, 3, n) if kind == "ties" else rng.standard_normal(n)).astype(np.float32)
    if kind == "normal":  # large blocks' bests outside the ranges
        A[rng.integers(0, n, n // 700 + 1)] -= 50.0
    Q = ranges(n, rng)
    m = range_min(composites(A), Q[:, 0], Q[:, 1])
    ei = (m & np.uint64(0xffffffff)).astype(np.int64) >> 1
    dA, dQ = torch.from_numpy(A).to(cuda), torch.from_numpy(Q.astype(np.int32)).to(cuda)
    for bs in (0, 128, 1000, 1 << 15):
        with R.RMQIndex(dA, min(bs, n)) as ix:
            v, i = ix.query(dQ)
            st = ix.query_stats(dQ)
            np.testing.assert_array_equal(i.cpu().numpy(), ei)
            np.testing.assert_array_equal(v.cpu().numpy(), A[ei])
            assert sum(st[k] for k in ("first_probe", "second_probe", "full", "micro_scan")) == len(Q)


@pytest.mark.parametrize("n", [8192 * 512 + 1, 1 << 23])
@pytest.mark.parametrize("levels", [2, 256, 4096])
@pytest.mark.parametrize("op", ["min", "max"])
def test_long_ranges_of_few_values(cuda, native, n, levels, op):
    """Nearly every probe finds the best value left of the range: answered by
    the micro-blocks from l's on, or not when the value only comes later."""
    import torch

    import rtxrmq_gb300 as R
    rng = np.random.default_rng(levels)
    A = rng.integers(0, levels, n).astype(np.float32)
    A[n // 2:n // 2 + 300_000] = np.where(rng.random(300_000) < 1e-4, 0.0, 5.0)  # rare least values
    size = np.exp(rng.uniform(np.log(2000), np.log(n), 40_000)).astype(np.int64)
    l = (rng.random(40_000) * (n - size + 1)).astype(np.int64)
    l[::3] = n // 2 + rng.integers(0, 200_000, len(l[::3]))
    size = np.minimum(size, n - l)
    Q = np.stack([l, l + size - 1], 1)
    B = A if op == "min" else -A  # the leftmost largest is the leftmost least of -A
    m = range_min(composites(B + 0.0), Q[:, 0], Q[:, 1])
    ei = (m & np.uint64(0xffffffff)).astype(np.int64) >> 1
    with R.RMQIndex(torch.from_numpy(A).to(cuda), op=op) as ix:
        v, i = ix.query(torch.from_numpy(Q.astype(np.int32)).to(cuda))
        np.testing.assert_array_equal(i.cpu().numpy(), ei)
        np.testing.assert_array_equal(v.cpu().numpy(), A[ei])
