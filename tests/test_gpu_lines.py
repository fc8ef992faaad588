"""GPU: queries settled from one 32-element line of values by the warp (8
lanes per query), where that can go wrong: lines cut by the array's end,
values off a 16-byte boundary, query counts around a warp and a step, lines
holding only NaN or only the key order's largest value (the first element of
the range, not of the line, is the answer), signed zeros. Exact against the
engine's key order, no tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys(A, op):
    """uint32 keys in the engine's order (smallest = best)."""
    if A.dtype == np.int32:
        return A.view(np.uint32) ^ np.uint32(0x80000000 if op == "min" else 0x7fffffff)
    from test_gpu_light import key_order
    return key_order(A.view(np.uint32), op)


def want(A, Q, op):
    k = keys(A, op)
    ei = np.array([l + int(np.argmin(k[l:r + 1])) for l, r in Q], dtype=np.int32)
    ev = A.view(np.uint32)[ei].copy()
    if A.dtype == np.float32:
        ev[k[ei] == np.uint32(0xffffffff)] = 0x7fc00000
    return ev, ei


def line_values(kind, n):
    rng = np.random.default_rng(n)
    if kind == "int":
        A = rng.integers(-3, 3, n).astype(np.int32)
        A[: n // 2] = rng.choice([2**31 - 1, -2**31], n // 2)
        A[n // 4: n // 3] = 2**31 - 1
        return A
    A = rng.integers(-2, 3, n).astype(np.float32)
    A[rng.random(n) < 0.3] = -0.0
    b = A.view(np.uint32)
    b[: n // 2] = rng.choice(np.array([0x7fc00000, 0xffbfffff, 0x7f800001], np.uint32), n // 2)
    A[rng.integers(0, n, n // 8)] = np.inf
    return A


@pytest.mark.parametrize("kind", ["float", "int"])
@pytest.mark.parametrize("op", ["min", "max"])
@pytest.mark.parametrize("light", [False, True])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_line_queries(cuda, native, kind, op, light, off):
    import torch

    import rtxrmq_gb300 as R
    for n in (64, 95, 97, 1030):
        A = line_values(kind, n)
        big = torch.from_numpy(np.concatenate([np.zeros(off, A.dtype), A])).to(cuda)
        pairs = [(l, r) for l in range(n) for r in range(l, min(n, l + 70))]
        Q = np.array(pairs, np.int32)
        Q = Q[np.random.default_rng(1).permutation(len(Q))]
        ev, ei = want(A, Q, op)
        with R.RMQIndex(big[off:off + n], 64, op=op, light=light) as ix:
            for q in (1, 31, 32, 33, 511, 513, len(Q)):
                v, i = ix.query(torch.from_numpy(Q[-q:].copy()).to(cuda))
                np.testing.assert_array_equal(i.cpu().numpy(), ei[-q:])
                np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), ev[-q:])
            assert ix.invalid_count() == 0
