"""GPU: the micro table (masks of the windows of up to 32 micro-blocks, rows
of offsets above) where it can go wrong: windows of 31 .. 65 micro-blocks and
around every further power of two, starting and ending at the edges of the
builder's tiles (256, 1024 and 2048 positions) and of the array, block sizes
with no row, 1-byte and 2-byte rows, blocks above 2^15 (answered through
smaller ones) and block sizes that are not multiples of 32; ties. Exact
against a host sparse table over the engine's composites."""
import struct

import numpy as np
import pytest

from test_gpu_stats import composites, range_min

pytestmark = pytest.mark.gpu


def window_queries(n, widths, edges, rng):
    """Queries over `w` micro-blocks that start or end at micro-block `e` + a
    few, at random elements of their end micro-blocks."""
    nm = (n + 31) // 32
    out = []
    for w in widths:
        for e in edges:
            for d in range(-3, 4):
                for ml in (e + d, e + d - w + 1):
                    mr = ml + w - 1
                    if 0 <= ml and mr < nm:
                        a, b = rng.integers(0, 32, 2)
                        l, r = 32 * ml + a, min(32 * mr + b, n - 1)
                        if l <= r:
                            out.append((l, r))
    return np.array(out, np.int32)


@pytest.mark.parametrize("n,edges", [(32 * 1024 + 5, (0, 256, 512, 1024)),
                                     (32 * 160_000 + 31, (0, 1024, 2048, 4096, 159_999))])
@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("bs", [33, 64, 1000, 1024, 2048, 4096, 12207, 1 << 14, 1 << 15, 1 << 16])
def test_windows(cuda, native, n, edges, ties, bs):
    import torch

    import rtxrmq_gb300 as R
    rng = np.random.default_rng(bs)
    A = (rng.integers(0, 3, n) if ties else rng.standard_normal(n)).astype(np.float32)
    widths = [1, 2, 3, 16, 31, 32, 33, 34, 47, 62, 63, 64, 65, 66, 100, 127, 128, 129, 255, 256, 257,
              511, 513, 1023, 1024, 1025, 2047]
    Q = window_queries(n, widths, edges, rng)
    m = range_min(composites(A), Q[:, 0].astype(np.int64), Q[:, 1].astype(np.int64))
    ei = (m & np.uint64(0xffffffff)).astype(np.int64) >> 1
    with R.RMQIndex(torch.from_numpy(A).to(cuda), bs) as ix:
        v, i = ix.query(torch.from_numpy(Q).to(cuda))
        v, i = v.cpu().numpy(), i.cpu().numpy()
    bad = np.nonzero(i != ei)[0]
    assert bad.size == 0, f"{bad.size} wrong, first {tuple(Q[bad[0]])}: {i[bad[0]]} not {ei[bad[0]]}"
    np.testing.assert_array_equal(v.view(np.uint32), A[ei].view(np.uint32))


def mix64(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def as_version_5(raw, n, bs, light, micro):
    """The bytes of a version-5 file for the index whose file is `raw`: its
    header fields and payload size, with a payload that is not an index."""
    def ilog2(x):
        return int(x).bit_length() - 1

    def pad(x):
        return (x + 255) // 256 * 256
    touched = bs // 32 if bs % 32 == 0 else (bs + 30) // 32 + 1
    mlev = ilog2(touched) + 1 if micro and bs >= 64 else 0
    nm = (n + 31) // 32 if mlev else 0
    nb = (n + bs - 1) // bs
    levels = ilog2(nb) + 1
    ent = 0 if light else pad(8 * n)
    size = 2 * ent + pad(8 * nb * levels) + 256
    if mlev:
        width = 1 if mlev <= 9 else 2 if mlev <= 17 else 4
        size += pad(8 * nm) + 2 * ent + pad(width * nm * (mlev - 1))
    flags = struct.unpack_from("<I", raw, 20)[0] & ~1 | (0 if mlev else 1)
    head = raw[:16] + struct.pack("<II7Q", 5, flags, n, bs, nb, levels, nm, mlev, size) + raw[80:88]
    x = 0
    for byte in head:
        x = mix64(x ^ byte)
    return head + struct.pack("<Q", x) + bytes(size)


@pytest.mark.parametrize("bs,light,micro", [(1024, False, True), (1000, False, True), (40, False, True),
                                            (70_000, False, True), (1024, False, False), (2048, True, True)])
def test_version_5_files(cuda, native, oracle_lib, tmp_path, bs, light, micro):
    """Files of version 5 load: layout, values and length are checked as
    before, and the index answers."""
    import torch

    import rtxrmq_gb300 as R
    n = 100_003
    A = R.gen_values_int(n, 500, 3)
    Q = np.concatenate([R.gen_queries(5000, n, L, 4) for L in (-1, -3, 20)])
    dA = torch.from_numpy(A).to(cuda)
    path = tmp_path / "ix"
    with R.RMQIndex(dA, bs, light=light, micro=micro) as ix:
        ix.save(path)
        info = ix.info()
    old = as_version_5(path.read_bytes(), n, bs, light, micro)
    path.write_bytes(old)
    with R.RMQIndex.load(dA, path) as ix:
        v, i = ix.query(torch.from_numpy(Q).to(cuda))
        np.testing.assert_array_equal(i.cpu().numpy(), oracle_lib.base_idx(A, Q))
        assert ix.info()["bs"] == info["bs"] and ix.info()["light"] == info["light"]
    path.write_bytes(old[:-1])
    with pytest.raises(R.RMQError, match="truncated"):
        R.RMQIndex.load(dA, path)
    path.write_bytes(old)
    with pytest.raises(R.RMQError, match="values differ"):
        R.RMQIndex.load(dA + 1, path)


def test_noalloc_limits(cuda, native):
    """The sizes rmq_query_noalloc refuses are those of an index with
    per-element entries, whatever the table index needs."""
    import torch
    n_max = (32 << 20) // 16 - 2048
    dA = torch.rand(n_max + 4096, device=cuda)
    dQ = torch.tensor([[5, 500]], dtype=torch.int32, device=cuda)
    out = torch.empty(1, dtype=torch.int32, device=cuda)
    s = torch.cuda.current_stream().cuda_stream
    for n, bs, rc in ((n_max, 1 << 15, 0), (n_max + 4096, 1 << 15, -1), (1_000_000, 1, -1), (150_000, 1, 0)):
        assert native.rmq_query_noalloc(dA.data_ptr(), n, bs, dQ.data_ptr(), 1, None, out.data_ptr(), s) == rc
        if rc == 0:
            assert out.item() == 5 + int(dA[5:501].argmin())


def test_probe_gather_capture(cuda, native):
    """rmq_probe_gather's first call on a table index builds its entries, also
    inside a stream capture; the captured probe answers on every replay."""
    import torch

    import rtxrmq_gb300 as R
    n, bs = 50_000, 1000
    A = torch.rand(n, device=cuda)
    l = torch.randint(0, n - 2 * bs, (3000,), device=cuda, dtype=torch.int32)
    Q = torch.stack((l, (l // bs + 1) * bs + 7), 1).to(torch.int32)  # adjacent blocks
    with R.RMQIndex(A, bs) as ix, R.RMQIndex(A, bs) as warm:
        _, want = warm.probe_gather(Q)
        v = torch.empty(len(Q), device=cuda)
        i = torch.empty(len(Q), dtype=torch.int32, device=cuda)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ix.probe_gather(Q, v, i)
        for _ in range(2):
            i.zero_()
            g.replay()
            assert torch.equal(i, want)
        assert torch.equal(ix.probe_gather(Q)[1], want)
        assert torch.equal(ix.query(Q)[1], want)
