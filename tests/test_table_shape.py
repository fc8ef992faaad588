"""Every query of a table index fits the table it is sent to: a range whose end
micro-blocks are fewer than micro_span apart goes through the micro table,
which must hold windows that long, and any other range must have its ends in
different blocks (what settles open ranges adds the parts of two end blocks).
So a block holds at most micro_span micro-blocks. Checked on the host over the
classes of element counts and block sizes; on the GPU, exactly, where a block is
one micro-block wider than 511: ranges from the first to the last micro-block of
a block, with the block's best just outside of them."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_gpu_stats import composites, range_min

ROOT = Path(__file__).resolve().parent.parent

SHAPE_TEST = r"""
#include <cstdio>
#include <vector>
#include "engine.h"
using namespace rmq;
static std::vector<uint32_t> around(uint32_t most) {
  std::vector<uint32_t> v;
  for (uint32_t k = 0; k < 31; ++k)
    for (uint64_t f : {4, 5, 6, 7})
      for (int64_t d : {-33, -1, 0, 1, 33}) {
        const int64_t x = static_cast<int64_t>((f << k) / 4) + d;
        if (x >= 1 && x <= most) v.push_back(static_cast<uint32_t>(x));
      }
  v.push_back(most);
  return v;
}
int main() {
  long bad = 0;
  for (uint32_t n : around(0x7fffffffu)) {
    const bool wide = wide_masks((n + kMicro - 1) / kMicro);
    const IndexShape x = index_shape(n);
    // two windows of the masks' 2^(levels - 1) cover micro_span micro-blocks
    if (x.tbs < 64 || x.tbs % kMicro || x.tbs / kMicro > x.micro_span ||
        x.micro_span > (wide ? 64u : 63u) || (x.cbs && x.cbs % x.tbs)) {
      std::printf("index n=%u tbs=%u span=%u\n", n, x.tbs, x.micro_span);
      ++bad;
    }
    for (uint32_t bs : around(0x7fffffffu)) {
      const TableShape t = table_shape(n, bs < n ? bs : n);
      // rows are made for windows of up to 1024 micro-blocks, offsets of two bytes
      if (t.tbs < 64 || t.tbs % kMicro || t.tbs / kMicro > (1u << t.mlevels) - 1u || t.mlevels > 11 ||
          micro_offset_bytes(t.mlevels) > 2) {
        if (++bad < 20) std::printf("n=%u bs=%u: tbs=%u mlevels=%u\n", n, bs, t.tbs, t.mlevels);
      }
    }
  }
  std::printf(bad ? "%ld bad\n" : "ok\n", bad);
  return bad != 0;
}
"""


def test_blocks_fit_the_micro_table(tmp_path):
    src = tmp_path / "shape.cpp"
    src.write_text(SHAPE_TEST)
    exe = tmp_path / "shape"
    r = subprocess.run(["g++", "-O2", "-std=c++17", f"-I{ROOT / 'rtxrmq_gb300' / 'csrc'}",
                        "-I/usr/local/cuda/include", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


def fringe_case(n, lead):
    """Values and ranges of one array: per block of 2^14 positions (counted from
    `lead` elements before the array's first), the least values lie in the
    block's first and last micro-block, and the ranges run from the first to the
    last micro-block between them, around them, and beyond."""
    rng = np.random.default_rng(n + lead)
    A = (rng.integers(1000, 2000, n)).astype(np.float32)
    Q = []
    for b, at in enumerate(range(-lead, n, 1 << 14)):
        lo, hi = max(at, 0), min(at + (1 << 14), n) - 1
        a, z = lo + 3, hi - 3
        if z - a < 64:
            continue
        A[a], A[z] = (1 + b % 3, 2 + b % 2) if b % 2 else (2 + b % 2, 1 + b % 3)
        for l in (lo, a, a + 1, a + 9, lo + 31 if lo + 31 > a else a + 1):
            for r in (hi, z, z - 1, z - 9, hi - 31):
                Q.append((l, r))
        Q += [(lo + 32, hi - 32), (lo + 32, z - 1), (a + 1, hi - 32), (a + 1, min(z + 4000, n - 1)),
              (max(a - 4000, 0), z - 1)]
    l = rng.integers(0, n - 20_000, 4000)
    w = rng.integers(510 * 32, 514 * 32, 4000)
    Q = np.concatenate([np.array(Q), np.stack([l, np.minimum(l + w, n) - 1], 1)])
    m = range_min(composites(A), Q[:, 0], Q[:, 1])
    return A, Q.astype(np.int32), ((m & np.uint64(0xffffffff)).astype(np.int64) >> 1)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [16384, 16416, 20000, 32768])
@pytest.mark.parametrize("lead", [0, 5])
def test_widest_blocks_of_a_batch(cuda, native, bs, lead):
    import torch

    from rtxrmq_gb300.batch import RMQBatch
    cases = [fringe_case(n, lead) for n in (1 << 19, 600_000, (1 << 20) - 33)]
    starts, parts, at = [], [], 0
    for A, _, _ in cases:
        start = (at + 31) // 32 * 32 + lead
        parts += [np.full(start - at, -1e9, np.float32), A]  # less than every value
        starts.append(start)
        at = start + len(A)
    V = np.concatenate(parts)
    Q = np.concatenate([c[1] for c in cases])
    ei = np.concatenate([c[2] for c in cases])
    ev = np.concatenate([c[0][c[2]] for c in cases])
    qcounts = np.array([len(c[1]) for c in cases])
    qstarts = np.cumsum(qcounts) - qcounts
    dV, dQ = torch.from_numpy(V).to(cuda), torch.from_numpy(Q).to(cuda)
    with RMQBatch(starts, [len(c[0]) for c in cases], qstarts, qcounts, [bs] * 32) as b:
        runs = [b.run(dV, dQ)]
        runs.append(b.query(dV, dQ))
        runs.append(b.run_per_array(dV, dQ))
        for v, i in runs:
            np.testing.assert_array_equal(i.cpu().numpy(), ei)
            np.testing.assert_array_equal(v.cpu().numpy(), ev)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [0, 16416, 20000, 32768])
@pytest.mark.parametrize("n", [1 << 19, 600_000, (1 << 20) - 33])
def test_widest_blocks_of_the_counting_launch(cuda, native, bs, n):
    import torch

    import rtxrmq_gb300 as R
    A, Q, ei = fringe_case(n, 0)
    dA, dQ = torch.from_numpy(A).to(cuda), torch.from_numpy(Q).to(cuda)
    v = torch.empty(len(Q), dtype=torch.float32, device=cuda)
    i = torch.empty(len(Q), dtype=torch.int32, device=cuda)
    with R.RMQIndex(dA, bs) as ix:
        st = ix.query_stats(dQ, out_val=v, out_idx=i)
        np.testing.assert_array_equal(i.cpu().numpy(), ei)
        np.testing.assert_array_equal(v.cpu().numpy(), A[ei])
        assert sum(st[k] for k in ("first_probe", "second_probe", "full", "micro_scan")) == len(Q)
        assert st["full"] > 0
        q = ix.query(dQ)
        np.testing.assert_array_equal(q[1].cpu().numpy(), ei)
