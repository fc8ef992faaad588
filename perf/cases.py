"""Workloads that the engine's speed is judged on, through its public entry points.

A case is one call pattern of a user's program, with its sizes:

  query    queries in device memory against an index that is kept (RMQIndex.query)
  oneshot  index construction, one query batch, release (a new array per call,
           as rtx_rmq and the reference's command line use it)
  host     queries and results in pinned host memory (RMQIndex.query_host)
  batch    many arrays of uneven length, built and answered together (RMQBatch.run)
  grad     differentiable range minimum over ragged rows, forward and backward

Query lengths: "uniform" in [1, n], "medium" lognormal(0.6 ln n, 0.3), "short"
lognormal(0.3 ln n, 0.3) (the reference's three length modes), "ragged"
lognormal(0.5 ln n, 0.4), "rows" lognormal(0.4 ln n, 0.5), or a fixed number.
Values: "unit" uniform in [0, 1), "normal" N(0, 1), "ties" integers in [0, 256),
"int32" over the whole range of the type.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

import rtxrmq_gb300 as R
from rtxrmq_gb300.autograd import RaggedRangeMin
from rtxrmq_gb300.batch import RMQBatch

MU_SIGMA = {"medium": (0.6, 0.3), "short": (0.3, 0.3), "ragged": (0.5, 0.4), "rows": (0.4, 0.5)}


def listed():
    return [
        # a small array answered once: a service call where launches and
        # allocation count; block size left at the default (2^15)
        dict(name="oneshot_small", kind="oneshot", n=100_000, q=1024, length="uniform", bs=0,
             values="unit", op="min", light=False),
        # the plain workload that also runs on a CPU: n = 10^6, q = 2^20,
        # short ranges
        dict(name="query_1e6_short", kind="query", n=1_000_000, q=1 << 20, length="short",
             bs=1024, values="unit", op="min", light=False),
        # the headline: n = 10^8, q = 2^26, uniform lengths, default block size
        dict(name="query_1e8_uniform", kind="query", n=100_000_000, q=1 << 26, length="uniform",
             bs=0, values="unit", op="min", light=False),
        # the headline's medium lengths at the reference's own block count
        # (--nb 512) and an odd number of elements
        dict(name="query_1e8_medium", kind="query", n=99_999_989, q=1 << 26, length="medium",
             bs=99_999_989 // 512, values="unit", op="min", light=False),
        # the headline's short lengths at the reference's --nb 8192
        dict(name="query_1e8_short", kind="query", n=100_000_000, q=1 << 26, length="short",
             bs=100_000_000 // 8192, values="unit", op="min", light=False),
        # many equal minima, ranges of 32: most ranges straddle two 32-element lines
        dict(name="query_ties_len32", kind="query", n=1 << 27, q=1 << 26, length=32, bs=4096,
             values="ties", op="min", light=False),
        # a new large array per call: construction dominates
        dict(name="oneshot_1e8", kind="oneshot", n=100_000_000, q=1 << 22, length="medium", bs=0,
             values="unit", op="min", light=False),
        # the same with the light index, int32 values, range maximum, odd size
        dict(name="oneshot_light_int32", kind="oneshot", n=(1 << 26) + 13, q=1 << 22,
             length="short", bs=4096, values="int32", op="max", light=True),
        # queries from a host program over the host link
        dict(name="host_1e8_uniform", kind="host", n=100_000_000, q=1 << 24, length="uniform",
             bs=0, values="unit", op="min", light=False),
        # the ragged batch: 4096 arrays of 2^8 .. 2^22 elements, 2^26 queries
        dict(name="batch_full", kind="batch", arrays=4096, umin=8.0, umax=22.0, q=1 << 26,
             align=4, values="unit", op="min", light=False),
        dict(name="batch_light", kind="batch", arrays=4096, umin=8.0, umax=22.0, q=1 << 26,
             align=4, values="unit", op="min", light=True),
        # differentiable range minimum: 256 rows of 2^14 .. 2^20, 2^16 ranges per row
        dict(name="grad_rows", kind="grad", rows=256, lmin=1 << 14, lmax=1 << 20, per_row=1 << 16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query"] * 5 + ["oneshot"] * 3 + ["batch"] * 2 + ["grad", "host"])
    if kind == "batch":
        umin = rng.uniform(3.0, 10.0)
        return dict(kind=kind, arrays=_log_int(rng, 8, 4096), umin=umin,
                    umax=umin + rng.uniform(2.0, 12.0), q=_log_int(rng, 1000, 1 << 26),
                    align=rng.choice([1, 4, 4]), values=rng.choice(["unit", "ties", "int32"]),
                    op=rng.choice(["min", "max"]), light=rng.random() < 0.5)
    if kind == "grad":
        lmin = _log_int(rng, 16, 1 << 14)
        return dict(kind=kind, rows=_log_int(rng, 4, 256), lmin=lmin,
                    lmax=lmin * _log_int(rng, 2, 64), per_row=_log_int(rng, 16, 1 << 16))
    n = _log_int(rng, 1000, 100_000_000)
    q = _log_int(rng, 1, 1 << (26 if kind == "query" else 22 if kind == "oneshot" else 24))
    length = rng.choice(["uniform", "medium", "short", _log_int(rng, 1, n)])
    light = rng.random() < 0.25
    bs = rng.choice([0, 1 << rng.randint(7, 16), 32 * rng.randint(2, 3000)])
    if not light and rng.random() < 0.3:
        bs = max(1, n // rng.choice([512, 8192]))  # the reference's block counts
    if light and 0 < n < bs:
        bs = 0
    return dict(kind=kind, n=n, q=q, length=length, bs=bs,
                values=rng.choice(["unit", "unit", "normal", "ties", "int32"]),
                op=rng.choice(["min", "min", "max"]), light=light)


# ---- inputs ----

def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + salt) % (1 << 62))


def _values(kind, n, seed):
    g = _gen(seed, 1)
    if kind == "normal":
        return torch.randn(n, device="cuda", generator=g)
    if kind == "ties":
        return torch.randint(0, 256, (n,), device="cuda", generator=g, dtype=torch.int32).float()
    if kind == "int32":
        return torch.randint(-2**31, 2**31 - 1, (n,), device="cuda", generator=g, dtype=torch.int32)
    return torch.rand(n, device="cuda", generator=g)


def _ranges(length, n, q, g):
    """int32 [q, 2] inclusive ranges inside arrays of n elements (a number, or
    one per query as float64)."""
    n = torch.as_tensor(n, dtype=torch.float64, device="cuda")
    u = torch.rand(q, device="cuda", generator=g, dtype=torch.float64)
    if length == "uniform":
        size = 1 + torch.floor(u * n)
    elif isinstance(length, str):
        mu, sigma = MU_SIGMA[length]
        z = torch.randn(q, device="cuda", generator=g, dtype=torch.float64)
        size = torch.round(torch.exp(mu * torch.log(n) + sigma * z))
    else:
        size = torch.full((q,), float(length), device="cuda", dtype=torch.float64)
    size = torch.minimum(size.clamp_(min=1), n)
    u = torch.rand(q, device="cuda", generator=g, dtype=torch.float64)
    left = torch.minimum(torch.floor(u * (n - size + 1)), n - size)
    return torch.stack((left, left + size - 1), 1).to(torch.int32)


def _layout(case):
    """Host arrays (starts, lengths, qstarts, qcounts) of a batch or of rows: a
    plan's fixed layout, the same for every set of values and queries."""
    rng = np.random.default_rng(1321)
    if case["kind"] == "grad":
        lengths = rng.integers(case["lmin"], case["lmax"] + 1, case["rows"]).astype(np.int64)
        qcounts = np.full(case["rows"], case["per_row"], np.int64)
        align = 1
    else:
        u = rng.uniform(case["umin"], case["umax"], case["arrays"])
        lengths = np.maximum(np.round(2.0 ** u), 1).astype(np.int64)
        share = lengths / lengths.sum() * case["q"]
        qcounts = np.floor(share).astype(np.int64)
        rest = case["q"] - int(qcounts.sum())
        qcounts[np.argsort(qcounts - share, kind="stable")[:rest]] += 1
        align = case["align"]
    padded = (lengths + align - 1) // align * align
    starts = np.concatenate([[0], np.cumsum(padded)[:-1]]).astype(np.int64)
    qstarts = np.concatenate([[0], np.cumsum(qcounts)[:-1]]).astype(np.int64)
    return starts, lengths, qstarts, qcounts


def _batch_inputs(case, seed):
    starts, lengths, qstarts, qcounts = lay = _layout(case)
    values = _values(case.get("values", "normal"), int(starts[-1] + lengths[-1]), seed)
    counts = torch.from_numpy(qcounts).cuda()
    per_query = torch.repeat_interleave(torch.from_numpy(lengths).cuda().double(), counts)
    length = "rows" if case["kind"] == "grad" else "ragged"
    queries = _ranges(length, per_query, int(qcounts.sum()), _gen(seed, 2))
    return lay, values, queries


def _plain_inputs(case, seed):
    return (_values(case["values"], case["n"], seed),
            _ranges(case["length"], case["n"], case["q"], _gen(seed, 2)))


def prepare(case, seed):
    s = SimpleNamespace(kind=case["kind"])
    if case["kind"] in ("batch", "grad"):
        lay, s.values, s.queries = _batch_inputs(case, seed)
        if case["kind"] == "grad":
            s.rows = RaggedRangeMin(lay[1], lay[3])
            s.values.requires_grad_(True)
            s.grad_out = torch.randn(len(s.queries), device="cuda", generator=_gen(seed, 3))
        else:
            s.plan = RMQBatch(*lay, op=case["op"], light=case["light"],
                              dtype="int32" if case["values"] == "int32" else "float32")
        return s
    s.values, s.queries = _plain_inputs(case, seed)
    s.options = dict(bs=case["bs"], op=case["op"], light=case["light"])
    if case["kind"] != "oneshot":
        s.index = R.RMQIndex(s.values, **s.options)
    if case["kind"] == "host":
        s.queries = s.queries.cpu().pin_memory()
        s.out = (torch.empty(case["q"], dtype=s.values.dtype, pin_memory=True),
                 torch.empty(case["q"], dtype=torch.int32, pin_memory=True))
    return s


def run(s):
    if s.kind == "query":
        return s.index.query(s.queries)
    if s.kind == "oneshot":
        with R.RMQIndex(s.values, **s.options) as index:
            return index.query(s.queries)
    if s.kind == "host":
        s.index.query_host(s.queries, *s.out)
        torch.cuda.current_stream().synchronize()  # the host reads the results
        return s.out
    if s.kind == "batch":
        return s.plan.run(s.values, s.queries)
    best, where = s.rows(s.values, s.queries)
    grad, = torch.autograd.grad(best, s.values, s.grad_out)
    return best.detach(), where, grad


def work(case):
    """Every value of a new array once, 8 bytes in and 8 bytes out per query
    (against a kept index the queries and answers alone), no arithmetic but
    comparisons; backward: a gradient in per query, one out per value."""
    if case["kind"] in ("query", "host"):
        return {"bytes": 16 * case["q"], "flops": 0}
    if case["kind"] == "oneshot":
        return {"bytes": 4 * case["n"] + 16 * case["q"], "flops": 0}
    _, lengths, _, qcounts = _layout(case)
    n, q = int(lengths.sum()), int(qcounts.sum())
    if case["kind"] == "grad":
        return {"bytes": 8 * n + 20 * q, "flops": 0}
    return {"bytes": 4 * n + 16 * q, "flops": 0}


# ---- 64-bit answers in plain torch ----

def _range_best(values, left, right, largest):
    """(best value, its leftmost index) of every inclusive range, by windows of
    doubling length: two windows cover a range."""
    if largest:  # int32 has one more negative value than positive
        values = -values.long() if values.dtype == torch.int32 else -values
    best = values.clone()
    where = torch.arange(len(values), device="cuda", dtype=torch.int32)
    level = torch.floor(torch.log2((right - left + 1).double())).to(torch.int32)
    out = torch.empty(len(left), dtype=torch.float64 if values.is_floating_point() else torch.int64,
                      device="cuda")
    at = torch.empty(len(left), dtype=torch.int64, device="cuda")
    chunk = 1 << 27
    for k in range(int(level.max()) + 1 if len(left) else 0):
        if k:
            half = 1 << (k - 1)
            for c in range(0, len(best) - half, chunk):  # in order: reads lie at or past the writes
                e = min(c + chunk, len(best) - half)
                a, b = best[c:e], best[c + half:e + half].clone()
                take = b < a
                where[c:e] = torch.where(take, where[c + half:e + half], where[c:e])
                best[c:e] = torch.where(take, b, a)
        sel = torch.nonzero(level == k).squeeze(1)
        x, y = left[sel].long(), right[sel].long() + 1 - (1 << k)
        take = best[y] < best[x]
        at[sel] = torch.where(take, where[y], where[x]).long()
        out[sel] = torch.where(take, best[y], best[x]).to(out.dtype)
    return (-out if largest else out), at


def exact(case, seed):
    if case["kind"] not in ("batch", "grad"):
        values, queries = _plain_inputs(case, seed)
        out = _range_best(values, queries[:, 0], queries[:, 1], case["op"] == "max")
        return tuple(t.cpu() for t in out) if case["kind"] == "host" else out
    (starts, _, _, qcounts), values, queries = _batch_inputs(case, seed)
    first = torch.repeat_interleave(torch.from_numpy(starts).cuda(), torch.from_numpy(qcounts).cuda())
    best, at = _range_best(values, queries[:, 0] + first, queries[:, 1] + first,
                           case.get("op") == "max")
    if case["kind"] == "batch":
        return best, at - first
    grad_out = torch.randn(len(queries), device="cuda", generator=_gen(seed, 3))
    grad = torch.zeros(len(values), dtype=torch.float64, device="cuda")
    grad.index_add_(0, at, grad_out.double())
    return best, at - first, grad
