"""Benchmark of the batch RMQ hot path on one GB300 (replicas on N GPUs).

Workload (the reference's headline, README.md:6, csv-to-plot/perf-*-ALG5.csv):
plain RMQ over n = 1e8 float32 values uniform in [0,1) (seed 1321) with
q = 2^26 inclusive (l, r) queries, values and leftmost indices both returned.
The headline step is one rmq_query over the uniform-length queries (lr=-1);
the other length modes of the same configuration (lr=-2, lr=-3, fixed
len 2^10) are timed the same way and reported under "modes". The index takes
its blocks from the number of elements, so the block size it is asked for (the
default, or --bs) makes no difference; "bs_sweep_rmq_s" shows that over the
workload's range 2^10..2^16, and nothing is chosen from it.

Inputs are generated here with numpy (same seeds for both arms), so the
reference arm never loads this package.

value      -- RMQ/s of the device-resident step (inputs already in HBM),
              timed with CUDA events on the launching stream.
e2e        -- the same step through the C ABI with host buffers
              (rmq_query_host): the query kernel reads the pinned host queries
              and writes values + indices into pinned host memory over
              NVLink-C2C, all inside the timed region.
roofline   -- algorithmic HBM bytes per launch / kernel time against the
              measured copy bandwidth. The bytes are the query read and the
              result write (16 B per query) plus 32 B per sector of values
              that the launch reads, counted for this query set on the
              index's own tables (rmq_query_stats_ex). The small-table
              probes are L2-resident and reported apart, as is the
              un-pruned 80 B/query figure.
cpu_baseline -- the reference's CPU comparator HRMQ (restated in the
              oracle, hrmq_port.c) on this host's cores, on a bounded sample
              of the same queries.

Further sections: the tie-heavy configuration (n = 2^27 integers in
[0, 256), five fixed lengths), the CPU-runnable configuration (n = 1e6,
q = 2^20, lr=-3, L2 flushed before every timed step), the batched ragged
configuration and the differentiable one.

`--impl reference` times that CPU path alone (rank 0) and prints its own line.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

N_ELEMS = 10**8
N_QUERIES = 1 << 26
SEED = 1321
MODES = [("lr=-1", -1), ("lr=-2", -2), ("lr=-3", -3), ("len=2^10", 1024)]
BS_RANGE = [1 << k for k in range(10, 17)]       # the workload's block-size range
TIE_N = 1 << 27
TIE_LENGTHS = [1, 32, 1 << 10, 1 << 16, 1 << 22]
PUBLISHED_LR1 = 3.52e8  # RTXRMQ alg 5, RTX 6000 Ada (csv-to-plot/perf-RTX6000ADA-ALG5.csv:1586-1601)
L2_NOTE = ("no flush: the per-step working set (values, index tables, queries, outputs; "
           "1.5 GB at n=1e8) is larger than L2")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--n", type=int, default=N_ELEMS)
    ap.add_argument("--q", type=int, default=N_QUERIES)
    ap.add_argument("--modes", default="all", help="comma list of lr values or 'all'")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--bs", type=int, default=0, help="block size the indexes are asked for (default 2^15; skips the sweep)")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-buffer end-to-end step")
    ap.add_argument("--skip-plain", action="store_true", help="skip the plain modes (headline)")
    ap.add_argument("--skip-tie", action="store_true", help="skip the tie-heavy configuration")
    ap.add_argument("--skip-small", action="store_true", help="skip the n=1e6 configuration")
    ap.add_argument("--skip-batched", action="store_true")
    ap.add_argument("--batch-bs", type=int, default=0,
                    help="fixed block size for every bucket (skips the autotuner)")
    ap.add_argument("--skip-autograd", action="store_true")
    ap.add_argument("--batch-arrays", type=int, default=4096)
    ap.add_argument("--batch-q", type=int, default=1 << 26)
    ap.add_argument("--diff-rows", type=int, default=256)
    ap.add_argument("--diff-qpr", type=int, default=1 << 16)
    ap.add_argument("--probe-gib", type=int, default=4,
                    help="GiB of the layout-independent random-access probe's buffer")
    return ap.parse_args()


# ---------------------------------------------------------------- inputs (numpy)

def np_values_uniform(n: int, seed: int) -> np.ndarray:
    """float32 uniform in [0, 1) with 24-bit resolution."""
    return np.random.default_rng(seed).random(n, dtype=np.float32)


def np_values_int(n: int, vrange: int, seed: int) -> np.ndarray:
    """Integers uniform in [0, vrange) stored as float32 (tie-heavy)."""
    return np.random.default_rng(seed).integers(0, vrange, n).astype(np.float32)


def np_queries(q: int, n: int, lr: int, seed: int) -> np.ndarray:
    """int32 [q, 2] inclusive queries with the reference's length modes
    (src/rand.cuh:179-201): lr > 0 fixed length; -1 uniform in [1, n];
    -2 / -3 round(lognormal(0.6 / 0.3 * ln n, 0.3)) clamped to [1, n];
    l uniform in [0, n - len], r = l + len - 1."""
    rng = np.random.default_rng(seed)
    if lr > 0:
        ln = np.full(q, min(lr, n), dtype=np.int64)
    elif lr == -1:
        ln = rng.integers(1, n + 1, q)
    else:
        mu = {-2: 0.6, -3: 0.3}[lr] * math.log(n)
        ln = np.clip(np.rint(rng.lognormal(mu, 0.3, q)), 1, n).astype(np.int64)
    l = np.minimum((rng.random(q) * (n - ln + 1)).astype(np.int64), n - ln)
    return np.stack([l, l + ln - 1], axis=1).astype(np.int32)


def query_seed(rank: int, lr: int) -> int:
    """Seed of rank `rank`'s query set for length mode `lr` (replicas answer
    different query sets)."""
    return SEED + 1 + 1000 * rank + (0 if lr == -1 else 17 * abs(lr))


# ---------------------------------------------------------------- helpers

def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,utilization.gpu,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.dev), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                out, _ = self.proc.communicate(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
                out, _ = self.proc.communicate()
            self.lines = [ln for ln in out.splitlines() if ln.strip()]

    def summary(self):
        sm, mx, reasons, n_load = [], None, set(), 0
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                clk, cmax, util = float(f[1]), float(f[2]), float(f[4])
            except ValueError:
                continue
            mx = cmax
            if util >= 50:
                n_load += 1
                sm.append(clk)
                for nm, v in zip(names, f[5:9]):
                    if v.lower() == "active":
                        reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(self.lines), "samples_under_load": n_load}


def stats_bytes(st: dict, q: int, out_bytes: int = 8) -> dict:
    """Algorithmic bytes of one query launch from the kernel's own counts
    (query_stats(own=True)): the query read and result write, plus the 32-byte
    sectors of values read, one for a per-element entry (random HBM); the
    small-table words are L2-resident and reported apart."""
    hbm = q * (8 + out_bytes) + 32 * (st["entries"] + st["scan_sectors"])
    valid = max(1, q - st["invalid"])
    return {"alg_bytes": float(hbm), "alg_bytes_per_query": hbm / q,
            "unpruned_alg_bytes": float(q * (8 + out_bytes + 64)),
            "l2_table_words_per_query": st["table_words"] / valid,
            "entries_per_query": st["entries"] / valid,
            "entry_lookups_skipped": 1.0 - st["entries"] / (2.0 * valid),
            "settled": {k: st[k] / valid for k in ("first_probe", "second_probe", "full",
                                                   "micro_scan", "block_edge", "warp_scan")},
            "scan_sectors_per_query": st["scan_sectors"] / valid}


STEP_MIN = {}  # id(fn) -> fastest single step of the last time_steps(fn) call, ms


def time_steps(fn, steps, warmup, stream, barrier):
    """Mean ms per step over `steps` timed steps (CUDA events on `stream`,
    barrier + synchronize on both sides), the maximum over ranks under
    torchrun; the fastest single step goes to STEP_MIN[id(fn)]."""
    import torch
    for _ in range(warmup):
        fn()
    barrier()
    torch.cuda.synchronize()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
    ev[0].record(stream)
    for k in range(steps):
        fn()
        ev[k + 1].record(stream)
    torch.cuda.synchronize()
    barrier()
    from rtxrmq_gb300.replicas import max_over_ranks
    dev = torch.cuda.current_device()
    STEP_MIN[id(fn)] = max_over_ranks(min(ev[k].elapsed_time(ev[k + 1]) for k in range(steps)), dev)
    return max_over_ranks(ev[0].elapsed_time(ev[steps]) / steps, dev)


def time_steps_flushed(fn, steps, warmup, stream, barrier, flush_buf):
    """As time_steps, for working sets that fit in L2: before every step a
    write of `flush_buf` (larger than L2) evicts it, outside the timed
    events."""
    import torch
    for _ in range(warmup):
        flush_buf.zero_()
        fn()
    barrier()
    torch.cuda.synchronize()
    total, best = 0.0, float("inf")
    for _ in range(steps):
        flush_buf.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        fn()
        b.record(stream)
        torch.cuda.synchronize()
        t = a.elapsed_time(b)
        total += t
        best = min(best, t)
    barrier()
    from rtxrmq_gb300.replicas import max_over_ranks
    dev = torch.cuda.current_device()
    return max_over_ranks(total / steps, dev), max_over_ranks(best, dev)


# ---------------------------------------------------------------- CPU side

CPU_KIND = ("HRMQ restated (oracle/hrmq_port.c: balanced-parentheses RMQ of the reference's "
            "hrmq/RMQRMM64.cpp, ties leftmost), queries on all host threads")

TRAFFIC_PROFILE = ROOT / "profiles" / "query_kernel_plain_n1e8_q2e26_lr1.md"
# the sources query_kernel is compiled from; a traffic capture holds their digest
QUERY_SOURCES = tuple(ROOT / "rtxrmq_gb300" / "csrc" / f
                      for f in ("query.cu", "query_kernel.cuh", "query_impl.cuh", "lines.cuh",
                                "tables_impl.cuh", "common.cuh", "engine.h"))


def query_sources_digest():
    """SHA-256 over the query kernel's source files, in a fixed order."""
    import hashlib
    h = hashlib.sha256()
    for f in QUERY_SOURCES:
        h.update(f.name.encode() + b"\0" + f.read_bytes() + b"\0")
    return h.hexdigest()


def profiled_traffic(q):
    """DRAM bytes (read + write) per query_kernel launch of q queries, from
    the ncu capture summarised in TRAFFIC_PROFILE (its lines
    `traffic_bytes_per_query: X`, `traffic_bs: B` and
    `traffic_sources_sha256: H`, measured on this workload), and a
    description of it. The bytes are None when the profile is missing or was
    captured from other kernel sources than the ones built now."""
    fields = {}
    try:
        for line in TRAFFIC_PROFILE.read_text().splitlines():
            key, sep, val = line.strip().partition(":")
            if sep and key in ("traffic_bytes_per_query", "traffic_bs", "traffic_sources_sha256"):
                fields[key] = val.strip()
    except OSError:
        return None, {"source": None, "stale": "no traffic profile"}
    info = {"source": TRAFFIC_PROFILE.name, "bs": int(fields.get("traffic_bs", 0)) or None,
            "bytes_per_query": float(fields.get("traffic_bytes_per_query", "nan"))}
    if fields.get("traffic_sources_sha256") != query_sources_digest():
        info["stale"] = "query kernel sources changed since the ncu capture"
        return None, info
    if "traffic_bytes_per_query" not in fields:
        return None, info
    return info["bytes_per_query"] * q, info


def headline_config(n, q, lr):
    default = n == N_ELEMS and q == N_QUERIES and lr == -1
    label = "n=1e8 q=2^26 lr=-1" if default else f"n={n} q={q} lr={lr}"
    return default, label, {
        "workload": ("plain RMQ n=1e8 q=2^26 lr=-1 (uniform length), values+indices" if default
                     else f"plain RMQ {label}, values+indices"),
        "n": n, "q": q, "lr": lr, "seed": SEED, "l2": L2_NOTE}


def cpu_sample_rate(A, Q, target_s=12.0, nt=0):
    """The reference's CPU comparator (HRMQ, restated) on the host cores over
    a bounded random sample of the step's queries; build timed apart."""
    import oracle
    nt = nt or os.cpu_count() or 1
    t = time.perf_counter()
    h = oracle.HRMQ(A, strict=True, nt=nt)
    build_s = time.perf_counter() - t
    rng = np.random.default_rng(5)
    probe = Q[rng.integers(0, len(Q), 4096)]
    t = time.perf_counter()
    h.query(probe, nt)
    per = (time.perf_counter() - t) / len(probe)
    m = int(min(len(Q), max(4096, target_s / max(per, 1e-9))))
    sample = Q[rng.integers(0, len(Q), m)]
    t = time.perf_counter()
    h.query(sample, nt)
    dt = time.perf_counter() - t
    h.close()
    return m / dt, {"cores": nt, "sample": f"{m} random queries of the step's query set "
                    f"(n={len(A)}), {dt:.1f} s; construction {build_s:.2f} s", "construction_s": build_s}


def run_reference(args, rank):
    """--impl reference: the reference's CPU path for this workload (HRMQ,
    restated in the oracle; the reference's compiled code cannot run on the
    GPU host), rank 0 only, every step a bounded sample of the queries.
    Inputs come from the same numpy generators and seeds as the GPU arm;
    this package is not imported."""
    if rank != 0:
        return
    import oracle
    oracle.build(with_ref=False)
    nt = os.cpu_count() or 1
    n, q = args.n, args.q
    A = np_values_uniform(n, SEED)
    Q = np_queries(q, n, -1, query_seed(0, -1))
    t = time.perf_counter()
    h = oracle.HRMQ(A, strict=True, nt=nt)
    build_s = time.perf_counter() - t
    rng = np.random.default_rng(9)
    probe = Q[rng.integers(0, q, 4096)]
    t = time.perf_counter()
    h.query(probe, nt)
    per = (time.perf_counter() - t) / len(probe)
    m = int(max(4096, min(q, 1.5 / max(per, 1e-9))))  # ~1.5 s of work per step
    for _ in range(args.warmup):
        h.query(Q[rng.integers(0, q, m)], nt)
    times = []
    for _ in range(args.steps):
        s = Q[rng.integers(0, q, m)]
        t = time.perf_counter()
        h.query(s, nt)
        times.append(time.perf_counter() - t)
    v = m * args.steps / sum(times)
    default, label, config = headline_config(n, q, -1)
    line = {"metric": f"RMQ/s {label} (values+indices)", "value": v, "unit": "RMQ/s",
            "impl": "reference", "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * sum(times) / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config,
            "cpu_baseline": {"value": v, "unit": "RMQ/s", "cores": nt, "kind": "port",
                             "sample": f"{m} random queries per step from the {q}-query set; "
                                       f"{CPU_KIND}; construction {build_s:.2f} s"},
            "e2e": {"value": v, "unit": "RMQ/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------- GPU side

def graph_of(fn, stream):
    """Capture fn() once in a CUDA graph (after a warm run on a side stream)."""
    import torch
    s = torch.cuda.Stream()
    s.wait_stream(stream)
    with torch.cuda.stream(s):
        fn()
    stream.wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fn()
    torch.cuda.synchronize()
    return g


def sweep_block_sizes(R, dA, dQ, out_v, out_i, stream, barrier, q, world):
    """RMQ/s at every block size of the workload's range (3 timed steps each)."""
    sweep = {}
    for bs in BS_RANGE:
        with R.RMQIndex(dA, bs) as ix:
            fn = lambda: ix.query(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
            ms = time_steps(fn, 3, 1, stream, barrier)
        sweep[str(bs)] = q * world / (ms / 1e3)
    return sweep


def timed_build(make, reps: int = 5):
    """(index, median wall-clock ms of `reps` constructions including the
    allocation, as the reference's `construction` column counts it); all but
    the last index are freed."""
    import torch
    times, ix = [], None
    for r in range(reps):
        if ix is not None:
            ix.close()
        torch.cuda.synchronize()
        t = time.perf_counter()
        ix = make()
        torch.cuda.synchronize()
        times.append((time.perf_counter() - t) * 1e3)
    return ix, statistics.median(times)


def bench_plain_mode(R, dA, n, Q, out_v, out_i, args, stream, barrier, world, dev, rbuf):
    """One length mode of the headline configuration: construction, the timed
    steps, the counts of the same launch, and the two random-access probes."""
    import torch

    from rtxrmq_gb300.replicas import job_rate
    q = len(Q)
    dQ = torch.from_numpy(Q).to(dev)
    sweep = None if args.bs else sweep_block_sizes(R, dA, dQ, out_v, out_i, stream, barrier, q, world)
    bs = args.bs or R.DEFAULT_BS
    ix, construction_ms = timed_build(lambda: R.RMQIndex(dA, bs))
    fn = lambda: ix.query(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
    ms = time_steps(fn, args.steps, args.warmup, stream, barrier)
    st = ix.query_stats(dQ, own=True)
    acc = stats_bytes(st, q)
    res = {"value": job_rate(q, world, ms), "ms_per_step": ms, "ms_per_step_min": STEP_MIN[id(fn)],
           "bs": bs, "bs_sweep_rmq_s": sweep, "construction_ms": construction_ms, "query_stats": st, "accounting": acc,
           "achieved_gbs": acc["alg_bytes"] / (ms / 1e3) / 1e9,
           "unpruned_achieved_gbs": acc["unpruned_alg_bytes"] / (ms / 1e3) / 1e9,
           "info": ix.info()}
    # random-access probes with the query kernel's grid and query stream:
    # two random 8-B lookups per query into prefix / suffix minima per element
    # in blocks of bs (rmq_probe_gather, which makes them), and into a 4 GiB
    # buffer (rmq_probe_random, independent of the index layout)
    gfn = lambda: ix.probe_gather(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
    gms = time_steps(gfn, args.steps, args.warmup, stream, barrier)
    rfn = lambda: R.probe_random(rbuf, dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
    rms = time_steps(rfn, args.steps, args.warmup, stream, barrier)
    res["random_access"] = {
        "probe_buffer_gib": rbuf.numel() * 8 / 2**30,
        "probe_random_ms": rms, "probe_random_rmq_s": job_rate(q, world, rms),
        "probe_random_gbs": q * 80 / (rms / 1e3) / 1e9,
        "query_vs_probe_random": rms / ms,
        "probe_gather_ms": gms, "query_vs_probe_gather": gms / ms,
        "pattern": "per query: 8-B query read, two random 8-B loads, 8-B result write; "
                   "probe_random over a 4 GiB buffer (hashed positions), probe_gather at "
                   "suf[l] / pre[r]"}
    return res, ix, dQ


def bench_e2e(ix, Q, dQ, out_v, out_i, args, stream, barrier, world, dev):
    """rmq_query_host with pinned host buffers read and written in place,
    and the host link's ceiling for the same bytes."""
    import torch

    from rtxrmq_gb300.replicas import job_rate
    q = len(Q)
    hQ = torch.from_numpy(Q).pin_memory()
    hV = torch.empty(q, dtype=torch.float32).pin_memory()
    hI = torch.empty(q, dtype=torch.int32).pin_memory()

    def e2e():
        ix.query_host(hQ, hV, hI)

    e2e_ms = time_steps(e2e, args.steps, args.warmup, stream, barrier)
    torch.cuda.synchronize()
    dQc = torch.empty_like(dQ)
    dR = torch.empty(2 * q, dtype=torch.int32, device=dev)
    hR = torch.empty(2 * q, dtype=torch.int32).pin_memory()
    s_in, s_out = torch.cuda.Stream(), torch.cuda.Stream()

    def link():
        s_in.wait_stream(stream)
        s_out.wait_stream(stream)
        with torch.cuda.stream(s_in):
            dQc.copy_(hQ, non_blocking=True)
        with torch.cuda.stream(s_out):
            hR.copy_(dR, non_blocking=True)
        stream.wait_stream(s_in)
        stream.wait_stream(s_out)

    link_ms = time_steps(link, max(3, args.steps // 2), 2, stream, barrier)
    del dQc, dR, hR
    ix.query(dQ, out_val=out_v, out_idx=out_i)
    torch.cuda.synchronize()
    ok = (np.array_equal(hI.numpy(), out_i.cpu().numpy()) and
          np.array_equal(hV.numpy().view(np.uint32), out_v.cpu().numpy().view(np.uint32)))
    return {"value": job_rate(q, world, e2e_ms), "unit": "RMQ/s",
            "h2d_bytes_per_step": int(Q.nbytes),
            "d2h_bytes_per_step": int(hV.numel() * 4 + hI.numel() * 4),
            "ms_per_step": e2e_ms,
            "path": "rmq_query_host, pinned host buffers read and written in place",
            "matches_device_path": bool(ok),
            "link_ceiling": {"ms_per_step": link_ms, "rmq_s": job_rate(q, world, link_ms),
                             "gbs_per_direction": Q.nbytes / (link_ms / 1e3) / 1e9,
                             "frac": link_ms / e2e_ms,
                             "how": "the step's query bytes in and result bytes out copied "
                                    "concurrently (pinned, two streams)"}}


def bench_energy(fn, ms, q, local):
    import torch

    from rtxrmq_gb300.power import PowerSampler
    reps_e = max(1, int(1500.0 / max(ms, 1e-3)))
    torch.cuda.synchronize()
    with PowerSampler(local, sample_ms=50) as ps:
        for _ in range(reps_e):
            fn()
        torch.cuda.synchronize()
    if ps.available and ps.energy_joules:
        return {"rmq_per_joule": q * reps_e / ps.energy_joules, "avg_watts": ps.avg_watts,
                "seconds": ps.seconds, "reps": reps_e, "source": "NVML board power, 50 ms samples",
                "reference": "RTXRMQ on RTX 6000 Ada: 1.20e6 RMQ/J (2^26 x 512 queries / "
                             "28625.93 J, scripts/plot_rmq_per_joule.py:69)"}
    return {"unavailable": f"NVML status {ps.status}"}


def bench_tie_heavy(R, args, stream, barrier, world, rank, dev):
    """Tie-heavy configuration: n = 2^27 floats holding integers uniform in
    [0, 256), q = 2^26 queries of each fixed length. Bit-exactness at this size
    is asserted by tests/test_gpu_fullscale.py."""
    import torch

    from rtxrmq_gb300.replicas import job_rate
    n, q = TIE_N, args.q
    dA = torch.from_numpy(np_values_int(n, 256, SEED + 3)).to(dev)
    out_v = torch.empty(q, dtype=torch.float32, device=dev)
    out_i = torch.empty(q, dtype=torch.int32, device=dev)
    res = {"workload": "n=2^27 float32 integers U{0..255}, q=2^26 per fixed length, "
                       "values+indices", "l2": L2_NOTE}
    for length in TIE_LENGTHS:
        Q = np_queries(q, n, length, query_seed(rank, length) + 5)
        dQ = torch.from_numpy(Q).to(dev)
        with R.RMQIndex(dA, args.bs) as ix:
            fn = lambda: ix.query(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
            ms = time_steps(fn, args.steps, args.warmup, stream, barrier)
            st = ix.query_stats(dQ, own=True)
        acc = stats_bytes(st, q)
        res[f"len={length}"] = {"rmq_s": job_rate(q, world, ms), "ms_per_step": ms,
                                "settled": acc["settled"],
                                "alg_bytes_per_query": acc["alg_bytes_per_query"],
                                "achieved_gbs": acc["alg_bytes"] / (ms / 1e3) / 1e9}
        del dQ
    del dA, out_v, out_i
    torch.cuda.empty_cache()
    return res


def bench_small(R, args, stream, barrier, world, rank, dev):
    """CPU-runnable configuration: n = 1e6 U[0,1), q = 2^20, lr=-3. Its
    working set fits in L2, so L2 is flushed (a 512 MB write) before every
    timed step."""
    import torch

    from rtxrmq_gb300.replicas import job_rate
    n, q = 10**6, 1 << 20
    dA = torch.from_numpy(np_values_uniform(n, SEED)).to(dev)
    Q = np_queries(q, n, -3, query_seed(rank, -3))
    dQ = torch.from_numpy(Q).to(dev)
    out_v = torch.empty(q, dtype=torch.float32, device=dev)
    out_i = torch.empty(q, dtype=torch.int32, device=dev)
    flush = torch.empty(1 << 27, dtype=torch.float32, device=dev)
    with R.RMQIndex(dA, args.bs) as ix:
        fn = lambda: ix.query(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
        ms, best = time_steps_flushed(fn, args.steps, args.warmup, stream, barrier, flush)
        st = ix.query_stats(dQ, own=True)
    acc = stats_bytes(st, q)
    del dA, dQ, out_v, out_i, flush
    torch.cuda.empty_cache()
    return {"workload": "n=1e6 U[0,1), q=2^20, lr=-3 (lognormal 0.3 ln n), values+indices",
            "l2": "flushed (512 MB write) before every timed step: the working set fits in L2",
            "rmq_s": job_rate(q, world, ms), "ms_per_step": ms, "ms_per_step_min": best,
            "settled": acc["settled"], "alg_bytes_per_query": acc["alg_bytes_per_query"]}


def bench_batched(args, dev, stream, barrier):
    """Batched ragged config: 4096 arrays, lengths round(2^U), U ~ U[8,22],
    2^26 queries proportional to length, lognormal(0.5 ln len, 0.4) lengths.
    Step = build every array + answer every query."""
    import torch

    from rtxrmq_gb300 import workloads as W
    from rtxrmq_gb300.batch import RMQBatch, autotune
    t = time.perf_counter()
    w = W.ragged(narrays=args.batch_arrays, total_q=args.batch_q, seed=SEED)
    gen_s = time.perf_counter() - t
    dV = torch.from_numpy(w.values).to(dev)
    dQ = torch.from_numpy(w.queries).to(dev)
    ov = torch.empty(w.total_q, dtype=torch.float32, device=dev)
    oi = torch.empty(w.total_q, dtype=torch.int32, device=dev)
    t = time.perf_counter()
    if args.batch_bs:
        cfg = [(args.batch_bs, 0, 0)] * 32
    else:
        # per bucket: block size, queries per query item, entries per level item
        cfg = autotune(w.starts, w.lengths, w.qstarts, w.qcounts, dV, dQ, reps=2,
                       queries_host=w.queries, cache=None, tiles=True)
    tune_s = time.perf_counter() - t
    res = {"workload": "4096 arrays, len round(2^U) U~U[8,22], 2^26 queries proportional to "
                       "length, query len lognormal(0.5 ln len, 0.4), values U[0,1)",
           "arrays": int(len(w.lengths)), "elements": int(w.lengths.sum()), "queries": w.total_q,
           "generate_s": gen_s, "autotune_s": tune_s,
           "bucket_tiles": {str(b): {"bs": v[0], "query_chunk": v[1], "level_chunk": v[2]}
                            for b, v in enumerate(cfg) if v[0]}}
    with RMQBatch(w.starts, w.lengths, w.qstarts, w.qcounts, cfg) as b:
        info = b.info()
        res["workspace_gb"] = info["workspace_bytes"] / 1e9
        fn = lambda: b.run(dV, dQ, ov, oi)  # noqa: E731
        ms = time_steps(fn, args.steps, args.warmup, stream, barrier)
        g = graph_of(fn, stream)
        gms = time_steps(g.replay, args.steps, args.warmup, stream, barrier)
        # the two halves: build every array, then answer from the built index
        bms = time_steps(lambda: b.build(dV), args.steps, args.warmup, stream, barrier)
        qms = time_steps(lambda: b.query(dV, dQ, ov, oi), args.steps, args.warmup, stream, barrier)
        v1, i1 = ov.clone(), oi.clone()
        pms = time_steps(lambda: b.run_per_array(dV, dQ, ov, oi), max(2, args.steps // 3), 1,
                         stream, barrier)
        match = bool(torch.equal(i1, oi) and torch.equal(v1.view(torch.int32), ov.view(torch.int32)))
        del g
    with RMQBatch(w.starts, w.lengths, w.qstarts, w.qcounts, None) as b:
        dms = time_steps(lambda: b.run(dV, dQ, ov, oi), args.steps, 1, stream, barrier)
    from rtxrmq_gb300.replicas import job_rate, world
    q, nr = w.total_q, world()[1]
    res.update({"batched_graph_rmq_s": job_rate(q, nr, gms), "batched_graph_ms": gms,
                "batched_rmq_s": job_rate(q, nr, ms), "batched_ms": ms,
                "per_array_rmq_s": job_rate(q, nr, pms), "per_array_ms": pms,
                "speedup_vs_per_array": pms / gms,
                "default_bs_rmq_s": job_rate(q, nr, dms),
                "per_array_matches_batched": match,
                "build_only_ms": bms, "query_only_ms": qms,
                "query_only_rmq_s": job_rate(q, nr, qms),
                # bytes that one step cannot do without (each value read once, a query's
                # pair read and 8 B written) against the graph-launched step
                "alg_bytes_per_step": int(w.lengths.sum()) * 4 + q * 16,
                "alg_gbs": (int(w.lengths.sum()) * 4 + q * 16) / (gms / 1e3) / 1e9,
                "launches_per_step": {"batched": 1, "per_array": "one build + level + query "
                                      "launch sequence per array"}})
    del dV, dQ, ov, oi
    torch.cuda.empty_cache()
    return res


def bench_autograd(args, dev, stream, barrier):
    """Differentiable config: 256 rows N(0,1), lengths U[2^14, 2^20], 2^16
    ranges per row with lengths lognormal(0.4 ln len, 0.5); grad_out N(0,1).
    Forward and forward+backward each captured in a CUDA graph."""
    import torch

    from rtxrmq_gb300 import workloads as W
    from rtxrmq_gb300.autograd import RaggedRangeMin
    from rtxrmq_gb300.batch import autotune
    d = W.differentiable_rows(nrows=args.diff_rows, q_per_row=args.diff_qpr, seed=SEED)
    x = torch.from_numpy(d.values).to(dev)
    dQ = torch.from_numpy(d.queries).to(dev)
    gout_h = np.random.default_rng(SEED).standard_normal(d.total_q).astype(np.float32)
    go = torch.from_numpy(gout_h).to(dev)
    cfg = autotune(d.starts, d.lengths, d.qstarts, d.qcounts, x, dQ, reps=2,
                   queries_host=d.queries, cache=None, tiles=True)
    m = RaggedRangeMin(d.lengths, d.qcounts, cfg)
    xg = x.clone().requires_grad_(True)

    def fwd():
        with torch.no_grad():
            return m(x, dQ)

    def fwd_bwd():
        xg.grad = None
        y, _ = m(xg, dQ)
        y.backward(go)

    fwd_bwd()  # allocate grad once outside capture
    gf = graph_of(fwd, stream)
    xg.grad = None
    gb = graph_of(fwd_bwd, stream)
    from rtxrmq_gb300.replicas import job_rate, world
    fms = time_steps(gf.replay, args.steps, args.warmup, stream, barrier)
    bms = time_steps(gb.replay, args.steps, args.warmup, stream, barrier)
    # full-size check of the gradient against an FP64 scatter of the same argmins
    y, idx = fwd()
    torch.cuda.synchronize()
    gidx = idx.cpu().numpy().astype(np.int64) + np.repeat(d.starts, d.qcounts)
    g64 = np.zeros(d.span, np.float64)
    np.add.at(g64, gidx, gout_h.astype(np.float64))
    scale = np.zeros(d.span, np.float64)  # sum of |contributions| per element
    np.add.at(scale, gidx, np.abs(gout_h.astype(np.float64)))
    gb.replay()
    torch.cuda.synchronize()
    g = xg.grad.cpu().numpy().astype(np.float64)
    nz = scale > 0
    rel = float((np.abs(g[nz] - g64[nz]) / scale[nz]).max()) if nz.any() else 0.0
    zero_ok = bool(np.all(g[~nz] == 0))
    q = d.total_q
    res = {"workload": "256 rows N(0,1), len U[2^14,2^20], 2^16 ranges/row, len lognormal("
                       "0.4 ln len, 0.5), grad_out N(0,1)",
           "elements": d.span, "queries": q,
           "bucket_tiles": {str(b): {"bs": v[0], "query_chunk": v[1], "level_chunk": v[2]}
                            for b, v in enumerate(cfg) if v[0]},
           "fwd_ms": fms, "fwd_bwd_ms": bms, "fwd_bwd_over_fwd": bms / fms,
           "fwd_rmq_s": job_rate(q, world()[1], fms), "fwd_bwd_rmq_s": job_rate(q, world()[1], bms),
           "graph_captured": True, "grad_max_rel_err_vs_fp64": rel, "grad_zero_elsewhere": zero_ok}
    del gf, gb, x, xg, dQ, go
    torch.cuda.empty_cache()
    return res


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return

    import torch
    import torch.distributed as dist

    import rtxrmq_gb300 as R
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))

    def barrier():
        if world > 1:
            dist.barrier()

    dev = torch.device("cuda", local)
    stream = torch.cuda.current_stream()
    n, q = args.n, args.q
    hbm_peak, peak_kind = peaks()

    modes = MODES if args.modes == "all" else [(f"lr={m}", int(m)) for m in args.modes.split(",")]
    if args.skip_plain:
        modes = []

    results = {}
    headline = None
    tie = small = batched = autograd = None
    A = None
    sampler = ClockSampler(local)
    with sampler:
        if modes:
            A = np_values_uniform(n, SEED)
            dA = torch.from_numpy(A).to(dev)
            out_v = torch.empty(q, dtype=torch.float32, device=dev)
            out_i = torch.empty(q, dtype=torch.int32, device=dev)
            # words for the layout-independent random-access probe (4 GiB)
            rbuf = torch.arange(args.probe_gib << 27, dtype=torch.int64, device=dev)
            for name, lr in modes:
                Q = np_queries(q, n, lr, query_seed(rank, lr))
                res, ix, dQ = bench_plain_mode(R, dA, n, Q, out_v, out_i, args, stream, barrier,
                                               world, dev, rbuf)
                if lr == -1:
                    headline = (name, lr, Q)
                    if not args.no_e2e:
                        res["e2e"] = bench_e2e(ix, Q, dQ, out_v, out_i, args, stream, barrier,
                                               world, dev)
                    fn = lambda: ix.query(dQ, out_val=out_v, out_idx=out_i)  # noqa: E731
                    res["energy"] = bench_energy(fn, res["ms_per_step"], q, local)
                ix.close()
                results[name] = res
                del dQ
            del rbuf
            del dA, out_v, out_i
            torch.cuda.empty_cache()
        if not args.skip_tie and args.modes == "all":
            tie = bench_tie_heavy(R, args, stream, barrier, world, rank, dev)
        if not args.skip_small and args.modes == "all":
            small = bench_small(R, args, stream, barrier, world, rank, dev)
        batched = None if args.skip_batched else bench_batched(args, dev, stream, barrier)
        autograd = None if args.skip_autograd else bench_autograd(args, dev, stream, barrier)
    clocks = sampler.summary()

    if rank != 0:
        if world > 1:
            dist.destroy_process_group()
        return
    if not results:  # a run of the other sections only
        print(json.dumps({"metric": "sections other than the headline only", "value": None,
                          "clocks": clocks, "tie_heavy": tie, "small_config": small,
                          "batched": batched, "autograd": autograd}), flush=True)
        if world > 1:
            dist.destroy_process_group()
        return
    name, lr, Q = headline if headline else (modes[0][0], modes[0][1], None)
    h = results[name]
    achieved = h["achieved_gbs"]
    default, label, config = headline_config(n, q, lr)
    traffic, traffic_info = profiled_traffic(q) if default else (None, None)
    line = {
        "metric": f"RMQ/s {label} (values+indices)",
        "value": h["value"], "unit": "RMQ/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": h["ms_per_step"],
        "ms_per_step_min": h["ms_per_step_min"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": h["value"] / PUBLISHED_LR1,
        "vs_baseline_ref": "RTXRMQ (alg 5) on RTX 6000 Ada, 3.52e8 RMQ/s, n=1e8 q=2^26 lr=-1",
        "dtype": "f32", "data": "synthetic (numpy generators, seed 1321)",
        "config": config,
        "bs": h["bs"],
        "parallelism": f"replicas x{world}" if world > 1 else "single GPU",
        "e2e": h.get("e2e"),
        "gpu_launches": args.steps,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm_peak, "unit": "GB/s",
                     "frac": achieved / hbm_peak,
                     # DRAM bytes captured by ncu on the headline workload only,
                     # from the same kernel sources
                     "traffic": traffic,
                     "traffic_source": traffic_info,
                     "peak_kind": f"{peak_kind} copy bandwidth",
                     "kernel": "query_kernel",
                     "alg_bytes_per_launch": h["accounting"]["alg_bytes"],
                     "alg_bytes_basis": "16 B per query (query read, value + index write) + 32 B "
                                        "per sector of values read, counted on this query set "
                                        "and the launch's own tables (rmq_query_stats_ex)",
                     "l2_table_words_per_query": h["accounting"]["l2_table_words_per_query"],
                     "unpruned_alg_bytes_per_launch": h["accounting"]["unpruned_alg_bytes"],
                     "unpruned_achieved": h["unpruned_achieved_gbs"],
                     "unpruned_frac": h["unpruned_achieved_gbs"] / hbm_peak},
        "random_access_roofline": h.get("random_access"),
        "clocks": clocks,
        "modes": {k: {kk: vv for kk, vv in v.items() if kk not in ("info",)} for k, v in results.items()},
        "energy": h.get("energy"),
        "tie_heavy": tie,
        "small_config": small,
        "batched": batched,
        "autograd": autograd,
    }
    if not args.no_cpu and world == 1 and A is not None and Q is not None:
        v, meta = cpu_sample_rate(A, Q)
        line["cpu_baseline"] = {"value": v, "unit": "RMQ/s", "cores": meta["cores"], "kind": "port",
                                "sample": meta["sample"] + "; " + CPU_KIND}
    print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
