#!/usr/bin/env python
"""AMEn solves/s and p50/p99 latency at relative residual 1e-8 on B200.

Workload (``--preset config5``, the default): the serving mix of requests,
each drawn from one seeded generator (``problems.serving_request``): 10 %
large diffusion solves (d = 24, n = 64, random rank-8 right-hand side), the
rest in equal parts parametric diffusion (d ~ U{4..12}, n ~ U{16, 32, 64},
theta ~ U(-1, 1)) and 2-D QTT Poisson problems with 6-20 cores.  Every
request is solved to relative residual 1e-8 with at most 30 sweeps; a
request that stops above the tolerance counts as not solved.  A step is one
batch of ``--requests`` consecutive requests of the stream (every step a
different batch).  ``--preset small`` is a reduced mix (diffusion d in
{4, 5}, n in {16, 32}).

``value``: the warm-up and timed steps' requests are uploaded to the device
first; the timed steps' requests are then queued at once, longest first, to
the continuous-batching server on the persistent whole-solve kernel
(``persistent_serving``), and value = solved requests / device time of the
whole run.  ``e2e``: the same server fed from host memory through its public
API (inputs copied per launch, solutions read back) with a seeded Poisson
stream arriving at twice the measured capacity; one more pass at 0.8x of it
(``--serve-loads``) reports the latency at a sustainable load.

Prints one JSON line (rank 0).  ``--impl reference`` times the CPU oracle
(the NumPy/SciPy restatement of the reference path, kept within a few
percent of the reference's own speed) on the host cores instead, on bounded
samples of the same stream.

Launch: ``python bench.py`` (1 GPU) or, for N GPUs,
``python -m torch.distributed.run --nproc-per-node N ... bench.py --gpus N``:
every rank serves its own copy of the stream (replicas; independent solves
need no collective), ``value`` = all ranks' solves / max time.
"""

from __future__ import annotations

import argparse
import json
import multiprocessing as mp
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "AMEn solves/s at relative residual 1e-8"
UNIT = "solves/s"
TOL = 1e-8
MAX_SWEEPS = 30
KINDS = ("qtt", "diffusion", "large")


def parse(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--preset", default="config5", choices=["config5", "small"])
    ap.add_argument("--requests", type=int, default=148,
                    help="requests per step (148 = one per SM of a B200)")
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--serve-requests", type=int, default=1000,
                    help="requests in each served pass (a slice of the stream after the "
                         "timed steps' requests)")
    ap.add_argument("--serve-loads", default="0.8",
                    help="arrival rates of the latency passes, as fractions of the measured "
                         "capacity (the throughput pass arrives at twice it)")
    ap.add_argument("--serve-mem-gb", type=float, default=96.0,
                    help="device memory the server may hold in work areas of requests in flight")
    ap.add_argument("--streams", type=int, default=32, help="server launch streams")
    ap.add_argument("--max-batch", type=int, default=8, help="requests per server launch")
    ap.add_argument("--light-streams", type=int, default=8,
                    help="high-priority server streams for light requests (0: one lane)")
    ap.add_argument("--plain-sample", type=int, default=64,
                    help="requests timed through the plain one-at-a-time drop-in (0: skip)")
    ap.add_argument("--cpu-sample", type=int, default=0,
                    help="requests in the CPU baseline sample (0: two per host core)")
    ap.add_argument("--plain-limit", type=float, default=2.0,
                    help="per-solve time limit (s) of the plain drop-in sample (shorter than "
                         "--time-limit, which can only favour the plain baseline)")
    ap.add_argument("--time-limit", type=float, default=30.0,
                    help="per-solve time limit (s), the same for every arm: device time of a "
                         "solve on the GPU, host time on the CPU; a solve stopped by it counts "
                         "as not solved")
    ap.add_argument("--cluster", action="store_true",
                    help="run mode-64 requests on clusters of four thread blocks")
    ap.add_argument("--profile-case", action="store_true",
                    help="only run the small profiling case (one persistent launch of 8 "
                         "requests, twice) and print its per-request device times")
    ap.add_argument("--profile-mixed", action="store_true",
                    help="with --profile-case: mixed precision (3xTF32 tensor-core products "
                         "inside float64 refinement) and iterative local solves above 50 "
                         "unknowns")
    return ap.parse_args(argv)


# ---------------------------------------------------------------------------
# workload
# ---------------------------------------------------------------------------


def make_requests(count: int, seed: int, preset: str = "config5"):
    """The first ``count`` requests of the seeded stream."""
    from ttnumpy_b200 import problems as P

    if preset == "config5":
        return P.serving_requests(count, seed)
    return P.serving_requests(count, seed, large_share=0.0, dims=(4, 5), modes=(16, 32))


def solve_kwargs(p):
    return dict(residual_tol=TOL, symmetric=True, max_sweeps=MAX_SWEEPS, seed=0,
                stagnation_factor=None)


def x0_cores(p):
    """Initial guess: rank-3 all-ones for QTT Poisson (the reference
    benchmark's choice), the default (all-ones with b's ranks) otherwise."""
    if p.meta.get("kind") == "qtt":
        return 3
    return None


def x0_host(p):
    r = x0_cores(p)
    if r is None:
        return None
    modes = [c.shape[1] for c in p.b]
    ranks = [1] + [r] * (len(modes) - 1) + [1]
    return [np.ones((ranks[i], modes[i], 1, ranks[i + 1])) for i in range(len(modes))]


def host_request(p):
    """(A, b, x0, kwargs) as the server's public ``serve`` takes it."""
    return (p.A, p.b, x0_host(p), solve_kwargs(p))


def aggregate_rate(solved: int, ms: float, world: int, device: str = "cuda"):
    """Whole-job rate over the ranks: all ranks' solves over the slowest
    rank's time.  Returns (solves per second, max milliseconds); a single
    process needs no process group."""
    if world > 1:
        import torch
        import torch.distributed as dist

        t = torch.tensor([float(solved), float(ms)], dtype=torch.float64, device=device)
        mx = t.clone()
        dist.all_reduce(t, op=dist.ReduceOp.SUM)
        dist.all_reduce(mx, op=dist.ReduceOp.MAX)
        solved, ms = float(t[0].item()), float(mx[1].item())
    return solved / (ms * 1e-3), ms


def class_stats(kinds, solved, seconds=None):
    """Per request class: requests, solved, and (with per-request
    ``seconds``) their mean."""
    out = {}
    for k in KINDS:
        idx = [i for i, kk in enumerate(kinds) if kk == k]
        if not idx:
            continue
        row = {"requests": len(idx), "solved": int(sum(bool(solved[i]) for i in idx))}
        if seconds is not None:
            row["mean_s"] = float(np.mean([seconds[i] for i in idx]))
        out[k] = row
    return out


# ---------------------------------------------------------------------------
# CPU oracle (reference arm and cpu_baseline)
# ---------------------------------------------------------------------------


def _cpu_solve(args):
    p, limit = args
    os.environ["OPENBLAS_NUM_THREADS"] = "1"
    from threadpoolctl import threadpool_limits

    from oracle import tt_oracle as O

    with threadpool_limits(1):
        A, b = O.Train(p.A), O.Train(p.b)
        x0 = None
        r = x0_cores(p)
        if r is not None:
            x0 = O.orthonormalize(O.ones(b.row_modes, ranks=r), "right")
        t0 = time.perf_counter()
        x, info = O.amen(A, b, x0=x0, time_limit=limit, **solve_kwargs(p))
        dt = time.perf_counter() - t0
    return dt, str(info.stop_reason) == "converged", p.meta.get("kind")


def cpu_run(reqs, workers: int, limit: float):
    """Solve ``reqs`` on a spawn pool of single-threaded workers, each solve
    capped at ``limit`` seconds; returns (wall seconds, per-request
    (seconds, converged, class))."""
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    with ctx.Pool(workers) as pool:
        res = pool.map(_cpu_solve, [(p, limit) for p in reqs], chunksize=1)
    return time.perf_counter() - t0, res


def cpu_cores() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def cpu_baseline(reqs, cores, limit):
    """CPU rate on a sample of the stream: solved requests over the CPU
    time they took divided by the cores (the pool's sustained rate, not
    bound by its slowest worker); capped solves count as unsolved at the
    cap's time, which can only favour the CPU."""
    wall, res = cpu_run(reqs, cores, limit)
    cpu_s = sum(r[0] for r in res)
    solved = sum(1 for r in res if r[1])
    kinds = [r[2] for r in res]
    return {"value": solved / (cpu_s / cores), "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"the first {len(reqs)} requests of the stream, {cores} single-threaded "
                      f"oracle workers, each solve capped at {limit:g} s; value = solved / "
                      f"(sum of solve seconds / cores)",
            "wall_s": wall, "cpu_s": cpu_s,
            "classes": class_stats(kinds, [r[1] for r in res], [r[0] for r in res])}


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.lines:
            parts = [v.strip() for v in line.split(",")]
            if len(parts) < 7:
                continue
            try:
                sm.append(float(parts[0]))
                mx = max(mx, float(parts[1]))
            except ValueError:
                continue
            for name, v in zip(names, parts[3:7]):
                if v.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------


def fp64_peak_tflops(K, torch):
    """Measured FP64 FMA throughput of this GPU (own probe kernel)."""
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    lib = K.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks, iters = sms * 8, 4096
    lib.ttb_fma_peak(out.data_ptr(), blocks, iters, K.stream())
    torch.cuda.synchronize()
    best = 0.0
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        lib.ttb_fma_peak(out.data_ptr(), blocks, iters, K.stream())
        b.record()
        torch.cuda.synchronize()
        flops = 2.0 * 8 * iters * 256 * blocks
        best = max(best, flops / (a.elapsed_time(b) * 1e-3) / 1e12)
    return best


def _solved(job) -> bool:
    r = job.result
    return r is not None and r.status == 0 and bool(r.info.converged)


def make_server(args, resident: bool, download: bool):
    from ttnumpy_b200.persistent_serving import PersistentServer

    from ttnumpy_b200.persistent import cluster_size

    return PersistentServer(streams=args.streams, max_batch=args.max_batch,
                            mem_budget=int(args.serve_mem_gb * 2**30), resident=resident,
                            download=download, time_limit=args.time_limit,
                            cluster_for=cluster_size if args.cluster else None,
                            light_streams=args.light_streams)


def resident_run(args, preps, torch):
    """Closed-loop run of the server over device-resident requests, all
    queued at once, longest first.  Returns (device ms, jobs, launches)."""
    from ttnumpy_b200 import kernels as K
    from ttnumpy_b200.persistent import _cost

    order = sorted(range(len(preps)), key=lambda i: -_cost(preps[i]))
    server = make_server(args, resident=True, download=False)
    torch.cuda.synchronize()
    l0 = K.launch_count()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    jobs = server.serve([preps[i] for i in order], [0.0] * len(order))
    e.record()
    torch.cuda.synchronize()
    back = [None] * len(preps)
    for j, i in enumerate(order):
        back[i] = jobs[j]
    return s.elapsed_time(e), back, K.launch_count() - l0, server


def served_pass(args, reqs, rate, torch, seed):
    """One pass of the server through its public API: host requests
    arriving as a seeded Poisson stream at ``rate`` per second, inputs
    copied per launch, solutions read back.  Timed with CUDA events around
    the whole stream."""
    host = [host_request(p) for p in reqs]
    rng = np.random.default_rng(seed)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, size=len(host)))
    arrivals -= arrivals[0]
    server = make_server(args, resident=False, download=True)
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    jobs = server.serve(host, list(arrivals))
    torch.cuda.synchronize()
    e.record()
    e.synchronize()
    seconds = s.elapsed_time(e) * 1e-3
    solved = sum(1 for j in jobs if _solved(j))
    lats = [1e3 * j.latency for j in jobs if j.latency is not None]
    out = {"rate": rate, "requests": len(jobs), "solved": solved, "seconds": seconds,
           "throughput": solved / seconds,
           "latency_ms": {"p50": percentile(lats, 50), "p99": percentile(lats, 99)},
           "h2d": server.h2d_bytes, "d2h": server.d2h_bytes, "launches": server.launches,
           "peak_gb": server.peak_bytes / 2**30}
    jobs = server = None
    torch.cuda.empty_cache()
    return out


def plain_run(reqs, limit, torch):
    """The plain one-solve-at-a-time FP64 GPU AMEn (the drop-in ``amen``,
    every contraction and factorisation a library call) on the first
    requests of the stream, each solve capped at ``limit`` seconds."""
    import ttnumpy_b200 as tt
    from ttnumpy_b200.solvers.amen import solve_time_limit

    def one(p):
        A, b = tt.TensorTrain(p.A), tt.TensorTrain(p.b)
        r = x0_cores(p)
        x0 = tt.ones(b.physical_dims(), ranks=r).orthonormalize("right") if r else None
        with solve_time_limit(limit):
            x, info = tt.amen(A, b, x0=x0, return_info=True, **solve_kwargs(p))
        return bool(info.converged)

    one(reqs[0])  # warm-up
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    ok = [one(p) for p in reqs]
    e.record()
    torch.cuda.synchronize()
    kinds = [p.meta["kind"] for p in reqs]
    return {"value": sum(ok) / (s.elapsed_time(e) * 1e-3), "unit": UNIT,
            "sample": f"the first {len(reqs)} requests of the stream, solved one after another "
                      f"by the drop-in amen, each capped at {limit:g} s",
            "classes": class_stats(kinds, ok)}


def config1_problem():
    """Config 1: the 8-D Laplacian with n = 32 (h = 1/33) and a rank-4
    uniform right-hand side (tt.rand seed 0)."""
    from ttnumpy_b200 import problems as P

    return P.Problem("config1", P.laplacian_nd(8, 32), P.random_tt([32] * 8, 4, seed=0),
                     meta={"kind": "config1"})


def config1_run(torch):
    """Single-solve latency of config 1 (max_sweeps 20): one request alone
    in a persistent launch (one SM) and the drop-in (the whole GPU)."""
    import ttnumpy_b200 as tt
    from ttnumpy_b200.persistent import amen_persistent

    p = config1_problem()
    kw = dict(residual_tol=TOL, symmetric=True, max_sweeps=20, seed=0, stagnation_factor=None)
    out = {}
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    r = amen_persistent([(p.A, p.b, None, kw)], rmax=64, cluster=1)[0]
    torch.cuda.synchronize()
    out["persistent_s"] = time.perf_counter() - t0
    out["persistent_device_s"] = r.device_ms * 1e-3
    out["persistent"] = {"status": r.status, "sweeps": r.info.num_sweeps_run,
                         "residual": r.info.residuals[-1] if r.info.residuals else None}
    for cl in (4, 8):  # the same solve on a cluster of blocks (same bits, shorter wall time)
        t0 = time.perf_counter()
        rc = amen_persistent([(p.A, p.b, None, kw)], rmax=64, cluster=cl)[0]
        torch.cuda.synchronize()
        out[f"cluster{cl}_s"] = time.perf_counter() - t0
        out[f"cluster{cl}_same_bits"] = bool(
            rc.status == 0 and rc.info.residuals == r.info.residuals
            and all(np.array_equal(u, v) for u, v in zip(rc.x.to_numpy(), r.x.to_numpy())))
    t0 = time.perf_counter()
    x, info = tt.amen(tt.TensorTrain(p.A), tt.TensorTrain(p.b), return_info=True, **kw)
    torch.cuda.synchronize()
    out["dropin_s"] = time.perf_counter() - t0
    out["dropin"] = {"sweeps": info.num_sweeps_run, "residual": info.residuals[-1]}
    return out


def rounding_run(torch, pairs=1024, reps=5):
    """Config 2: ``(p_i + q_i).truncate(1e-6)`` for 1024 pairs of uniform
    rank-32 trains with d = 16, n = 4 (seeds 2i, 2i + 1), all pairs in one
    launch of the batched rounding kernel.  Pairs per second over ``reps``
    launches (inputs resident), and the relative Frobenius error of a sample
    of results against the float64 oracle's rounding of the same sums."""
    from oracle import tt_oracle as O
    from ttnumpy_b200 import problems as P
    from ttnumpy_b200.rounding import PackedTrains, RoundPlan

    ps = [P.random_tt([4] * 16, 32, seed=2 * i) for i in range(pairs)]
    qs = [P.random_tt([4] * 16, 32, seed=2 * i + 1) for i in range(pairs)]
    pk, qk = PackedTrains.from_numpy(ps), PackedTrains.from_numpy(qs)
    plan = RoundPlan(pairs, 16, pk.modes, pk.bonds, qk.bonds, pk.offsets, qk.offsets)
    res = plan.run(pk.data, qk.data, 1e-6, None)
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(reps):
        res = plan.run(pk.data, qk.data, 1e-6, None)
    e.record()
    torch.cuda.synchronize()
    ms = s.elapsed_time(e) / reps
    errs, same = [], 0
    for i in range(0, pairs, pairs // 8):
        got = O.Train(res.train(i).to_numpy())
        want = O.truncate(O.add(O.Train(ps[i]), O.Train(qs[i])), 1e-6)
        errs.append(O.tt_norm(O.add(got, O.scale(want, -1.0))) / O.tt_norm(want))
        same += int(list(got.bonds) == list(want.bonds))
    in_bytes = 8 * (pk.data.numel() + qk.data.numel())
    return {"workload": "1024 pairs of uniform rank-32 trains, d=16, n=4, summed to rank 64, "
                        "truncate(1e-6), one launch of ttb_round_batch", "pairs_per_s":
            pairs / (ms * 1e-3), "ms_per_launch": ms, "input_gb_s": in_bytes / (ms * 1e-3) / 1e9,
            "sample_rel_err_vs_fp64_oracle_max": max(errs),
            "sample_bonds_equal": f"{same}/{len(errs)}",
            "precision": "float64 (no 3xTF32 rounding variant)"}


def profile_case(mixed: bool = False):
    """The small case profiled with ncu: one persistent launch of 8 requests
    (2-D QTT Poisson with 8, 12, 16, 20 cores; diffusion d = 4, 6 with
    n = 16, 32), run twice (the second launch is the captured one).  With
    ``mixed`` the local solves above 50 unknowns are iterative and run in
    mixed precision, and the two d = 6 requests are left out (a capture of
    a few seconds per pass)."""
    import torch

    from ttnumpy_b200 import problems as P
    from ttnumpy_b200.persistent import PersistentBatch, prepare

    torch.cuda.set_device(0)
    kw = dict(residual_tol=TOL, symmetric=True, max_sweeps=MAX_SWEEPS, seed=0,
              stagnation_factor=None)
    if mixed:
        kw.update(precision="mixed", direct_solve_size=50)
    rng = np.random.default_rng(11)
    reqs = []
    for N in (4, 6, 8, 10):
        p = P.qtt_poisson_2d(N)
        p.meta["kind"] = "qtt"
        reqs.append((p.A, p.b, x0_host(p), kw))
    for d, n in ((4, 16), (4, 32)) + (() if mixed else ((6, 16), (6, 32))):
        q = P.parametric_diffusion(d, n, rng.uniform(-1, 1, size=d))
        reqs.append((q.A, q.b, None, kw))
    batch = PersistentBatch(prepare(reqs), 64)
    for _ in range(2):
        batch.launch()
        torch.cuda.synchronize()
    res = batch.collect()
    print(json.dumps({"status": [r.status for r in res],
                      "gflop": sum(r.flops for r in res) / 1e9,
                      "gflop_tc": sum(r.flops_tc for r in res) / 1e9,
                      "device_ms": [round(r.device_ms, 1) for r in res]}))


def main():
    args = parse()
    if args.profile_case:
        profile_case(args.profile_mixed)
        return
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        if rank == 0:
            reference_main(args)
        return  # the reference arm runs on rank 0's host cores alone

    import torch

    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=900))
    else:
        torch.cuda.set_device(0)
    from ttnumpy_b200 import kernels as K
    from ttnumpy_b200.persistent import prepare

    K.lib()
    B = args.requests
    n_value = (args.warmup + args.steps) * B
    reqs = make_requests(n_value + args.serve_requests, args.seed, args.preset)
    warm_reqs, timed_reqs = reqs[:args.warmup * B], reqs[args.warmup * B:n_value]
    serve_reqs = reqs[n_value:]
    kinds = [p.meta["kind"] for p in timed_reqs]

    def barrier():
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize()

    # inputs made resident before any timing
    warm = prepare([(p.A, p.b, x0_host(p), solve_kwargs(p)) for p in warm_reqs])
    timed = prepare([(p.A, p.b, x0_host(p), solve_kwargs(p)) for p in timed_reqs])
    for p in warm + timed:
        p.resident()
    torch.cuda.synchronize()
    if warm:
        resident_run(args, warm, torch)
    for p in warm:
        p.drop_resident()
    flush = torch.empty(64 << 20, dtype=torch.float64, device="cuda")  # 512 MB > L2
    K.fill_(flush, 0.0)
    barrier()
    with ClockSampler(local) as clocks:
        ms, jobs, launches, server = resident_run(args, timed, torch)
    barrier()
    solved = [_solved(j) for j in jobs]
    dev_s = [j.result.device_ms * 1e-3 if j.result is not None else 0.0 for j in jobs]
    flops = sum(j.result.flops for j in jobs if j.result is not None)
    peak_gb = server.peak_bytes / 2**30
    value, total_ms = aggregate_rate(sum(solved), ms, world)
    lats = [1e3 * j.latency for j in jobs if j.latency is not None]
    jobs = server = None
    for p in timed:
        p.drop_resident()
    del flush
    torch.cuda.empty_cache()

    # end to end through the server's public API from host memory
    cap = value / world
    sat = served_pass(args, serve_reqs, 2.0 * cap, torch, args.seed + 1)
    loads = []
    for f in [float(v) for v in args.serve_loads.split(",") if v.strip()]:
        r = served_pass(args, serve_reqs, f * cap, torch, args.seed + 2)
        loads.append({"load": f, "rate": r["rate"], "throughput": r["throughput"],
                      "solved": f"{r['solved']}/{r['requests']}", "latency_ms": r["latency_ms"]})
    e2e_value, _ = aggregate_rate(sat["solved"], 1e3 * sat["seconds"], world)
    n_pass = max(1, sat["requests"])
    e2e = {"value": e2e_value, "unit": UNIT,
           "h2d_bytes_per_step": int(sat["h2d"] * B / n_pass),
           "d2h_bytes_per_step": int(sat["d2h"] * B / n_pass),
           "mode": f"served: {sat['requests']} requests of the stream from host memory arriving "
                   f"as a Poisson stream at {sat['rate']:.2f}/s (twice the measured capacity), "
                   f"continuous batching over {args.streams} streams (and {args.light_streams} "
                   "high-priority streams for light requests) of persistent launches of "
                   f"at most {args.max_batch} requests admitted by a {args.serve_mem_gb:g} GB "
                   "work-area budget, inputs copied per launch, solutions read back; bytes per "
                   f"step scaled to {B} requests",
           "solved": f"{sat['solved']}/{sat['requests']}",
           "latency_ms": sat["latency_ms"], "peak_work_gb": sat["peak_gb"],
           "launches": sat["launches"], "sustainable_load": loads}

    plain = None
    if world == 1 and args.plain_sample > 0:
        plain = plain_run(reqs[:args.plain_sample], args.plain_limit, torch)
    secondary = None
    if world == 1:
        secondary = {"config2_rounding": rounding_run(torch), "config1_single_solve":
                     config1_run(torch)}
    if rank != 0:
        if world > 1:
            torch.distributed.destroy_process_group()
        return
    fp64 = fp64_peak_tflops(K, torch)
    ach = flops / (ms * 1e-3) / 1e12
    roof = {"kernel": "k_amen (ttb_amen_persistent)", "bound": "tensor", "unit": "TFLOP/s",
            "achieved": ach, "peak": fp64, "peak_source": "measured FP64 FMA probe "
            "(ttb_fma_peak); MEASURED_PEAKS.json has no FP64 figure",
            "frac": ach / fp64, "traffic": None,
            "traffic_source": "not measured for this workload in this run (ncu DRAM counters "
                              "come from a separate small-case capture)",
            "flops_counted": "2mnk of every dense product and 2 nnz n of every sparse "
                             "operator-core product the blocks ran; QR/SVD/LU not counted",
            "timing": "device time of the whole timed run (all steps' requests queued at once)"}
    cpu = None
    if world == 1:
        n_cpu = args.cpu_sample or 2 * cpu_cores()
        cpu = cpu_baseline(reqs[:n_cpu], cpu_cores(), args.time_limit)
        # config 1 on one host core, uncapped (the secondary single-solve line)
        dt, conv, _ = cpu_run([config1_problem()], 1, 1e9)[1][0]
        secondary["config1_single_solve"]["cpu_oracle_s"] = dt
        secondary["config1_single_solve"]["cpu_oracle_converged"] = conv
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": config(args),
            "solved": f"{sum(solved)}/{len(solved)}",
            "classes": class_stats(kinds, solved, dev_s),
            "latency_ms": {"p50": percentile(lats, 50), "p99": percentile(lats, 99)},
            "peak_work_gb": peak_gb,
            "roofline": roof, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches,
            "plain_gpu": plain, "clocks": clocks.summary(), "secondary": secondary}
    print(json.dumps(line), flush=True)
    if world > 1:
        torch.distributed.destroy_process_group()


def reference_main(args):
    """The reference arm: the CPU oracle on the host cores.  Each step
    solves the next ``cores`` requests of the stream (one per worker), each
    capped at ``--cpu-limit`` seconds; warm-up steps solve one small
    request per worker."""
    cores = cpu_cores()
    B = args.requests
    reqs = make_requests((args.warmup + args.steps) * B, args.seed, args.preset)
    small = [p for p in reqs if p.meta["kind"] == "qtt"][:cores] or reqs[:1]
    for _ in range(args.warmup):
        cpu_run(small, cores, args.time_limit)
    total, cpu_s, res_all = 0.0, 0.0, []
    for k in range(args.steps):
        start = (args.warmup + k) * B
        sample = reqs[start:start + min(cores, B)]
        dt, res = cpu_run(sample, cores, args.time_limit)
        total += dt
        cpu_s += sum(r[0] for r in res)
        res_all += res
    solved = sum(1 for r in res_all if r[1])
    value = solved / (cpu_s / cores)
    sample_txt = (f"{min(cores, B)} requests per step (the first of each step's batch of the "
                  "stream), "
                  f"{cores} single-threaded oracle workers, each solve capped at "
                  f"{args.time_limit:g} s; value = solved / (sum of solve seconds / cores)")
    line = {"metric": METRIC, "value": value, "unit": UNIT, "impl": "reference",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * total / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": config(args, engine="reference"),
            "solved": f"{solved}/{len(res_all)}",
            "classes": class_stats([r[2] for r in res_all], [r[1] for r in res_all],
                                   [r[0] for r in res_all]),
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": sample_txt},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def percentile(v, q):
    if not v:
        return None
    return float(np.percentile(np.asarray(v, dtype=np.float64), q))


def config(args, engine="persistent server"):
    if args.preset == "config5":
        work = ("AMEn serving mix (stream of requests): 10% large diffusion d=24 n=64 with "
                "rank-8 right-hand side, 45% parametric diffusion d~U{4..12} n~U{16,32,64}, 45% "
                "2-D QTT Poisson with 6-20 cores; residual 1e-8, at most 30 sweeps")
    else:
        work = ("AMEn reduced mix: 2-D QTT Poisson (6-20 cores) and parametric diffusion "
                "(d in 4,5, n in 16,32); residual 1e-8, at most 30 sweeps")
    out = {"workload": work, "requests_per_step": args.requests, "engine": engine,
           "max_sweeps": MAX_SWEEPS, "stagnation_factor": None,
           "per_solve_time_limit_s": args.time_limit,
           "time_limit_rule": "the same in every arm (device time of a solve on the GPU, host "
                              "time of a solve on the CPU); a solve stopped by it is not solved",
           "parallelism": f"replicas x{args.gpus}"}
    if engine != "reference":
        out["cluster"] = "mode-64 requests on clusters of 4 blocks" if args.cluster else "one block per solve"
    if engine != "reference":
        out["l2"] = ("inputs larger than L2 (each request's work area is tens to hundreds of "
                     "MB); 512 MB flush before the timed region")
        out["steps"] = ("the timed steps' requests (consecutive batches of the stream) queued "
                        "at once, longest first, to the server on device-resident inputs")
    return out


if __name__ == "__main__":
    main()
