#!/usr/bin/env python
"""Benchmark of the GB300 sparse-FFT engine on its headline workload.

Workload (one "step" = one batch of transforms): sFFT v2, n = 2^22,
k = 100, magnitudes log-uniform in [0.1, 10], uniform phases, complex
Gaussian noise at 20 dB SNR (seeded synthetic signals of that shape; no
dataset is involved).  The headline `value` is the FP32 form's whole-job
throughput in solves/s on inputs resident in HBM (a pool of signals larger
than L2, cycled through); the FP64 parity form is measured beside it, with
p50/p99 latencies and the FP32-vs-FP64 per-entry L1 error.  `e2e` is the
same metric through the drop-in C call sfft_exec_many with page-locked host
buffers (input copies and dense outputs inside the timed region).

    python bench.py [--gpus N --steps K --warmup W] [--impl reference]

Multi-GPU: requests are independent, so N GPUs run N replicas (weak
scaling, no collective on the data path); torchrun launches one rank per GPU.
"""
import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "sFFT solves/s + p50/p99 latency (n=2^22,k=100), FP32 vs FP64 at L1 err ≤1e-4"
N_SIG, K_SIG, VERSION = 1 << 22, 100, 2
MAG, SNR, SEED = (0.1, 10.0), 20.0, 7
L2_BYTES = 129 * 1024 * 1024


def args_():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--batch", type=int, default=32)
    ap.add_argument("--pool", type=int, default=64)
    ap.add_argument("--only", default="all", choices=["all", "device", "uneven", "stream", "configs"],
                    help="device: only the device-resident timed legs (for profiler captures); "
                         "uneven: only the 256-signal uneven batch; stream: only the mixed serving stream")
    ap.add_argument("--stream-requests", type=int, default=10000, help="requests in the mixed serving stream")
    ap.add_argument("--stream-limit", type=float, default=240.0,
                    help="seconds each form of the serving stream may take (plan builds included)")
    a = ap.parse_args()
    a.warmup = max(a.warmup, 3)
    return a


# Process-group backend: nccl on GPUs; gloo (SFFT_BENCH_BACKEND=gloo) lets
# the rank logic run on CPU.
BACKEND = os.environ.get("SFFT_BENCH_BACKEND", "nccl")


def dist_init():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch
        import torch.distributed as dist
        if BACKEND == "nccl":
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", device_id=torch.device("cuda", local))
        else:
            dist.init_process_group(BACKEND)
    return ws, rank, local


def barrier(ws):
    if ws > 1:
        import torch.distributed as dist
        dist.barrier()


def max_over_ranks(ws, v):
    """The largest of the ranks' values (the job's time is its slowest rank's)."""
    if ws == 1:
        return v
    import torch
    import torch.distributed as dist
    t = torch.tensor([v], dtype=torch.float64, device="cuda" if BACKEND == "nccl" else "cpu")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ------------------------------------------------------------------ clocks --

class Clocks:
    """nvidia-smi samples during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu):
        self.gpu = gpu
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), "--query-gpu=" + self.Q,
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.p:
            self.p.terminate()
            self.p.wait()

    def summary(self):
        self.f.flush()
        rows = []
        with open(self.f.name) as fh:
            for line in fh:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        os.unlink(self.f.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        pw = [float(r[3]) for r in rows if r[3].replace(".", "").isdigit()]
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows), "power_w_max": max(pw) if pw else None}


# --------------------------------------------------------------- CPU legs --

def cpu_signals(count):
    from sfft_gb300 import signals
    return [signals.make_signal(N_SIG, K_SIG, SEED + i, mag=MAG, snr_db=SNR)[0] for i in range(count)]


def _omp_threads(t):
    """Sets the OpenMP thread count of this process (libgomp, shared by the
    reference build and the oracle)."""
    try:
        ctypes.CDLL("libgomp.so.1").omp_set_num_threads(int(t))
    except OSError:
        pass


def cpu_reference_throughput(steps, warmup, sample, threads=None):
    """The reference's CPU implementation on this host: the unmodified
    sFFT 0.1 build with its own flags (-O3 -ffast-math -march=native,
    wscript:10) when it was built here (oracle/_ref), else the oracle port,
    OpenMP over signals like sfft_exec_many on `threads` threads (default:
    every core).  Returns (solves/s, kind, threads, step times)."""
    from oracle import oracle as O
    cores = threads or os.cpu_count() or 1
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
    _omp_threads(cores)       # before the plan: its scratch is per OpenMP thread
    kind = "port"
    sigs = cpu_signals(min(4, sample))
    ins = [sigs[i % len(sigs)] for i in range(sample)]
    ref = None
    try:
        ref = O.RefLib("libsfft_ref_fast.so")
        kind = "reference"
    except (OSError, FileNotFoundError):
        ref = None
    if ref is not None:
        plan = ref.plan(N_SIG, K_SIG, VERSION - 1)
        outs = [np.empty(N_SIG, dtype=np.complex128) for _ in ins]
        pin = (ctypes.c_void_p * len(ins))(*[x.ctypes.data for x in ins])
        pout = (ctypes.c_void_p * len(ins))(*[o.ctypes.data for o in outs])

        def one():
            ref.L.sfft_exec_many(plan, len(ins), pin, pout)
    else:
        O.build()
        plan = O.OraclePlan(N_SIG, K_SIG, VERSION - 1)

        def one():
            plan.exec_many_dense(ins)
    O.seed_libc(SEED)
    for _ in range(warmup):
        one()
    times = []
    for _ in range(steps):
        t0 = time.perf_counter()
        one()
        times.append(time.perf_counter() - t0)
    if ref is not None:
        ref.free(plan)
    _omp_threads(os.cpu_count() or 1)
    return sample * steps / sum(times), kind, cores, times


def reference_arm(a, ws, rank):
    if rank != 0:
        return
    # a bounded sample per step (one transform per core): the default
    # --steps 200 run ends in under two minutes on 16 cores
    sample = max(2, min(os.cpu_count() or 1, 16))
    sps, kind, cores, times = cpu_reference_throughput(a.steps, a.warmup, sample)
    sps1, kind1, _, _ = cpu_reference_throughput(2, 1, 1, threads=1)
    line = {
        "metric": METRIC, "value": sps, "unit": "solves/s", "n_gpus": a.gpus, "steps": a.steps,
        "warmup": a.warmup, "ms_per_step": 1e3 * statistics.mean(times), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "impl": "reference",
        "config": config(a),
        "cpu_baseline": {"value": sps, "unit": "solves/s", "cores": cores, "kind": kind,
                         "sample": f"{sample} transforms per step (v2 n=2^22 k=100), OpenMP over signals"},
        "e2e": {"value": sps, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "cpu_baseline_1t": {"value": sps1, "unit": "solves/s", "cores": 1, "kind": kind1,
                            "sample": "1 transform x 2 steps, one thread"},
    }
    print(json.dumps(line), flush=True)


def config(a):
    return {"workload": "sfft_v2_n4194304_k100_snr20_mag0.1-10", "version": "v2", "n": N_SIG, "k": K_SIG,
            "global_batch": a.batch * a.gpus, "batch_per_gpu": a.batch, "parallelism": f"replicas{a.gpus}",
            "l2": f"inputs larger than L2: pool of {a.pool} signals x {N_SIG * 16 >> 20} MiB cycled per step",
            "precision": "fp32 headline, fp64 beside"}


# ------------------------------------------------------------------- GPU ---

def gb300_arm(a, ws, rank, local):
    import torch
    from sfft_gb300 import _lib, build, signals
    from sfft_gb300.sfft import sfft

    torch.cuda.set_device(local)
    build.build()
    L = _lib.load()
    dev = torch.device("cuda", local)
    pool = [signals.make_signal_torch(N_SIG, K_SIG, SEED + 1000 * rank + i, mag=MAG, snr_db=SNR,
                                      device=dev)[0] for i in range(a.pool)]
    torch.cuda.synchronize()
    B = a.batch
    p32 = sfft(N_SIG, K_SIG, VERSION, precision="fp32", device=local, max_batch=B)
    p64 = sfft(N_SIG, K_SIG, VERSION, precision="fp64", device=local, max_batch=B)
    cap = p32.capacity
    oidx = torch.empty((B, cap), dtype=torch.int32, device=dev)
    oval32 = torch.empty((B, cap), dtype=torch.complex64, device=dev)
    oval64 = torch.empty((B, cap), dtype=torch.complex128, device=dev)
    ocnt = torch.empty(B, dtype=torch.int32, device=dev)
    stream = torch.cuda.Stream(device=dev)     # a real handle: the library launches on it
    torch.cuda.set_stream(stream)
    ptr_sets = []
    for s in range(max(1, a.pool // B) + 1):
        ptrs = [pool[(s * B + j) % a.pool].data_ptr() for j in range(B)]
        ptr_sets.append((ctypes.c_void_p * B)(*ptrs))

    def step(plan, oval, i):
        rc = L.sfft_exec_batch(plan.sfft_plan, B, ptr_sets[i % len(ptr_sets)], _lib.SFFT_IN_C128,
                               oidx.data_ptr(), oval.data_ptr(), ocnt.data_ptr(), cap,
                               ctypes.c_void_p(stream.cuda_stream))
        if rc != 0:
            raise RuntimeError(_lib.last_error())

    def timed(plan, oval, steps, warmup, profile=False, clocks=None):
        for i in range(warmup):
            step(plan, oval, i)
        torch.cuda.synchronize()
        if profile:
            L.sfft_profile(plan.sfft_plan, 1)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
        barrier(ws)
        torch.cuda.synchronize()
        launches0 = L.sfft_kernel_launches()
        ev[0].record(stream)
        for i in range(steps):
            step(plan, oval, warmup + i)
            ev[i + 1].record(stream)
        torch.cuda.synchronize()
        barrier(ws)
        launches = L.sfft_kernel_launches() - launches0
        per = [ev[i].elapsed_time(ev[i + 1]) for i in range(steps)]
        total = ev[0].elapsed_time(ev[steps])
        stages = None
        if profile:
            ms = (ctypes.c_double * 8)()
            cnt = L.sfft_profile_read(plan.sfft_plan, ms, 8)
            L.sfft_profile(plan.sfft_plan, 0)
            stages = (list(ms)[:4], cnt)
        return total, per, launches, stages

    if a.only == "stream":
        if rank == 0:
            print(json.dumps({"serving_stream_fp32": stream_leg(L, _lib, local, 1, a.stream_requests, limit_s=420),
                              "serving_stream_fp64": stream_leg(L, _lib, local, 0, a.stream_requests, limit_s=300)}),
                  flush=True)
        return
    if a.only == "configs":
        if rank == 0:
            print(json.dumps({"other_configs": configs_leg(L, _lib, local)}), flush=True)
        return
    if a.only == "uneven":
        if rank == 0:
            print(json.dumps({"uneven_batch": uneven_leg(L, _lib, local),
                              "uneven_batch_persistent": uneven_leg(L, _lib, local, persistent=True),
                              "uneven_batch_fp64": uneven_leg(L, _lib, local, precision=0)}), flush=True)
        return

    # ---- FP32 headline (clocks sampled during its timed region)
    with Clocks(local) as clk:
        t32, per32, launches32, st32 = timed(p32, oval32, a.steps, a.warmup, profile=True)
    clocks = clk.summary()
    t32max = max_over_ranks(ws, t32)
    value = ws * B * a.steps / (t32max / 1e3)
    # ---- FP32 in the opt-in v2 voted mode (estimates voted candidates only)
    p32v = sfft(N_SIG, K_SIG, VERSION, precision="fp32", device=local, max_batch=B)
    if L.sfft_plan_v2_voted(p32v.sfft_plan, 1) != 0 or L.sfft_output_capacity(p32v.sfft_plan) > cap:
        raise RuntimeError("voted mode: " + _lib.last_error())
    t32v, per32v, _, st32v = timed(p32v, oval32, a.steps, a.warmup, profile=True)
    value_voted = ws * B * a.steps / (max_over_ranks(ws, t32v) / 1e3)
    # ---- FP64 parity form
    s64 = max(3, a.steps // 8)
    t64, per64, _, st64 = timed(p64, oval64, s64, 3, profile=True)
    t64max = max_over_ranks(ws, t64)
    value64 = ws * B * s64 / (t64max / 1e3)
    if a.only == "device":
        if rank == 0:
            print(json.dumps({"metric": METRIC, "value": value, "unit": "solves/s", "fp64_value": value64,
                              "fp32_voted_value": value_voted,
                              "only": "device", "stage_ms_per_launch_fp32": stage_table(st32),
                              "stage_ms_per_launch_fp32_voted": stage_table(st32v),
                              "stage_ms_per_launch_fp64": stage_table(st64)}), flush=True)
        return

    # ---- single-request latency (batch of one)
    def lat(plan, oval, runs=30):
        out = []
        for i in range(runs + 3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            rc = L.sfft_exec_batch(plan.sfft_plan, 1, ptr_sets[0], _lib.SFFT_IN_C128, oidx.data_ptr(),
                                   oval.data_ptr(), ocnt.data_ptr(), cap, ctypes.c_void_p(stream.cuda_stream))
            assert rc == 0, _lib.last_error()
            e1.record(stream)
            e1.synchronize()
            if i >= 3:
                out.append(e0.elapsed_time(e1))
        return out
    lat32, lat64 = lat(p32, oval32), lat(p64, oval64)

    # ---- serving: Poisson arrivals at 80% of each form's batched throughput
    serve32 = serving_leg(L, _lib, pool, 1, 0.8, 4000, local)
    serve64 = serving_leg(L, _lib, pool, 0, 0.65, 1500, local)   # smaller batches under Poisson arrivals

    # ---- accuracy: FP32 vs FP64 on the same draws, and both vs the truth
    acc = accuracy(p32, p64, signals, p32v)

    # ---- roofline of the dominant stage (live CUDA events)
    roof, pipeline = roofline(p32, st32, B)

    # ---- e2e through the drop-in call with page-locked host buffers, and
    # the same transforms with sparse host outputs
    e2e = e2e_leg(L, p32, pool, B, a)
    e2e["sparse_outputs"] = e2e_sparse_leg(L, p32, pool, B, a)

    # ---- 256 signals of uneven (n, k) as one CUDA graph: per-plan kernel
    # branches, and the persistent executor (one kernel launch per call)
    uneven = uneven_leg(L, _lib, local)
    uneven_p = uneven_leg(L, _lib, local, persistent=True)
    # ---- the other named configurations (C1 v1, C2 v3)
    other = configs_leg(L, _lib, local)
    # ---- C5: the mixed serving stream (10,000 requests), both forms, each
    # within its own time limit (plans are built before its timed region)
    del pool
    torch.cuda.empty_cache()
    stream5 = {"fp32": stream_leg(L, _lib, local, 1, a.stream_requests, limit_s=a.stream_limit),
               "fp64": stream_leg(L, _lib, local, 0, a.stream_requests, limit_s=a.stream_limit)}

    line = {
        "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": ws, "steps": a.steps,
        "warmup": a.warmup, "ms_per_step": t32max / a.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded k-sparse + AWGN, device-generated)",
        "config": config(a),
        "p50_ms": serve32["p50_ms"], "p99_ms": serve32["p99_ms"],
        "latency_basis": "submit-to-completion of requests arriving as a Poisson process at 80% (FP32) / 65% "
                         "(FP64) of the server's burst capacity, through the continuous-batching server "
                         "(sfft_server_*)",
        "serving": {"fp32": serve32, "fp64": serve64},
        "batch_step_ms": {"p50": pct(per32, 50), "p99": pct(per32, 99)},
        "fp32_over_fp64": value / value64,
        "fp64": {"value": value64, "unit": "solves/s", "ms_per_step": t64max / s64,
                 "p50_ms": serve64["p50_ms"], "p99_ms": serve64["p99_ms"],
                 "batch_step_p50_ms": pct(per64, 50), "batch_step_p99_ms": pct(per64, 99),
                 "fp32_speedup": value / value64},
        "fp32_voted": {"value": value_voted, "unit": "solves/s", "ms_per_step": max_over_ranks(ws, t32v) / a.steps,
                       "batch_step_p50_ms": pct(per32v, 50), "batch_step_p99_ms": pct(per32v, 99),
                       "stage_ms_per_launch": stage_table(st32v),
                       "mode": "opt-in v2 voted mode (sfft_plan_v2_voted): only candidates that reach the vote "
                               "threshold are estimated; the reference estimates and returns every comb "
                               "candidate"},
        "latency_single_ms": {"fp32_p50": pct(lat32, 50), "fp32_p99": pct(lat32, 99),
                              "fp64_p50": pct(lat64, 50), "fp64_p99": pct(lat64, 99)},
        "accuracy": acc,
        "roofline": roof,
        "pipeline_roofline": pipeline,
        "stage_ms_per_launch_fp32": stage_table(st32),
        "stage_ms_per_launch_fp64": stage_table(st64),
        "e2e": e2e,
        "uneven_batch": uneven,
        "uneven_batch_persistent": uneven_p,
        "other_configs": other,
        "serving_stream": stream5,
        "gpu_launches": launches32,
        "clocks": clocks,
    }
    if rank == 0 and ws == 1:
        sample = max(2, min(2 * (os.cpu_count() or 1), 32))
        sps, kind, cores, _ = cpu_reference_throughput(2, 1, sample)
        line["cpu_baseline"] = {"value": sps, "unit": "solves/s", "cores": cores, "kind": kind,
                                "sample": f"{sample} transforms x 2 steps of the same workload, "
                                          "OpenMP over signals"}
        sps1, kind1, _, _ = cpu_reference_throughput(2, 1, 1, threads=1)
        line["cpu_baseline_1t"] = {"value": sps1, "unit": "solves/s", "cores": 1, "kind": kind1,
                                   "sample": "1 transform x 2 steps of the same workload, one thread"}
    if rank == 0:
        print(json.dumps(line), flush=True)


def configs_leg(L, _lib, local, reps=20):
    """The other named configurations, FP64 (their plain form): C1 v1
    n = 2^16, k = 50 and C2 v3 n = 2^24, k = 1000, noiseless |X| = 1: batched
    throughput, single-request latency and recovery against the truth."""
    import torch
    from sfft_gb300 import signals
    out = {}
    for name, n, k, ver, batch, seed in (("C1_v1_n65536_k50", 1 << 16, 50, 0, 64, 0),
                                         ("C2_v3_n16777216_k1000", 1 << 24, 1000, 2, 4, 1)):
        sig = [signals.make_signal_torch(n, k, seed + s, device=torch.device("cuda", local)) for s in range(batch)]
        o = _lib.Options(0, local, batch)
        p = L.sfft_make_plan_ex(n, k, ver, 0, ctypes.byref(o))
        if not p:
            out[name] = {"error": _lib_err(L)}
            continue
        cap = L.sfft_output_capacity(p)
        idx = torch.empty((batch, cap), dtype=torch.int32, device=sig[0][0].device)
        val = torch.empty((batch, cap), dtype=torch.complex128, device=sig[0][0].device)
        cnt = torch.zeros(batch, dtype=torch.int32, device=sig[0][0].device)
        stream = torch.cuda.ExternalStream(L.sfft_plan_stream(p))
        ins = (ctypes.c_void_p * batch)(*[x.data_ptr() for x, _, _ in sig])
        seeds = (ctypes.c_uint * batch)(*range(batch))

        def run(m):
            if L.sfft_exec_batch_ex(p, m, ins, 0, seeds, ctypes.c_void_p(idx.data_ptr()),
                                    ctypes.c_void_p(val.data_ptr()), ctypes.c_void_p(cnt.data_ptr()), cap, None):
                raise RuntimeError(_lib_err(L))

        def timed(m):
            ts = []
            for i in range(reps + 3):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                run(m)
                e1.record(stream)
                e1.synchronize()
                if i >= 3:
                    ts.append(e0.elapsed_time(e1))
            return ts

        tb, t1 = timed(batch), timed(1)
        # per-stage device time of single requests (v1: comb, fold, bucket, estimate; v3: filters, peel)
        L.sfft_sync(p)
        L.sfft_profile(p, 1)
        for _ in range(5):
            run(1)
        L.sfft_sync(p)
        ms = (ctypes.c_double * 8)()
        nprof = L.sfft_profile_read(p, ms, 8)
        L.sfft_profile(p, 0)
        names = ["filters", "peel"] if ver == 2 else STAGES
        stages1 = {nm: ms[i] / nprof for i, nm in enumerate(names)} if nprof > 0 else None
        run(batch)
        L.sfft_sync(p)
        scores = []
        for s in range(batch):
            c = int(cnt[s])
            x, pos, vals = sig[s]
            scores.append(score_result(x, pos, vals, idx[s, :c].cpu().numpy(), val[s, :c].cpu().numpy(), ver < 2))
        L.sfft_free_plan(p)
        out[name] = {"solves_per_s": batch / (1e-3 * float(np.median(tb))), "batch": batch,
                     "batch_ms_p50": pct(tb, 50), "single_ms_p50": pct(t1, 50), "single_ms_p99": pct(t1, 99),
                     "single_stage_ms": stages1, "accuracy": merge_scores(scores), "precision": "fp64"}
        del sig
        torch.cuda.empty_cache()
    return out


def uneven_shapes(count=256):
    """(n, k) of the uneven batch: n log-uniform over 2^16..2^22, k uniform
    in [10, 500], drawn from seed s for signal s."""
    out = []
    for s in range(count):
        r = np.random.default_rng(s)
        out.append((1 << int(r.integers(16, 23)), int(r.integers(10, 501))))
    return out


def uneven_leg(L, _lib, local, steps=20, warmup=3, precision=1, persistent=False):
    """256 v2 signals of uneven (n, k) (k-sparse, magnitude 1, 40 dB SNR,
    seeds 0..255) through sfft_mixed_*: autotuned constants per (n, k
    bucket), every plan's batched pipeline a branch of one CUDA graph that is
    replayed per call."""
    import torch
    from sfft_gb300 import signals
    shapes = uneven_shapes()
    num = len(shapes)
    sigs = [signals.make_signal_torch(n, k, s, snr_db=40.0, device=torch.device("cuda", local))
            for s, (n, k) in enumerate(shapes)]
    torch.cuda.synchronize()
    arr = lambda vals: (ctypes.c_int * num)(*vals)
    t0 = time.perf_counter()
    m = L.sfft_mixed_create(num, arr([n for n, _ in shapes]), arr([k for _, k in shapes]), arr([1] * num),
                            arr([precision] * num), 0, 2, local)
    if not m:
        return {"error": _lib_err(L)}
    if persistent and L.sfft_mixed_set_persistent(m, 1) != 0:
        return {"error": _lib_err(L)}
    ins = (ctypes.c_void_p * num)(*[x.data_ptr() for x, _, _ in sigs])
    seeds = (ctypes.c_uint * num)(*range(num))

    def run():
        if L.sfft_mixed_exec(m, ins, seeds) != 0:
            raise RuntimeError(_lib_err(L))

    l0 = L.sfft_kernel_launches()
    run()
    first_launches = L.sfft_kernel_launches() - l0   # the direct first call; later calls replay its graph
    if L.sfft_mixed_sync(m) != 0:
        raise RuntimeError(_lib_err(L))
    setup = time.perf_counter() - t0
    stream = torch.cuda.ExternalStream(L.sfft_mixed_stream(m))
    for _ in range(warmup):
        run()
    L.sfft_mixed_sync(m)
    dev, wall = [], []
    for _ in range(steps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        w0 = time.perf_counter()
        e0.record(stream)
        run()
        e1.record(stream)
        e1.synchronize()
        wall.append(time.perf_counter() - w0)
        dev.append(e0.elapsed_time(e1) * 1e-3)
    L.sfft_mixed_sync(m)
    # accuracy of the last call against the dense FFT of each input and the drawn spectra
    scores = []
    for s, (x, pos, vals) in enumerate(sigs):
        c = L.sfft_mixed_result_host(m, s, None, None, 0)
        hi = np.empty(max(c, 1), dtype=np.int32)
        hv = np.empty(max(c, 1), dtype=np.complex64 if precision else np.complex128)
        if L.sfft_mixed_result_host(m, s, hi.ctypes.data, hv.ctypes.data, c) != c:
            raise RuntimeError(_lib_err(L))
        scores.append(score_result(x, pos, vals, hi[:c], hv[:c], True))
    groups = L.sfft_mixed_groups(m)
    L.sfft_mixed_destroy(m)
    return {"signals": num, "plans": groups, "precision": "fp32" if precision else "fp64",
            "solves_per_s": num / float(np.median(dev)), "ms_per_call": 1e3 * float(np.median(dev)),
            "ms_per_call_p99": 1e3 * pct(dev, 99),
            "wall_solves_per_s": num / float(np.median(wall)),
            "setup_s": setup, "kernel_launches_per_call": first_launches,
            "accuracy": merge_scores(scores),
            "executor": "one persistent kernel over a device work queue" if persistent
                        else "one CUDA graph of per-plan kernel branches",
            "workload": "256 v2 signals, n log-uniform 2^16..2^22, k uniform [10,500], |X|=1, 40 dB SNR, "
                        "seeds 0..255; autotuned constants per (n, k bucket); one CUDA graph per call"}


def stream_requests(nreq, seed=42):
    """The mixed serving stream: n log-uniform over 2^14..2^26, k uniform in
    [1, min(2000, n/1024)], v2 (noisy, 30 dB SNR) or v3 (noiseless) 50/50,
    complex64 or complex128 input 50/50, all drawn from one seeded stream."""
    r = np.random.default_rng(seed)
    out = []
    for _ in range(nreq):
        n = 1 << int(r.integers(14, 27))
        k = int(r.integers(1, min(2000, n // 1024) + 1))
        version = 3 if r.random() < 0.5 else 2
        c64 = bool(r.random() < 0.5)
        out.append((n, k, version, c64))
    return out


def stream_leg(L, _lib, local, precision, nreq, **kw):
    """stream_leg_ with its time limit turned into an error entry."""
    try:
        return stream_leg_(L, _lib, local, precision, nreq, **kw)
    except TimeoutError as e:
        return {"error": str(e)}


def stream_leg_(L, _lib, local, precision, nreq, budget_gb=160, max_batch=8, load=0.8, seed=42, limit_s=900):
    """The mixed stream through the continuous-batching server: plans are
    built once per (n, k bucket, version) and kept on the device under an
    HBM budget; a closed-loop burst measures capacity, then the requests
    arrive as a Poisson process at `load` x capacity."""
    import threading
    import torch
    from sfft_gb300 import signals
    t_start = time.perf_counter()
    reqs = stream_requests(nreq, seed)
    dev = torch.device("cuda", local)
    sig = {}

    def signal_for(n, k, version, c64):
        t = 1 << (k.bit_length() - 1)              # tones: largest power of two <= k
        key = (n, t, version, c64)
        if key not in sig:
            base = (n, t, version, False)
            if base not in sig:
                x, _, _ = signals.make_signal_torch(n, t, (n * 31 + t) * 2 + version, device=dev,
                                                    snr_db=30.0 if version == 2 else None)
                sig[base] = x
            if c64:
                sig[key] = sig[base].to(torch.complex64)
        return sig[key]

    ptr = [ctypes.c_void_p(signal_for(*q).data_ptr()) for q in reqs]
    torch.cuda.synchronize()
    sig_bytes = sum(x.numel() * x.element_size() for x in sig.values())
    voted = 1 if precision == 1 else 0          # the FP32 serving form runs v2 in the voted mode
    opts = _lib.ServerOptions(local, max_batch, int(budget_gb * (1 << 30)), 2, 2, voted)
    srv = L.sfft_server_create(ctypes.byref(opts))
    if not srv:
        return {"error": _lib.last_error()}
    lat = ctypes.c_double()
    try:
        return _stream_phases(L, srv, reqs, ptr, precision, nreq, load, seed, limit_s, lat, t_start, sig, voted,
                              budget_gb)
    finally:
        L.sfft_server_destroy(srv)
        sig.clear()
        torch.cuda.empty_cache()


def _stream_phases(L, srv, reqs, ptr, precision, nreq, load, seed, limit_s, lat, t_start, sig, voted, budget_gb):
    import threading
    sig_bytes = sum(x.numel() * x.element_size() for x in sig.values())

    def submit(i, seed_):
        n, k, version, c64 = reqs[i]
        return L.sfft_server_submit(srv, n, k, version - 1, precision, ptr[i], 1 if c64 else 0, seed_)

    deadline = [time.perf_counter() + limit_s]

    def wait(rid):
        # bounded: a stream that stops making progress ends the leg with an error
        left_ms = 1e3 * (deadline[0] - time.perf_counter())
        c = L.sfft_server_wait_for(srv, rid, None, None, 0, ctypes.byref(lat), max(1.0, left_ms))
        if c == -2:
            raise TimeoutError("serving stream made no progress within its time limit")
        return c, lat.value

    def log(msg):
        print(f"[stream {'fp32' if precision == 1 else 'fp64'}] {msg} ({time.perf_counter() - t_start:.0f} s)",
              file=sys.stderr, flush=True)

    log(f"{len(sig)} signals ({sig_bytes / 2**30:.1f} GiB) on the device")
    # plans: one request per distinct plan, outside the timed region
    t0 = time.perf_counter()
    first = {}
    for i, (n, k, version, c64) in enumerate(reqs):
        kk = L.sfft_tuned_k(k) if version == 2 else max(8, 1 << (max(k, 1) - 1).bit_length())
        first.setdefault((n, kk, version), i)
    fails, errors = 0, set()
    for i in first.values():
        c, _ = wait(submit(i, i))
        if c < 0:
            fails += 1
            errors.add(f"{reqs[i][:3]}: {L.sfft_last_error().decode()}")
    plan_s = time.perf_counter() - t0
    log(f"{len(first)} plans built")
    # capacity: every request submitted at once
    burst = min(nreq, 2000)
    t0 = time.perf_counter()
    ids = [submit(i, 7 + i) for i in range(burst)]
    for rid in ids:
        wait(rid)
    capacity = burst / (time.perf_counter() - t0)
    log(f"burst of {burst}: {capacity:.0f} solves/s")
    # the timed stream
    rate = load * capacity
    gaps = np.random.default_rng(seed + 1).exponential(1.0 / rate, size=nreq)
    ids = [None] * nreq
    lats = [0.0] * nreq
    failed = [0]
    done_t = [0.0]

    fail_msgs = {}

    def waiter():
        for i in range(nreq):
            while ids[i] is None:
                time.sleep(0)
            c, ms = wait(ids[i])
            lats[i] = ms
            if c < 0:
                failed[0] += 1
                key = (reqs[i][2], L.sfft_last_error().decode()[:120])
                fail_msgs.setdefault(key, []).append(reqs[i][:2])
        done_t[0] = time.perf_counter()

    err = []

    def waiter_safe():
        try:
            waiter()
        except TimeoutError as e:
            err.append(str(e))

    th = threading.Thread(target=waiter_safe)
    th.start()
    t0 = time.perf_counter()
    t_next = t0
    for i in range(nreq):
        t_next += gaps[i]
        while time.perf_counter() < t_next:
            pass
        if time.perf_counter() > deadline[0] or err:  # out of time: stop offering load
            for j in range(i, nreq):
                ids[j] = -1
            break
        ids[i] = submit(i, 100000 + i)
    th.join()
    log("stream done" if not err else err[0])
    if err:
        return {"error": err[0]}
    stats = (ctypes.c_long * 9)()
    L.sfft_server_stats(srv, stats, 9)
    by_v = {v: [lats[i] for i in range(nreq) if reqs[i][2] == v] for v in (2, 3)}
    return {"requests": nreq, "precision": "fp32" if precision == 1 else "fp64 (v3 always fp64)",
            "solves_per_s": nreq / (done_t[0] - t0), "offered_rate": rate, "capacity_burst_solves_per_s": capacity,
            "p50_ms": pct(lats, 50), "p99_ms": pct(lats, 99),
            "p50_ms_v2": pct(by_v[2], 50), "p99_ms_v2": pct(by_v[2], 99),
            "p50_ms_v3": pct(by_v[3], 50), "p99_ms_v3": pct(by_v[3], 99),
            "failed": failed[0], "plans_failed": fails, "plan_errors": sorted(errors)[:5],
            "failures": [{"version": v, "error": m, "count": len(nk), "n_k_examples": nk[:4]}
                         for (v, m), nk in sorted(fail_msgs.items(), key=lambda t: -len(t[1]))[:5]],
            "plans_built": len(first), "plan_build_s": plan_s,
            "batches": int(stats[0]), "plans_evicted": int(stats[2]), "deferred": int(stats[3]),
            "batches_spilled_to_host": int(stats[8]), "v2_mode": "voted" if voted else "reference (all comb candidates)",
            "hbm_budget_gb": budget_gb, "signal_pool_gb": sig_bytes / 2**30,
            "workload": "n log-uniform 2^14..2^26, k uniform [1, min(2000, n/1024)], v2 (30 dB SNR) or v3 "
                        "(noiseless) 50/50, complex64/complex128 50/50, seed 42; Poisson arrivals at "
                        f"{load:.0%} of the burst capacity; v1/v2 autotuned per (n, k bucket), v3 k rounded "
                        "up to a power of two (at least 8)"}


def serving_leg(L, _lib, pool, precision, load, nreq, device):
    """Requests of the bench workload submitted at Poisson times to a
    continuous-batching server, at `load` times the server's own capacity
    (measured first with every request of a burst submitted at once);
    latency = submit to completion on the device."""
    import threading
    opts = _lib.ServerOptions(device, 32, 0, 0, 0)
    srv = L.sfft_server_create(ctypes.byref(opts))
    if not srv:
        return {"error": _lib.last_error()}
    ptrs = [ctypes.c_void_p(t.data_ptr()) for t in pool]
    lat = ctypes.c_double()
    # warm the plan and the allocator
    warm = [L.sfft_server_submit(srv, N_SIG, K_SIG, VERSION - 1, precision, ptrs[i % len(ptrs)], 0, i)
            for i in range(64)]
    for w in warm:
        L.sfft_server_wait(srv, w, None, None, 0, ctypes.byref(lat))
    burst = min(nreq, 2000)
    t0 = time.perf_counter()
    ids = [L.sfft_server_submit(srv, N_SIG, K_SIG, VERSION - 1, precision, ptrs[i % len(ptrs)], 0, 500 + i)
           for i in range(burst)]
    for rid in ids:
        L.sfft_server_wait(srv, rid, None, None, 0, ctypes.byref(lat))
    capacity = burst / (time.perf_counter() - t0)
    rate = load * capacity
    rng = np.random.default_rng(SEED)
    gaps = rng.exponential(1.0 / rate, size=nreq)
    ids = [None] * nreq
    lats = [0.0] * nreq
    done_t = [0.0]

    def waiter():
        ln = ctypes.c_double()
        for i in range(nreq):
            while ids[i] is None:
                time.sleep(0)
            L.sfft_server_wait(srv, ids[i], None, None, 0, ctypes.byref(ln))
            lats[i] = ln.value
        done_t[0] = time.perf_counter()

    th = threading.Thread(target=waiter)
    th.start()
    t0 = time.perf_counter()
    t_next = t0
    for i in range(nreq):
        t_next += gaps[i]
        while time.perf_counter() < t_next:
            pass
        ids[i] = L.sfft_server_submit(srv, N_SIG, K_SIG, VERSION - 1, precision, ptrs[i % len(ptrs)], 0,
                                      1000 + i)
    th.join()
    stats = (ctypes.c_long * 8)()
    L.sfft_server_stats(srv, stats, 8)
    L.sfft_server_destroy(srv)
    return {"offered_rate": rate, "capacity_burst_solves_per_s": capacity, "load": load, "requests": nreq,
            "solves_per_s": nreq / (done_t[0] - t0),
            "p50_ms": pct(lats, 50), "p99_ms": pct(lats, 99), "batches": int(stats[0]),
            "precision": "fp32" if precision == 1 else "fp64"}


def pct(xs, q):
    return float(np.percentile(np.asarray(xs), q)) if xs else None


def score_result(x, pos, vals, idx, val, conj, X=None):
    """Accuracy of one sparse result.  Against the dense FP64 FFT of the
    same (noisy) input, X = fft(x) / n -- the reference's inputs are
    unnormalised inverse DFTs (simulation.cc:95-112), so sFFT returns X --
    and against the drawn spectrum.  Support = the drawn tones; tau = half
    the smallest drawn magnitude; missed = a drawn tone whose estimate is
    below tau; spurious = an estimate >= tau off the drawn support; the
    per-entry L1 error |dRe| + |dIm| is taken on the recovered support
    (estimates >= tau).  v1/v2 return conjugates (conj=True)."""
    import torch
    dev = torch.device("cuda")
    xt = x.to(torch.complex128) if hasattr(x, "is_cuda") else torch.as_tensor(x).to(dev, torch.complex128)
    n = xt.numel()
    if X is None:
        X = torch.fft.fft(xt) / n
    E = torch.zeros(n, dtype=torch.complex128, device=dev)
    vv = torch.as_tensor(np.asarray(val)).to(dev, torch.complex128)
    E[torch.as_tensor(np.asarray(idx, dtype=np.int64), device=dev)] = vv.conj() if conj else vv
    T = torch.zeros(n, dtype=torch.complex128, device=dev)
    pd = torch.as_tensor(np.asarray(pos, dtype=np.int64), device=dev)
    T[pd] = torch.as_tensor(np.asarray(vals), device=dev)
    tau = 0.5 * float(np.min(np.abs(vals)))
    rec = E.abs() >= tau
    missed = int((~rec[pd]).sum())
    spurious = int(rec.sum()) - (len(pos) - missed)
    d = (E - X)[rec]
    l1 = d.real.abs() + d.imag.abs()
    dt = (E - T)[pd]
    return {"missed": missed, "spurious": spurious, "tau": tau, "entries": int(rec.sum()),
            "l1_sum": float(l1.sum()), "l1_max": float(l1.max()) if l1.numel() else 0.0,
            "truth_err_sum": float(dt.abs().sum()), "truth_err_max": float(dt.abs().max()), "tones": len(pos)}


def merge_scores(scores):
    """Totals over signals: missed / spurious counts (and per signal), mean
    and max L1 per recovered entry against the dense FFT, mean and worst
    error per drawn tone against the drawn spectrum."""
    ent = sum(s["entries"] for s in scores)
    tones = sum(s["tones"] for s in scores)
    return {"signals": len(scores), "missed": sum(s["missed"] for s in scores),
            "spurious": sum(s["spurious"] for s in scores),
            "missed_per_signal": [s["missed"] for s in scores][:16],
            "spurious_per_signal": [s["spurious"] for s in scores][:16],
            "vs_dense_fft": {"mean_l1": sum(s["l1_sum"] for s in scores) / max(ent, 1),
                             "max_l1": max((s["l1_max"] for s in scores), default=0.0), "entries": ent},
            "vs_drawn_spectrum": {"mean_abs_err": sum(s["truth_err_sum"] for s in scores) / max(tones, 1),
                                  "max_abs_err": max((s["truth_err_max"] for s in scores), default=0.0)},
            "tau": min((s["tau"] for s in scores), default=None),
            "definition": "dense oracle X = fft(x)/n in FP64 of the same noisy input; support = drawn tones; "
                          "tau = half the smallest drawn magnitude; L1 = |dRe|+|dIm| per entry >= tau"}


STAGES = ["comb", "fold", "bucket_fft_select_vote", "estimate"]


def stage_table(st):
    if not st or not st[1]:
        return None
    ms, cnt = st
    return {STAGES[i]: ms[i] / cnt for i in range(4)}


def algorithmic_bytes(plan_params, e_in, e_out, nnz):
    """Per-solve algorithmic bytes of the whole pipeline: every input sample
    the fold and comb read, plus the sparse output (index + value)."""
    p = plan_params
    sw = p["loops_loc"] * p["w_loc"] + p["loops_est"] * p["w_est"]
    return {"fold_in": e_in * sw, "comb_in": e_in * p["Comb_loops"] * p["W_Comb"],
            "xs_out": e_out * p["x_samp_size"], "out": (e_out + 4) * nnz}


def roofline(p32, st32, B):
    """Roofline of the dominant stage's kernel (live CUDA-event duration,
    algorithmic bytes per launch) and of the fold, the HBM-bound kernel."""
    from sfft_gb300.sfft import describe_plan
    peaks = {}
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as fh:
            peaks = json.load(fh)
    except OSError:
        pass
    peak = peaks.get("hbm_gbs", 6800.0)
    peak_src = "measured" if "hbm_gbs" in peaks else "fallback"
    pp = describe_plan(N_SIG, K_SIG, VERSION)
    nnz = min(pp["W_Comb"], pp["Comb_loops"] * pp["B_thresh"]) * (N_SIG // pp["W_Comb"])
    ab = algorithmic_bytes(pp, 16, 8, nnz)
    per = stage_table(st32) or {}
    traffic = {}
    try:
        with open(os.path.join(ROOT, "profiles", "dram_traffic.json")) as fh:
            traffic = json.load(fh)
    except (OSError, ValueError):
        pass
    # per-kernel algorithmic HBM bytes of one signal
    kernels = {
        "fold": ("k_fold_split<double2,4> (permuted-filter fold, FP32)", ab["fold_in"] + ab["xs_out"],
                 "k_fold_fp32_v2_n4194304_k100"),
        "estimate": ("k_estimate_comb32<20> (median estimation by comb residue)", ab["out"] + ab["xs_out"],
                     "k_estimate_comb32_v2_n4194304_k100"),
    }
    out = {}
    for stage, (name, bytes_sig, tkey) in kernels.items():
        ms = per.get(stage)
        ach = B * bytes_sig / (ms / 1e3) / 1e9 if ms else None
        tr = traffic.get(tkey, {}).get("bytes_per_signal")
        out[stage] = {"kernel": name, "bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s",
                      "frac": ach / peak if ach else None, "traffic": tr * B if tr else None,
                      "algorithmic_bytes_per_launch": B * bytes_sig, "launch_ms": ms,
                      "peak_source": f"{peak_src} hbm_gbs (copy bandwidth)"}
    out["fold"]["note"] = ("random 16-byte gathers touch most DRAM bursts of the 64 MB signal: DRAM moves "
                           "3.4x the algorithmic bytes (58.8 MB per signal, 8.7 us at the measured copy rate: "
                           "the floor; the kernel takes ~10 us)")
    out["estimate"]["note"] = ("bound by the ALU pipe, not HBM: the two lower-median selection networks "
                               "(FMNMX, 2 x 125 per candidate) keep it at 65% of peak in ncu "
                               "(profiles/k_estimate_comb32_*); every staged bucket byte is read once (58 MB of L2 "
                               "reads per signal); its HBM bytes are the sparse output")
    out["estimate"]["alu_pipe_pct_ncu"] = 65.1
    dominant = max(per, key=per.get) if per else "estimate"
    roof = dict(out.get(dominant, out["estimate"]))
    roof["stage"] = dominant
    roof["other_kernels"] = {k: v for k, v in out.items() if k != dominant}
    tot_ms = sum(per.values()) if per else None
    pipe_bytes = B * sum(ab.values())
    pipeline = {"algorithmic_bytes_per_solve": sum(ab.values()), "breakdown": ab,
                "achieved_gbs": pipe_bytes / (tot_ms / 1e3) / 1e9 if tot_ms else None,
                "frac": (pipe_bytes / (tot_ms / 1e3) / 1e9 / peak) if tot_ms else None}
    return roof, pipeline


def accuracy(p32, p64, signals, p32v=None, count=8):
    """C4 accuracy on `count` signals (seeds SEED..SEED+count-1): the FP32,
    FP64 and voted FP32 results of the same draws, each scored against the
    dense FP64 FFT of its input and against the drawn spectrum, plus FP32
    against FP64 entry by entry."""
    import torch
    from oracle import oracle as O
    res = {"fp32": [], "fp64": [], "fp32_voted": []}
    same_support, l1_32_64, voted_same = True, 0.0, True
    for i in range(count):
        x, pos, vals = signals.make_signal(N_SIG, K_SIG, SEED + i, mag=MAG, snr_db=SNR)
        X = torch.fft.fft(torch.as_tensor(x).cuda()) / N_SIG
        outs = {}
        for name, plan in (("fp32", p32), ("fp64", p64), ("fp32_voted", p32v)):
            if plan is None:
                continue
            O.seed_libc(SEED + i)
            ii, vv = plan.execute_sparse(x)
            o = np.argsort(ii)
            outs[name] = (ii[o], vv[o])
            res[name].append(score_result(x, pos, vals, ii[o], vv[o], True, X=X))
        (i32, v32), (i64, v64) = outs["fp32"], outs["fp64"]
        if np.array_equal(i32, i64):
            l1_32_64 = max(l1_32_64, float(np.max(np.abs(v32.real - v64.real) + np.abs(v32.imag - v64.imag))))
        else:
            same_support = False
        if "fp32_voted" in outs:
            tau = 0.5 * float(np.min(np.abs(vals)))
            iv, vv = outs["fp32_voted"]
            sv, s64 = np.sort(iv[np.abs(vv) >= tau]), np.sort(i64[np.abs(v64) >= tau])
            voted_same &= bool(np.array_equal(sv, s64))
    out = {name: merge_scores(v) for name, v in res.items() if v}
    out["fp32_vs_fp64"] = {"support_identical": same_support, "max_l1": l1_32_64 if same_support else None,
                           "bound": 1e-4, "signals": count}
    if p32v is not None:
        out["fp32_voted"]["recovered_support_identical_to_fp64"] = voted_same
    out["workload"] = (f"C4: {count} signals, seeds {SEED}..{SEED + count - 1}, the same glibc draws per signal "
                       "for every form")
    return out


def e2e_leg(L, p32, pool, B, a):
    """sfft_exec_many (the drop-in call) on page-locked host buffers."""
    import torch
    nb = N_SIG * 16
    host_in = [L.sfft_malloc(nb) for _ in range(B)]
    host_out = [L.sfft_malloc(nb) for _ in range(B)]
    for j in range(B):
        src = pool[j % len(pool)].cpu().numpy()
        ctypes.memmove(host_in[j], src.ctypes.data, nb)
    pin = (ctypes.c_void_p * B)(*host_in)
    pout = (ctypes.c_void_p * B)(*host_out)
    steps = max(3, a.steps // 4)
    for _ in range(2):
        L.sfft_exec_many(p32.sfft_plan, B, pin, pout)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(steps):
        L.sfft_exec_many(p32.sfft_plan, B, pin, pout)
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    err = _lib_err(L)
    for p in host_in + host_out:
        L.sfft_free(p)
    return {"value": B * steps / dt, "unit": "solves/s", "h2d_bytes_per_step": B * nb,
            "d2h_bytes_per_step": B * nb, "api": "sfft_exec_many, dense complex128 in/out, pinned host",
            "error": err or None}


def copy_bandwidth(nbytes=1 << 30, reps=5):
    """Host<->device copy bandwidth of page-locked memory on this machine
    (one 1 GiB cudaMemcpyAsync per direction, CUDA-event timed): the bound
    of the host-buffer (e2e) legs."""
    import torch
    h = torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)
    d = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    out = {}
    for name, dst, src in (("h2d_gbs", d, h), ("d2h_gbs", h, d)):
        dst.copy_(src, non_blocking=True)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            dst.copy_(src, non_blocking=True)
        e1.record()
        e1.synchronize()
        out[name] = reps * nbytes / (e0.elapsed_time(e1) / 1e3) / 1e9
    # both directions at once, on two streams (what the dense e2e leg needs)
    h2, d2 = torch.empty_like(h).pin_memory(), torch.empty_like(d)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(reps):
        with torch.cuda.stream(s1):
            d.copy_(h, non_blocking=True)
        with torch.cuda.stream(s2):
            h2.copy_(d2, non_blocking=True)
    torch.cuda.synchronize()
    out["bidirectional_total_gbs"] = 2 * reps * nbytes / (time.perf_counter() - t0) / 1e9
    del h, d, h2, d2
    torch.cuda.empty_cache()
    return out


def e2e_sparse_leg(L, p32, pool, B, a):
    """sfft_exec_many_sparse on page-locked host buffers: host signals in,
    host (index, value) arrays out -- the same transforms as the dense
    drop-in call without the n-point outputs."""
    import torch
    nb = N_SIG * 16
    cap = L.sfft_output_capacity(p32.sfft_plan)
    host_in = [L.sfft_malloc(nb) for _ in range(B)]
    for j in range(B):
        src = pool[j % len(pool)].cpu().numpy()
        ctypes.memmove(host_in[j], src.ctypes.data, nb)
    hidx = L.sfft_malloc(4 * cap * B)
    hval = L.sfft_malloc(8 * cap * B)          # complex64 values of the FP32 form
    hcnt = np.zeros(B, dtype=np.int32)
    pin = (ctypes.c_void_p * B)(*host_in)

    def run():
        if L.sfft_exec_many_sparse(p32.sfft_plan, B, pin, ctypes.c_void_p(hidx), ctypes.c_void_p(hval),
                                   ctypes.c_void_p(hcnt.ctypes.data), cap) != 0:
            raise RuntimeError(_lib_err(L))
    steps = max(3, a.steps // 4)
    for _ in range(2):
        run()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(steps):
        run()
    torch.cuda.synchronize()
    dt = time.perf_counter() - t0
    d2h = int(hcnt.sum()) * 12
    for p in host_in + [hidx, hval]:
        L.sfft_free(p)
    return {"value": B * steps / dt, "unit": "solves/s", "h2d_bytes_per_step": B * nb, "d2h_bytes_per_step": d2h,
            "h2d_gbs_achieved": B * nb * steps / dt / 1e9, "copy_bandwidth": copy_bandwidth(),
            "api": "sfft_exec_many_sparse, complex128 host inputs, host (int32 index, complex64 value) outputs, "
                   "pinned host"}


def _lib_err(L):
    return L.sfft_last_error().decode()


def main():
    a = args_()
    ws, rank, local = dist_init()
    if a.impl == "reference":
        reference_arm(a, ws, rank)
    else:
        gb300_arm(a, ws, rank, local)
    if ws > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
