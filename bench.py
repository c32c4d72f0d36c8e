#!/usr/bin/env python3
"""Benchmark: target evaluations per second of the vortex-blob treecode.

Workload (default): 4,194,304 blobs -- two Gaussian patches (45% + 45%,
std 0.05, centres (0.4,0.5)/(0.6,0.5), Gamma = |N(0,1)|) and a perturbed
shear sheet (10%, y = 0.2 + 0.01 sin(8 pi x), Gamma = -1/N_sheet), stored
FP32, sigma 0.001, p = 12 (nterms 13), theta 0.5, at most 64 blobs per leaf;
every blob is a target.  Inputs are seeded synthetic data (there is no
public dataset for this path).

A step is one whole solve: tree build, upward pass and evaluation at all
targets.  `value` times the device-resident call (inputs already in HBM,
CUDA events on the launching stream, L2 flushed between steps); `e2e`
times the reference-facing calls with host buffers (make_tree + one batch
of biot_tree answers), copies included.  `cpu_baseline` times the
reference's own CPU code (ver-c/src built on the host from the staged
sources; the oracle, its restatement in C, where that build is absent) on
the host cores on a bounded sample.  `--impl reference` times that CPU
implementation alone.

Run:  python bench.py [--gpus N --steps K --warmup W] [--impl reference]
"""
from __future__ import annotations

import argparse
import importlib
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

METRIC = "target evals/s at 4M blobs (two patches + sheet), all blobs as targets, relL2 <= 1e-6 vs FP64 direct"
UNIT = "targets/s"
MODES = {"plain": 0, "mixed": 1, "learned": 2}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--mode", default="learned", choices=list(MODES))
    ap.add_argument("--weights", default=None, help="learned form: weights file (default: the packaged ones)")
    ap.add_argument("--direct-bias", type=float, default=1.0, help="learned form: logit bias towards direct evaluation")
    ap.add_argument("--order-margin", type=int, default=1, help="learned form: orders added to the network's choice")
    ap.add_argument("--far-orders", action="store_true",
                    help="learned form: the network also sets each W-list M2P's order")
    ap.add_argument("--pterms", type=int, default=16, help="mixed form: expansion length")
    ap.add_argument("--cutoff", type=float, default=2.5, help="mixed form: correction radius / max sigma")
    ap.add_argument("--cuda-core-m2l", action="store_true", help="mixed form: M2L on CUDA cores")
    ap.add_argument("--no-plain", action="store_true", help="skip timing the plain FP64 path beside")
    ap.add_argument("--eval-variant", type=int, default=-1,
                    help="mixed/learned: force a near-field kernel variant 0..4 (default: the tuner's choice)")
    ap.add_argument("--level-chain", action="store_true",
                    help="mixed/learned: one cooperative launch per M2M / L2L chain instead of one launch per level")
    ap.add_argument("--workload", default="two_patch_sheet",
                    choices=["two_patch_sheet", "lamb_oseen", "uniform", "batch_sets", "advected"])
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the compact measurements of the other configurations in the default line")
    ap.add_argument("--nsets", type=int, default=512, help="batch_sets: number of independent sets")
    ap.add_argument("--set-targets", type=int, default=4096, help="batch_sets: targets per set measured against the direct sum")
    ap.add_argument("--n", type=int, default=0, help="override the blob count (exploration only)")
    ap.add_argument("--leaf-blobs", type=int, default=-1,
                    help="mixed/learned: most blobs per leaf (-1: by set size, 0: the configuration's num_p - 1)")
    ap.add_argument("--err-targets", type=int, default=65536)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-sample", type=int, default=0, help="targets per CPU step (0: auto)")
    return ap.parse_args()


def workload(args, rank=0):
    W = importlib.import_module("2dfmm_gb300.workloads")
    if args.workload == "two_patch_sheet":
        kw = {"n": args.n} if args.n else {}
        return W.two_patch_sheet(seed=3 + rank, **kw), "two_patch_sheet_4M" if not args.n else f"two_patch_sheet_{args.n}"
    if args.workload == "lamb_oseen":
        kw = {"n": args.n} if args.n else {}
        return W.lamb_oseen(seed=2 + rank, **kw), "lamb_oseen_1M" if not args.n else f"lamb_oseen_{args.n}"
    kw = {"n": args.n} if args.n else {}
    return W.uniform(seed=1 + rank, **kw), "uniform_20k" if not args.n else f"uniform_{args.n}"


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def max_over_ranks(x, world, device="cpu"):
    """The largest of a per-rank time over all ranks (the job ends with the
    slowest replica); identity on one rank."""
    if world <= 1:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(n_per_rank, steps, total_ms, world):
    """Whole-job targets/s of `world` replicas that each solve `steps` sets of
    `n_per_rank` blobs (every blob a target) in at most `total_ms`."""
    return world * n_per_rank * steps / (total_ms * 1e-3)


# --------------------------------------------------------------------------
# clocks during the timed region

class Clocks:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.path = tempfile.mktemp(suffix=".csv")
        self.proc = None
        self.gpu = gpu_index

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        rows = []
        try:
            for line in open(self.path):
                f = [x.strip() for x in line.split(",")]
                if len(f) >= 9 and f[1].replace(".", "").isdigit():
                    rows.append(f)
        except OSError:
            pass
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"], "samples": 0}
        sm = [float(r[1]) for r in rows]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": float(rows[0][2]), "reasons": reasons,
                "samples": len(rows), "power_w_max": max(float(r[3]) for r in rows if r[3] not in ("[N/A]", ""))}


# --------------------------------------------------------------------------
# CPU baseline: the reference's own code (or the oracle, its restatement)

def mem_available_gb():
    try:
        for line in open("/proc/meminfo"):
            if line.startswith("MemAvailable:"):
                return int(line.split()[1]) / 1e6
    except OSError:
        pass
    return 0.0


def cpu_reference(b, depth_hint, steps, warmup, sample, threads=0):
    """Times the reference's CPU implementation of the path on `b`: its own
    build (ver-c/src compiled from the staged sources by oracle/Makefile,
    `kind: reference`) where it runs here, else the oracle (the reference's
    algorithm restated in C, `kind: port`).  make_tree runs once,
    single-threaded as in the reference, then `warmup + steps` batches of
    `sample` sampled targets over all host threads (biot_tree is re-entrant,
    as the reference caller's MPI target split uses it).  Returns (targets/s
    projected to the whole job, detail)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O  # noqa: WPS433
    W = importlib.import_module("2dfmm_gb300.workloads")
    use_ref = O.reference_available()
    threads = threads or O.max_threads()
    # the reference's dense complete tree: (4^(L+1)-1)/3 nodes of 64 B (56 in
    # the port), plus one num_nodes-int traversal stack per concurrent call
    nodes = (4 ** (depth_hint + 1) - 1) // 3
    need_gb = nodes * (64 if use_ref else 56) / 1e9 + 1.2 * b.n * 64 / 1e9
    per_thread_gb = nodes * 4 / 1e9
    avail = mem_available_gb()
    if avail and need_gb + per_thread_gb > 0.7 * avail:
        return None, {"unavailable": f"dense reference tree needs {need_gb:.1f} GB, {avail:.1f} GB available"}
    if avail:
        threads = max(1, min(threads, int((0.7 * avail - need_gb) / max(per_thread_gb, 1e-9))))
    if not sample:
        # about 2 s per batch: each call allocates and fills its num_nodes
        # stack (~0.5 ns per node) before a traversal of ~0.2 ms
        est = 0.5e-9 * nodes + 2e-4
        sample = int(min(200_000, b.n, max(1, round(2.0 / est)) * threads))
    idx = W.sample_targets(b.n, sample, seed=100)
    if use_ref:
        with tempfile.TemporaryDirectory() as d:
            t_make, per, levels = O.time_reference(d, b.xy, b.cir, b.cor, b.xy[idx], b.nterms, b.num_p, b.theta,
                                                   threads=threads, batches=warmup + steps)
        times = per[warmup:] or per
        kind = "reference"
        what = "the reference's own ver-c/src (gcc -O2, built on this host from the staged sources)"
    else:
        o = O.Oracle(b.nterms, b.num_p, b.theta)
        t0 = time.perf_counter()
        o.make_tree(b.xy, b.cir, b.cor, max_level_cap=30)
        t_make = time.perf_counter() - t0
        times = []
        for k in range(warmup + steps):
            t0 = time.perf_counter()
            o.biot(b.xy[idx], threads=threads)
            if k >= warmup:
                times.append(time.perf_counter() - t0)
        levels = o.levels()
        o.close()
        kind = "port"
        what = "the oracle (the reference's algorithm restated in C, oracle/tree2d_oracle.c)"
    per_target = statistics.median(times) / sample
    value = b.n / (t_make + b.n * per_target)
    detail = {"make_tree_s": round(t_make, 3), "biot_tree_s_per_target_per_job": per_target,
              "batch_s_median": statistics.median(times),
              "sample": f"{what}: make_tree over all {b.n} blobs (1 thread, as the reference), then {len(times)} "
                        f"timed batches of {sample} sampled targets over {threads} threads (after {warmup} "
                        f"untimed); value = N / (t_make + N * t_target)",
              "cores": threads, "levels": levels, "kind": kind}
    return value, detail


# --------------------------------------------------------------------------

def roofline_traffic():
    """DRAM bytes per launch of each mode's dominant kernel, from the
    committed ncu summary (profiles/dram_traffic.txt)."""
    out = {}
    try:
        with open(os.path.join(ROOT, "profiles", "dram_traffic.txt")) as f:
            for line in f:
                if line.strip() and not line.startswith("#"):
                    parts = line.split()
                    out[parts[0]] = int(parts[1])
    except (OSError, ValueError, IndexError):
        pass
    return out


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    b, wname = workload(args)
    depth_hint = {"two_patch_sheet": 14, "lamb_oseen": 10, "uniform": 6}[args.workload]
    value, det = cpu_reference(b, depth_hint, args.steps, args.warmup, args.cpu_sample)
    line = {"metric": METRIC, "impl": "reference", "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "higher_is_better": True, "dtype": "f64", "data": "synthetic (seeded)",
            "config": {"workload": wname, "n_blobs": b.n, "nterms": b.nterms, "num_p": b.num_p, "theta": b.theta}}
    if value is None:
        line.update({"value": None, "unavailable": det["unavailable"]})
    else:
        # a step is one timed batch of sampled targets (ms_per_step is its
        # measured time); value is the whole job's projected rate
        line.update({"value": value, "ms_per_step": 1e3 * det["batch_s_median"],
                     "cpu_baseline": {"value": value, "unit": UNIT, "cores": det["cores"], "kind": det["kind"],
                                      "sample": det["sample"]},
                     "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                     "detail": det})
    print(json.dumps(line), flush=True)


def _time_mode(P, torch, args, mode, arrays, stream, flush, clk=None):
    """Warm-up, then `steps` timed solves (CUDA events on the launch stream,
    L2 flushed between steps).  Returns (per-step ms, per-step stats)."""
    xy, cir, cor, uv, n = arrays
    P.set_mode(MODES[mode])
    sp = stream.cuda_stream

    def solve():
        P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), n, sp)

    for _ in range(args.warmup):
        solve()
    torch.cuda.synchronize()
    times, sts = [], []
    for _ in range(args.steps):
        flush.fill_(1)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(stream)
        solve()
        e1.record(stream)
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
        sts.append(P.stats())
    return times, sts


def _direct_reference(P, torch, arrays, n, ntgt, sp):
    """FP64 direct sum (the accuracy yardstick) at `ntgt` seeded targets sampled without
    replacement from the blobs; computed once per run and reused for every
    form measured."""
    xy, cir, cor, _, _ = arrays
    W = importlib.import_module("2dfmm_gb300.workloads")
    idx = W.sample_targets(n, ntgt, seed=7)
    tidx = torch.from_numpy(idx).to(xy.device)
    txy = xy[tidx].contiguous()
    ref = torch.empty_like(txy)
    P.direct_device(txy.data_ptr(), len(idx), xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), n, ref.data_ptr(), sp)
    torch.cuda.synchronize()
    return tidx, ref


def _accuracy(uv, yardstick):
    """relL2 and max relative error of the last solve's velocities against
    the FP64 direct sum."""
    tidx, ref = yardstick
    got = uv[tidx]
    rel_l2 = float((got - ref).norm() / ref.norm())
    max_rel = float(((got - ref).norm(dim=1) / ref.norm(dim=1).clamp_min(1e-300)).max())
    return {"relL2_vs_fp64_direct": rel_l2, "max_rel_vs_fp64_direct": max_rel, "targets": int(len(tidx))}


def _roofline(P, args, mode, b, wname, sts, sp):
    p = b.nterms - 1
    st = sts[-1]
    ms = statistics.mean(s["ms_eval"] for s in sts)
    tr = roofline_traffic().get(f"{mode}:{wname}")
    if mode == "plain" and b.theta <= 0.7:
        # 64-bit fixed point: the integer pipes' dispatch bounds it, for which
        # there is no probe; the rate is that of the FP64 method
        flops = st["n_m2s"] * (8 * p + 10) + st["n_pairs"] * 20
        return {"bound": "integer dispatch", "achieved": flops / (ms * 1e-3) / 1e12, "peak": None,
                "unit": "TFLOP/s (operations of the method in FP64)", "frac": None, "traffic": tr,
                "kernel": "k_eval (traversal + M2S + P2P, in 64-bit fixed point)", "peak_source": None,
                "algorithmic_flops_per_launch": flops, "ms_per_launch": ms}
    if mode == "plain":
        # larger opening angles: the multipole sums, and only they, in FP64
        flops = st["n_m2s"] * (8 * p + 10)
        peak = P.fp64_peak_tflops(stream=sp)
        return {"bound": "fp64", "achieved": flops / (ms * 1e-3) / 1e12, "peak": peak, "unit": "TFLOP/s",
                "frac": flops / (ms * 1e-3) / 1e12 / peak, "traffic": tr,
                "kernel": "k_eval (traversal + M2S in FP64 + P2P in 64-bit fixed point)",
                "peak_source": "measured: the library's DFMA probe (8 independent chains per thread)",
                "algorithmic_flops_per_launch": flops, "ms_per_launch": ms}
    # mixed and learned: the evaluation kernel (direct pairs, correction
    # pairs, L2P, M2P)
    flops = st["n_pairs"] * 20 + b.n * 8 * args.pterms
    peak = P.fp32_peak_tflops(stream=sp)
    return {"bound": "fp32", "achieved": flops / (ms * 1e-3) / 1e12, "peak": peak, "unit": "TFLOP/s",
            "frac": flops / (ms * 1e-3) / 1e12 / peak, "traffic": tr,
            "kernel": "k_eval_near (P2P + correction pairs + L2P/M2P, FP32)",
            "peak_source": "measured: the library's FFMA probe (8 independent chains per thread)",
            "algorithmic_flops_per_launch": flops, "ms_per_launch": ms}


def run_ours(args):
    import torch
    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    P = importlib.import_module("2dfmm_gb300")
    P.load()
    b, wname = workload(args, rank)
    P.set_params(b.nterms, b.num_p, b.theta)
    P.set_mixed_params(args.pterms, args.cutoff, not args.cuda_core_m2l)
    P.set_mixed_leaf(args.leaf_blobs)
    P.set_tuning(args.eval_variant < 0, args.eval_variant)
    P.set_level_chain(args.level_chain)
    learned_note = None
    if args.mode == "learned":
        L = importlib.import_module("2dfmm_gb300.learn")
        path = args.weights or L.DEFAULT_WEIGHTS
        theta = L.load_weights(path)
        if theta is None:
            learned_note = f"none found at {os.path.relpath(path, ROOT)}: fixed mixed form (the fallback)"
        else:
            P.learn_set_weights(theta)
            P.learn_set_options(args.direct_bias, args.order_margin)
            P.learn_set_far_orders(args.far_orders)
            envelope, env_cutoff = L.load_envelope(path)
            P.learn_set_envelope(envelope, env_cutoff)
            learned_note = (f"{os.path.relpath(path, ROOT)} (trained on configuration-5 steps 0-20 by "
                            f"2dfmm_gb300/learn.py); decisions applied up to {envelope:.1f} K-list source blobs "
                            f"per leaf counted at {env_cutoff:g} max sigma")
    n = b.n
    xy = torch.from_numpy(b.xy).to(dev).contiguous()
    cir = torch.from_numpy(b.cir).to(dev)
    cor = torch.from_numpy(b.cor).to(dev)
    uv = torch.empty((n, 2), dtype=torch.float64, device=dev)
    arrays = (xy, cir, cor, uv, n)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)  # > 129 MB L2
    stream = torch.cuda.current_stream()
    sp = stream.cuda_stream

    if world > 1:
        torch.distributed.barrier()
    with Clocks(local) as clk:
        times, sts = _time_mode(P, torch, args, args.mode, arrays, stream, flush)
    clocks = clk.summary()
    total_ms = max_over_ranks(float(sum(times)), world, dev)
    value = replica_throughput(n, args.steps, total_ms, world)
    yardstick = _direct_reference(P, torch, arrays, n, args.err_targets, sp)
    accuracy = _accuracy(uv, yardstick)
    roofline = _roofline(P, args, args.mode, b, wname, sts, sp)

    # the fixed mixed form and the plain FP64 path on the same set, timed the
    # same way, for the ratios
    beside = {}
    others = [] if args.no_plain else ["plain"]
    if args.mode == "learned":
        others.insert(0, "mixed")
    for other in others:
        otimes, _ = _time_mode(P, torch, args, other, arrays, stream, flush)
        o = {"value": n / (statistics.mean(otimes) * 1e-3), "unit": UNIT, "ms_per_step": statistics.mean(otimes),
             "accuracy": _accuracy(uv, yardstick)}
        o["speedup_of_headline"] = value / world / o["value"]
        beside["plain_fp64" if other == "plain" else "mixed_fixed"] = o
    P.set_mode(MODES[args.mode])

    # end to end through the reference-facing calls, host buffers
    P.set_mode(MODES[args.mode])
    h_xy = torch.empty((n, 2), dtype=torch.float64, pin_memory=True)
    h_cir = torch.empty(n, dtype=torch.float64, pin_memory=True)
    h_cor = torch.empty(n, dtype=torch.float64, pin_memory=True)
    h_xy.numpy()[:] = b.xy
    h_cir.numpy()[:] = b.cir
    h_cor.numpy()[:] = b.cor
    h_uv = torch.empty((n, 2), dtype=torch.float64, pin_memory=True)
    P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), n, sp)
    torch.cuda.synchronize()
    e2e_times = []
    e2e_steps = max(1, min(args.steps, 3))
    e2e_split = []
    for k in range(1 + e2e_steps):
        t0 = time.perf_counter()
        P.make_tree(h_xy.numpy(), h_cir.numpy(), h_cor.numpy())
        t1 = time.perf_counter()
        out = P.biot_tree_batch(h_xy.numpy(), out=h_uv.numpy())
        dt = time.perf_counter() - t0
        if k >= 1:
            e2e_times.append(dt)
            e2e_split.append((1e3 * (t1 - t0), 1e3 * (t0 + dt - t1)))
    e2e_t = max_over_ranks(statistics.mean(e2e_times), world, dev)
    e2e_match = bool(np.array_equal(out, uv.cpu().numpy()))

    extras = None
    if rank == 0 and world == 1 and not args.no_extras and args.workload == "two_patch_sheet" and not args.n:
        t0 = time.perf_counter()
        extras = other_configurations(P, torch, stream, flush)
        extras["wall_s"] = round(time.perf_counter() - t0, 1)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        depth = sts[-1]["depth"]
        v, det = cpu_reference(b, depth, 1, 0, args.cpu_sample)
        if v is None:
            cpu = {"value": None, "unit": UNIT, "cores": 0, "kind": "reference", "sample": det["unavailable"]}
        else:
            cpu = {"value": v, "unit": UNIT, "cores": det["cores"], "kind": det["kind"], "sample": det["sample"],
                   "make_tree_s": det["make_tree_s"]}

    if rank == 0:
        st = sts[-1]
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None,
            "dtype": "f64" if args.mode == "plain" else "f32 (tf32x3 tensor M2L, bf16 MLP, f64 final sum)",
            "data": "synthetic (seeded numpy PCG64), shapes and distributions of the configuration",
            "config": {"workload": wname, "n_blobs": n, "targets": "all blobs", "nterms": b.nterms,
                       "p": b.nterms - 1, "num_p": b.num_p, "theta": b.theta, "mode": args.mode,
                       "mixed_pterms": args.pterms, "cutoff_sigmas": args.cutoff,
                       "leaf_blobs": int(st["leaf_blobs"]),
                       "parallelism": f"replicas x{world} (independent blob sets, no collective)",
                       "l2": "flushed between steps (256 MiB write); inputs 134 MB > L2"},
            "gpu_launches": int(sum(s["n_launches"] for s in sts)),
            "tuned": {"eval_variant": int(st["eval_variant"]), "m2l_rows": int(st["m2l_rows"]),
                      "variants": "0/1 global loads, 2/3/4 bulk-copy staging; 4/8/4 warps per block (4: 80 registers, unroll 4); M2L 128 or 64 cells per CTA"},
            "learned_active": bool(st["learned_active"]),
            "k_list_per_leaf": st["n_list_k"] / max(1, st["n_leaves"]),
            "k_list_blobs_per_leaf": st["n_list_k_blobs"] / max(1, st["n_leaves"]),
            "e2e": {"value": world * n / e2e_t, "unit": UNIT, "h2d_bytes_per_step": n * 48,
                    "d2h_bytes_per_step": n * 16,
                    "api": "make_tree + biot_tree_batch (host buffers; the blobs go up in make_tree, "
                           "the query points in biot_tree_batch)",
                    "make_tree_ms": statistics.mean(a for a, _ in e2e_split),
                    "biot_tree_batch_ms": statistics.mean(b_ for _, b_ in e2e_split),
                    "matches_device_path": e2e_match},
            "roofline": roofline,
            "accuracy": accuracy,
            "stages_ms": {"build": statistics.mean(s["ms_build"] for s in sts),
                          "upward": statistics.mean(s["ms_upward"] for s in sts),
                          "eval": statistics.mean(s["ms_eval"] for s in sts)},
            "tree": {"cells": st["n_cells"], "leaves": st["n_leaves"], "depth": st["depth"],
                     "m2s_per_target": st["n_m2s"] / n, "pairs_per_target": st["n_pairs"] / n,
                     "m2l_pairs": st["n_m2l"]},
            "pairs_per_target": {"direct_u": (st["n_pairs"] - st["n_pairs_k"]) / n,
                                 "correction_k": st["n_pairs_k"] / n,
                                 "correction_k_listed": st["n_pairs_k_listed"] / n,
                                 "note": "correction pairs of the K leaves evaluated, after and before skipping "
                                         "16-blob chunks farther than the correction radius from the targets"},
            "clocks": clocks,
        }
        line.update(beside)
        if extras is not None:
            line["other_configurations"] = extras
        if learned_note:
            line["config"]["learned_weights"] = learned_note
        if cpu is not None:
            line["cpu_baseline"] = cpu
        print(json.dumps(line), flush=True)
    if world > 1:
        torch.distributed.destroy_process_group()


BATCH_METRIC = "target evals/s over 512 uneven blob sets solved as one batch, relL2 <= 1e-6 per set vs FP64 direct"


def run_batch(args):
    """Configuration 4: `nsets` independent sets (sizes log-uniform in
    [2,048, 200,000]) solved by one batched mixed solve per step
    (tree2d_solve_sets); every blob is a target.  Each set is measured against
    its own FP64 direct sum on `set_targets` sampled targets.  Beside it the
    same sets solved one call at a time."""
    import torch
    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    P = importlib.import_module("2dfmm_gb300")
    W = importlib.import_module("2dfmm_gb300.workloads")
    P.load()
    sets = W.batch_sets(nsets=args.nsets, seed=4 + rank)
    b0 = sets[0]
    P.set_params(b0.nterms, b0.num_p, b0.theta)
    P.set_mixed_leaf(args.leaf_blobs)
    P.set_mode(MODES["mixed"])
    P.set_mixed_params(args.pterms, args.cutoff, not args.cuda_core_m2l)
    P.set_tuning(args.eval_variant < 0, args.eval_variant)
    P.set_level_chain(args.level_chain)
    off = np.concatenate([[0], np.cumsum([b.n for b in sets])]).astype(np.int32)
    n = int(off[-1])
    h_xy = np.concatenate([b.xy for b in sets])
    h_cir = np.concatenate([b.cir for b in sets])
    h_cor = np.concatenate([b.cor for b in sets])
    xy = torch.from_numpy(h_xy).to(dev).contiguous()
    cir = torch.from_numpy(h_cir).to(dev)
    cor = torch.from_numpy(h_cor).to(dev)
    uv = torch.empty_like(xy)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream()
    sp = stream.cuda_stream

    def solve():
        P.solve_sets(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), off, sp)

    for _ in range(args.warmup):
        solve()
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    times, sts = [], []
    with Clocks(local) as clk:
        for _ in range(args.steps):
            flush.fill_(1)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record(stream)
            solve()
            e1.record(stream)
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
            sts.append(P.stats())
    total_ms = max_over_ranks(float(sum(times)), world, dev)
    value = replica_throughput(n, args.steps, total_ms, world)

    # per-set accuracy against the FP64 direct sum
    rels, maxrels = [], []
    uv_h = uv.cpu().numpy()
    for k, b in enumerate(sets):
        idx = W.sample_targets(b.n, args.set_targets, seed=1000 + k)
        s_xy = xy[int(off[k]):int(off[k + 1])]
        txy = s_xy[torch.from_numpy(idx).to(dev)].contiguous()
        ref = torch.empty_like(txy)
        P.direct_device(txy.data_ptr(), len(idx), s_xy.data_ptr(), cir[int(off[k]):].data_ptr(),
                        cor[int(off[k]):].data_ptr(), b.n, ref.data_ptr(), sp)
        torch.cuda.synchronize()
        ref = ref.cpu().numpy()
        got = uv_h[int(off[k]):int(off[k + 1])][idx]
        rels.append(float(np.linalg.norm(got - ref) / np.linalg.norm(ref)))
        maxrels.append(float((np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)).max()))

    # the same sets one call at a time (one pass after one warm-up pass)
    dev_sets = [(xy[int(off[k]):int(off[k + 1])], cir[int(off[k]):int(off[k + 1])],
                 cor[int(off[k]):int(off[k + 1])], uv[int(off[k]):int(off[k + 1])]) for k in range(len(sets))]
    seq_ms = None
    for rep in range(2):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for (a, c, r, u), b in zip(dev_sets, sets):
            P.solve_device(a.data_ptr(), c.data_ptr(), r.data_ptr(), u.data_ptr(), b.n, sp)
        torch.cuda.synchronize()
        seq_ms = 1e3 * (time.perf_counter() - t0)

    # end to end: pinned host buffers in, velocities out, every step
    hp_xy = torch.from_numpy(h_xy).pin_memory()
    hp_cir = torch.from_numpy(h_cir).pin_memory()
    hp_cor = torch.from_numpy(h_cor).pin_memory()
    hp_uv = torch.empty_like(hp_xy).pin_memory()
    e2e = []
    for k in range(1 + max(1, min(args.steps, 3))):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        xy.copy_(hp_xy, non_blocking=True)
        cir.copy_(hp_cir, non_blocking=True)
        cor.copy_(hp_cor, non_blocking=True)
        solve()
        hp_uv.copy_(uv, non_blocking=True)
        torch.cuda.synchronize()
        if k:
            e2e.append(time.perf_counter() - t0)
    e2e_t = max_over_ranks(statistics.mean(e2e), world, dev)

    if rank == 0:
        st = sts[-1]
        flops = st["n_pairs"] * 20 + n * 8 * args.pterms
        ms_eval = statistics.mean(x["ms_eval"] for x in sts)
        peak = P.fp32_peak_tflops(stream=sp)
        line = {
            "metric": BATCH_METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32 (tf32x3 tensor M2L, f64 final sum)",
            "data": "synthetic (seeded numpy PCG64), shapes and distributions of the configuration",
            "config": {"workload": f"batch_sets_{len(sets)}", "n_sets": len(sets), "n_blobs": n,
                       "set_sizes": [int(b.n) for b in sets][:4] + ["..."], "nterms": b0.nterms, "p": b0.nterms - 1,
                       "num_p": b0.num_p, "theta": b0.theta, "mode": "mixed (batched: one tree over all sets)",
                       "mixed_pterms": args.pterms, "cutoff_sigmas": args.cutoff,
                       "leaf_blobs": int(st["leaf_blobs"]),
                       "parallelism": f"replicas x{world} (independent batches, no collective)",
                       "l2": "flushed between steps (256 MiB write)"},
            "gpu_launches": int(sum(x["n_launches"] for x in sts)),
            "tuned": {"eval_variant": int(st["eval_variant"]), "m2l_rows": int(st["m2l_rows"]),
                      "variants": "0/1 global loads, 2/3/4 bulk-copy staging; 4/8/4 warps per block (4: 80 registers, unroll 4); M2L 128 or 64 cells per CTA"},
            "e2e": {"value": world * n / e2e_t, "unit": UNIT, "h2d_bytes_per_step": n * 32,
                    "d2h_bytes_per_step": n * 16, "api": "host->device copies + tree2d_solve_sets + device->host"},
            "roofline": {"bound": "fp32", "achieved": flops / (ms_eval * 1e-3) / 1e12, "peak": peak,
                         "unit": "TFLOP/s", "frac": flops / (ms_eval * 1e-3) / 1e12 / peak, "traffic": None,
                         "kernel": "k_eval_near (P2P + correction pairs + L2P/M2P, FP32)",
                         "peak_source": "measured: the library's FFMA probe"},
            "accuracy": {"sets": len(sets), "targets_per_set": args.set_targets,
                         "relL2_max_over_sets": max(rels), "relL2_median": float(np.median(rels)),
                         "max_rel_max_over_sets": max(maxrels), "sets_above_1e-6": int(sum(r > 1e-6 for r in rels))},
            "stages_ms": {"build": statistics.mean(x["ms_build"] for x in sts),
                          "upward": statistics.mean(x["ms_upward"] for x in sts), "eval": ms_eval},
            "tree": {"cells": st["n_cells"], "leaves": st["n_leaves"], "depth": st["depth"]},
            "one_call_per_set": {"ms_per_pass": seq_ms, "value": n / (seq_ms * 1e-3),
                                 "batched_speedup": seq_ms / (total_ms / args.steps)},
            "clocks": clk.summary(),
            "cpu_baseline": None,
        }
        print(json.dumps(line), flush=True)


# --------------------------------------------------------------------------
# the other configurations, compactly (appended to the default line)

def _events_ms(torch, stream, fn, steps, flush=None):
    """Per-step CUDA-event times of fn() on `stream` (L2 flushed first)."""
    out = []
    for _ in range(steps):
        if flush is not None:
            flush.fill_(1)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(stream)
        fn()
        e1.record(stream)
        torch.cuda.synchronize()
        out.append(e0.elapsed_time(e1))
    return out


def _dev(torch, b, dev):
    xy = torch.from_numpy(np.ascontiguousarray(b.xy)).to(dev)
    return xy, torch.from_numpy(b.cir).to(dev), torch.from_numpy(b.cor).to(dev), torch.empty_like(xy)


def _rel_l2_at(P, torch, xy, cir, cor, n, uvs, idx, sp):
    t = torch.from_numpy(idx).to(xy.device)
    txy = xy[t].contiguous()
    ref = torch.empty_like(txy)
    P.direct_device(txy.data_ptr(), len(idx), xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), n, ref.data_ptr(), sp)
    torch.cuda.synchronize()
    return [float(torch.linalg.norm(u[t] - ref) / torch.linalg.norm(ref)) for u in uvs]


def _use_learned(P, L, mode):
    if mode == "learned":
        P.learn_load(L.DEFAULT_RAW_WEIGHTS)
        P.learn_set_options(1.0, 1)


def advected(P, torch, stream, steps_total=100, train_until=20, dt=1e-3, score_every=10, score_targets=2048,
             n=1_048_576):
    """Configuration 5: the configuration-2 set (1M Lamb-Oseen blobs)
    advected 100 forward-Euler steps (dt 1e-3) on the device by its own
    velocity (the fixed mixed form's, P = 16), the tree rebuilt every step.
    The packaged network was trained on steps 0-20; on steps 21-100 every
    form solves the same state: learned, the fixed-order FMM at p = 12 and
    at P = 16, and the plain FP64 treecode (every `score_every` steps).
    relL2 against the FP64 direct sum on sampled targets every
    `score_every` steps."""
    W = importlib.import_module("2dfmm_gb300.workloads")
    L = importlib.import_module("2dfmm_gb300.learn")
    dev = torch.device("cuda", torch.cuda.current_device())
    sp = stream.cuda_stream
    b = W.lamb_oseen(n, seed=2)
    P.set_params(b.nterms, b.num_p, b.theta)
    P.set_mixed_leaf(-1)
    _use_learned(P, L, "learned")
    xy, cir, cor, uv = _dev(torch, b, dev)
    uvs = {k: torch.empty_like(xy) for k in ("learned", "p12", "p16", "plain")}
    forms = {"learned": (P.MODE_LEARNED, 16), "p12": (P.MODE_MIXED, 12), "p16": (P.MODE_MIXED, 16),
             "plain": (P.MODE_PLAIN, 16)}
    times = {k: [] for k in forms}
    rels = {k: [] for k in forms}
    pairs = {"learned": [], "p16": []}
    learned_active = []

    def solve(kind):
        mode, pt = forms[kind]
        P.set_mode(mode)
        P.set_mixed_params(pt, 2.5, True)
        out = uvs[kind]
        return _events_ms(torch, stream, lambda: P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(),
                                                                out.data_ptr(), n, sp), 1)[0]

    for k in ("learned", "p12", "p16"):  # warm-up: tuner and buffers of each form
        solve(k)
    for step in range(steps_total + 1):
        scored = step > train_until
        if scored:
            for k in ("learned", "p12"):
                times[k].append(solve(k))
                st = P.stats()
                if k == "learned":
                    pairs["learned"].append(st["n_pairs"])
                    learned_active.append(st["learned_active"])
        times_p16 = solve("p16")
        if scored:
            times["p16"].append(times_p16)
            pairs["p16"].append(P.stats()["n_pairs"])
            if (step - train_until - 1) % score_every == 0 or step == steps_total:
                times["plain"].append(solve("plain"))
                idx = W.sample_targets(n, score_targets, seed=step)
                for k, r in zip(forms, _rel_l2_at(P, torch, xy, cir, cor, n, [uvs[k] for k in forms], idx, sp)):
                    rels[k].append(r)
        P.advect_device(xy.data_ptr(), uvs["p16"].data_ptr(), n, dt, sp)
    torch.cuda.synchronize()
    P.set_mode(P.MODE_PLAIN)
    P.set_mixed_params(16, 2.5, True)
    nsc = steps_total - train_until
    res = {"workload": "advected_lamb_oseen_1M", "n_blobs": n, "steps_scored": f"{train_until + 1}-{steps_total}",
           "dt": dt, "trajectory": "forward Euler on the device by the fixed mixed form's velocity (P = 16)",
           "score_targets": score_targets, "scored_every": score_every}
    for k in forms:
        ms = statistics.mean(times[k])
        res[k] = {"ms_per_step": ms, "value": n / (ms * 1e-3), "unit": UNIT,
                  "max_relL2_vs_fp64_direct": max(rels[k]), "steps_timed": len(times[k])}
    res["learned"]["learned_active_steps"] = int(sum(learned_active))
    res["learned"]["pairs_ratio_vs_p16"] = float(np.mean(np.array(pairs["learned"]) / np.array(pairs["p16"])))
    res["learned_speedup"] = {"vs_fixed_p12": res["p12"]["ms_per_step"] / res["learned"]["ms_per_step"],
                              "vs_fixed_p16": res["p16"]["ms_per_step"] / res["learned"]["ms_per_step"],
                              "vs_plain": res["plain"]["ms_per_step"] / res["learned"]["ms_per_step"]}
    assert nsc == len(times["learned"])
    return res


def other_configurations(P, torch, stream, flush):
    """Compact measurements of configurations 1, 2, 4 and 5 for the default
    line (each a few steps; the headline is configuration 3)."""
    W = importlib.import_module("2dfmm_gb300.workloads")
    L = importlib.import_module("2dfmm_gb300.learn")
    dev = torch.device("cuda", torch.cuda.current_device())
    sp = stream.cuda_stream
    out = {}
    # configuration 1: the plain path against the reference's own outputs
    g = np.load(os.path.join(ROOT, "tests", "golden", "cfg1.npz"))
    b = W.uniform()
    assert np.array_equal(b.xy, g["xy"])
    P.set_params(int(g["nterms"]), int(g["num_p"]), float(g["theta"]))
    P.set_mode(P.MODE_PLAIN)
    xy, cir, cor, uv = _dev(torch, b, dev)
    solve = lambda: P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), b.n, sp)  # noqa
    _events_ms(torch, stream, solve, 3)
    ms = statistics.mean(_events_ms(torch, stream, solve, 5, flush))
    got = uv.cpu().numpy()
    ref = g["uv"][: b.n]
    comp = np.abs(got - ref) / np.maximum(np.abs(ref), 1e-300)
    nrm = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    out["config1_uniform_20k_plain"] = {
        "value": b.n / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms,
        "vs_reference_outputs": {"max_normwise": float(nrm.max()), "max_per_component": float(comp.max()),
                                 "components_beyond_1e-12": int((comp > 1e-12).sum()), "components": int(comp.size),
                                 "note": "golden outputs of the reference built from its sources; the components "
                                         "beyond 1e-12 are cancellation residues (tests/test_plain_parity.py)"}}
    # configuration 2: plain and learned at 1M
    b = W.lamb_oseen(seed=2)
    P.set_params(b.nterms, b.num_p, b.theta)
    xy, cir, cor, uv = _dev(torch, b, dev)
    idx = W.sample_targets(b.n, 2048, seed=7)
    c2 = {}
    for mode in ("plain", "learned"):
        P.set_mode(MODES[mode])
        _use_learned(P, L, mode)
        solve = lambda: P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), b.n, sp)  # noqa
        _events_ms(torch, stream, solve, 2)
        ms = statistics.mean(_events_ms(torch, stream, solve, 3, flush))
        rel = _rel_l2_at(P, torch, xy, cir, cor, b.n, [uv], idx, sp)[0]
        c2[mode] = {"value": b.n / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms, "relL2_vs_fp64_direct": rel}
    c2["learned_active"] = bool(P.stats()["learned_active"])
    out["config2_lamb_oseen_1M"] = c2
    # configuration 4: 512 sets in one batched solve
    sets = W.batch_sets(nsets=512, seed=4)
    P.set_params(sets[0].nterms, sets[0].num_p, sets[0].theta)
    P.set_mode(P.MODE_MIXED)
    off = np.concatenate([[0], np.cumsum([s_.n for s_ in sets])]).astype(np.int32)
    n = int(off[-1])
    xy = torch.from_numpy(np.concatenate([s_.xy for s_ in sets])).to(dev)
    cir = torch.from_numpy(np.concatenate([s_.cir for s_ in sets])).to(dev)
    cor = torch.from_numpy(np.concatenate([s_.cor for s_ in sets])).to(dev)
    uv = torch.empty_like(xy)
    solve = lambda: P.solve_sets(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), off, sp)  # noqa
    _events_ms(torch, stream, solve, 2)
    ms = statistics.mean(_events_ms(torch, stream, solve, 3, flush))
    rels = []
    for k, s_ in enumerate(sets):
        a, e = int(off[k]), int(off[k + 1])
        rels.append(_rel_l2_at(P, torch, xy[a:e], cir[a:e], cor[a:e], s_.n, [uv[a:e]],
                               W.sample_targets(s_.n, 1024, seed=1000 + k), sp)[0])
    out["config4_batch_512_sets"] = {"value": n / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms, "n_blobs": n,
                                     "relL2_max_over_sets": max(rels), "relL2_median": float(np.median(rels)),
                                     "sets_above_1e-6": int(sum(r > 1e-6 for r in rels)),
                                     "targets_per_set": 1024}
    del xy, cir, cor, uv
    # configuration 5: learned order selection on the advected set
    out["config5_advected"] = advected(P, torch, stream)
    P.set_mode(P.MODE_PLAIN)
    return out


def run_advected(args):
    """`--workload advected`: configuration 5 alone, as its own line."""
    import torch
    torch.cuda.set_device(0)
    P = importlib.import_module("2dfmm_gb300")
    P.load()
    stream = torch.cuda.current_stream()
    with Clocks(0) as clk:
        res = advected(P, torch, stream)
    line = {"metric": "target evals/s on configuration 5 (1M Lamb-Oseen advected), steps 21-100, learned order "
                      "selection, relL2 <= 1e-6 vs FP64 direct",
            "value": res["learned"]["value"], "unit": UNIT, "n_gpus": 1, "steps": len(range(21, 101)),
            "warmup": 3, "ms_per_step": res["learned"]["ms_per_step"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32 (tf32x3 tensor M2L, bf16 MLP, f64 final sum)",
            "data": "synthetic (seeded numpy PCG64)", "config": {"workload": res["workload"]},
            "advected": res, "clocks": clk.summary(), "cpu_baseline": None}
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
    elif args.workload == "batch_sets":
        run_batch(args)
    elif args.workload == "advected":
        run_advected(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
