"""Benchmark: OSTR subset-iterations/s on the clinical DBT workload.

Workload (``clinical``): volume 1024x512x60 @ 0.14x0.14x1.0 mm, detector
1664x832 @ 0.14 mm, 25 views over +-25 deg, 25 subsets (one view each), Huber
penalty delta 0.003/mm, beta 100, seeded synthetic breast phantom with 200
glandular ellipsoids and 40 calcifications, counts Poisson(5e3 exp(-Ax)).

Our arm: one step = one full OSTR iteration (25 sub-iterations, each a fused
forward-projection+gradient kernel and a fused back-projection+penalty+update
kernel) on device-resident data.  ``value`` = subset-iterations/s.  ``e2e`` =
the same metric through ``ostr.reconstruct`` (the public call) from pinned host
buffers: scan upload, gamma/d precompute, 50 iterations, volume download.

``--impl reference``: the reference's algorithm on the host cores (the FP32
CPU restatement of Tomo_OSTR_gold.cpp + Tomo_OSTR.cu, OpenMP over all
cores), one step = one sub-iteration of the same workload.

Multi-GPU (torchrun, N>1): independent replicas, one reconstruction per rank,
no data-path collective; timing is the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

METRIC = "OSTR subset-iterations/s"
UNIT = "subset-iters/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="clinical")
    ap.add_argument("--e2e-iters", type=int, default=None)
    ap.add_argument("--e2e-runs", type=int, default=2)
    ap.add_argument("--cpu-subiters", type=int, default=2)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-threads", type=int, default=0,
                    help="host threads of the CPU baseline (0: all cores)")
    ap.add_argument("--cpu-dtype", default="f32", choices=["f32", "f64"],
                    help="the CPU baseline's arithmetic: the FP32 restatement or the FP64 oracle")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-monotone", action="store_true",
                    help="skip the cost measurement of the monotone (FP64-checked) loops")
    ap.add_argument("--batch", type=int, default=0,
                    help="also time N batched reconstructions (shared launches, one CUDA graph)")
    ap.add_argument("--batch-steps", type=int, default=0,
                    help="batch steps to time (0: the whole run, every case to its last "
                         "iteration)")
    ap.add_argument("--batch-runs", type=int, default=2,
                    help="timed replays of the batch graph (the best is reported)")
    ap.add_argument("--batch-config", default="mixed", choices=["mixed", "fullres"],
                    help="mixed: uneven clinical-pitch cases; fullres: 2048x1024x70 breasts "
                         "at 0.085 mm, 3328x1664 detector, 15 views")
    ap.add_argument("--no-tune", action="store_true")
    ap.add_argument("--upd-tile", type=int, default=None, choices=[0, 1, 2],
                    help="force the OSTR update tile (0: one voxel per thread, 1: two, "
                         "2: one voxel per thread on a TMA-fed ring) "
                         "instead of the tuner's or the default choice")
    ap.add_argument("--algo", default="ostr", choices=["ostr", "ossart", "dual-energy"],
                    help="ostr (the headline), ossart (the SART family on the same workload) "
                         "or dual-energy (syncrecon.m's subtraction on clinical-size volumes)")
    ap.add_argument("--supersample", action="store_true",
                    help="--algo ossart with the 2 x 2 sub-ray (4R) projector")
    ap.add_argument("--no-warm", action="store_true",
                    help="skip the learned warm-start comparison")
    return ap.parse_args()


def _scan_name(cfg):
    g = cfg.geom
    return (f"{cfg.name}: {g.nx}x{g.ny}x{g.nz} vox @{g.vx:g}x{g.vy:g}x{g.vz:g}mm, "
            f"{g.nbx}x{g.nby} det @{g.bx:g}mm, {g.n_angles} views "
            f"+-{float(np.degrees(np.abs(cfg.angles).max())):.3g}deg, {cfg.subset_num} subsets")


def workload_name(cfg):
    return (f"{_scan_name(cfg)}, {cfg.potential} d={cfg.delta:g} b={cfg.beta:g}, "
            f"I0={cfg.I0:g}")


def sart_workload_name(cfg, supersample):
    """The OS-SART workload on a config's scan (both arms print this)."""
    return (f"{_scan_name(cfg)}, OS-SART lambda 0.8, cos projector"
            + (" (2x2 sub-rays per bin)" if supersample else "")
            + f", hyperbola prior beta -0.2 d={cfg.delta:g}, line integrals of "
              f"Poisson({cfg.I0:g}) counts")


def make_scan_gpu(cfg, seed):
    """Phantom + counts; the counts' forward projection runs on the GPU."""
    import torch

    from newrecon_gb300 import ostr
    from newrecon_gb300.phantom import breast_phantom, poisson_counts

    g = cfg.geom
    x = breast_phantom(g, seed, cfg.n_glandular, cfg.n_calc, thickness_mm=cfg.thickness_mm)
    ostr.set_geometry(g)
    idx = np.arange(g.n_angles, dtype=np.int32)
    line = torch.zeros(g.n_angles * g.n_bins, device="cuda")
    ostr.fprojectCB_1R_GPU_OSTR_cos(torch.from_numpy(x.ravel()).cuda(), line,
                                    torch.from_numpy(cfg.angles).cuda(),
                                    torch.from_numpy(idx).cuda(), 0, g.n_angles)
    y = poisson_counts(line.cpu().numpy(), cfg.I0, seed)
    b = np.full_like(y, cfg.I0)
    return x.ravel(), y, b


class Clocks:
    """nvidia-smi sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.p = None
        self.path = os.path.join("/tmp", f"nr_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.f = open(self.path, "w")
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "100"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
        time.sleep(0.3)

    def stop(self):
        if self.p is None:
            return None
        time.sleep(0.2)
        self.p.terminate()
        self.p.wait()
        self.f.close()
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in open(self.path):
            parts = [s.strip() for s in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = max(mx, float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def measured_peaks():
    path = os.path.join(HERE, "MEASURED_PEAKS.json")
    if os.path.isfile(path):
        d = json.load(open(path))
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def cpu_info():
    model = ""
    try:
        for ln in open("/proc/cpuinfo"):
            if ln.lower().startswith(("model name", "cpu part")):
                model = ln.split(":", 1)[1].strip()
                break
    except OSError:
        pass
    return os.cpu_count(), model


def cpu_port_subiters(cfg, x_true, y, b, d, n_sub: int, threads: int, dtype=np.float32):
    """The CPU restatement (FP32, or FP64 as the oracle), n_sub sub-iterations
    on `threads` host cores (s per sub-iter)."""
    from oracle.oracle import Oracle

    g = cfg.geom
    O = Oracle(dtype)
    O.set_threads(threads)
    M = cfg.subset_num
    A = g.n_angles
    ridx = O.reorder_index(A, M)
    yr = O.regroup(y, A, M)
    br = O.regroup(b, A, M)
    Vs = A // M
    x = np.zeros(g.n_voxels, dtype)
    d = np.ascontiguousarray(d, dtype)
    times = []
    for k in range(n_sub):
        a = k % M
        t0 = time.perf_counter()
        O.subiter(g, cfg.angles, ridx, a * Vs, (a + 1) * Vs, yr[a * Vs * g.n_bins:(a + 1) * Vs * g.n_bins],
                  br[a * Vs * g.n_bins:(a + 1) * Vs * g.n_bins], d, x, subset_num=M, beta=cfg.beta,
                  delta=cfg.delta, potential=cfg.potential)
        times.append(time.perf_counter() - t0)
    return times


def run_ours(args):
    import torch
    import torch.distributed as dist

    from newrecon_gb300 import native, ostr, replicas
    from newrecon_gb300.geometry import config

    ws, rank, local = replicas.env()
    if ws > 1:
        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    native.load()
    seed = replicas.case_seed(0, rank)
    cfg = config(args.config, seed=seed)
    g = cfg.geom
    x_true, y, b = make_scan_gpu(cfg, seed=seed)
    plan = ostr.OSTR(g, subset_num=cfg.subset_num, beta=cfg.beta, delta=cfg.delta,
                     potential=cfg.potential)
    plan.setup(cfg.angles, y, b)
    M = cfg.subset_num
    xa = torch.zeros(g.n_voxels, device="cuda")
    xb = torch.zeros(g.n_voxels, device="cuda")
    tuned = None if args.no_tune else plan.autotune(xa)
    if args.upd_tile is not None:
        plan.params.upd_tile = args.upd_tile
    stream = torch.cuda.current_stream()

    def step(evs=None):
        nonlocal xa, xb
        for a in range(M):
            if evs is not None:
                evs[0].record(stream)
            plan.project(xa, a)
            if evs is not None:
                evs[1].record(stream)
            plan.update(xa, xb, a)
            if evs is not None:
                evs[2].record(stream)
                evs = evs[3:]
            xa, xb = xb, xa

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    plan.check()
    events = [torch.cuda.Event(enable_timing=True) for _ in range(3 * M * args.steps)]
    clocks = Clocks(local)
    clocks.start()
    if ws > 1:
        dist.barrier()
    torch.cuda.synchronize()
    t_start = torch.cuda.Event(enable_timing=True)
    t_end = torch.cuda.Event(enable_timing=True)
    t_start.record(stream)
    for s in range(args.steps):
        step(events[3 * M * s:3 * M * (s + 1)])
    t_end.record(stream)
    torch.cuda.synchronize()
    if ws > 1:
        dist.barrier()
    clk = clocks.stop()
    elapsed = t_start.elapsed_time(t_end) / 1e3
    elapsed, n_sub = replicas.reduce_timing(elapsed, M * args.steps)
    plan.check()
    fp_ms = np.array([events[3 * k].elapsed_time(events[3 * k + 1]) for k in range(M * args.steps)])
    up_ms = np.array([events[3 * k + 1].elapsed_time(events[3 * k + 2])
                      for k in range(M * args.steps)])
    value = n_sub / elapsed
    N = g.n_voxels
    B = g.n_bins
    Vs = g.n_angles // M
    fp_bytes = 4 * N * Vs + 12 * B * Vs       # x read per view + y, b read + h written
    up_bytes = 12 * N + 4 * B * Vs            # x, d read + x' written + h read
    peak, peak_kind = measured_peaks()
    kern = {
        "ostr_fp_h": {"avg_ms": float(fp_ms.mean()), "bytes": fp_bytes,
                      "gbs": fp_bytes / (fp_ms.mean() / 1e3) / 1e9},
        "ostr_update": {"avg_ms": float(up_ms.mean()), "bytes": up_bytes,
                        "gbs": up_bytes / (up_ms.mean() / 1e3) / 1e9},
    }
    dom = max(kern, key=lambda k: kern[k]["avg_ms"])
    ach = kern[dom]["gbs"]
    traffic = None
    prof_traffic = os.path.join(HERE, "profiles", "dram_traffic.txt")
    if os.path.isfile(prof_traffic) and args.config == "clinical":
        for ln in open(prof_traffic):
            parts = ln.split()
            if len(parts) >= 2 and not ln.startswith("#") and parts[0] == dom:
                traffic = float(parts[1])
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": elapsed / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded breast phantom, Poisson counts)",
        "config": {"workload": workload_name(cfg),
                   "step": f"1 OSTR iteration = {M} sub-iterations",
                   "parallelism": f"replicas x{ws}",
                   "l2": f"inputs larger than L2 (x, x', d: 3 x {4 * g.n_voxels / 1e6:.0f} MB; "
                         f"y, b: 2 x {4 * g.n_angles * g.n_bins / 1e6:.0f} MB)"},
        "gpu_launches": 2 * M * args.steps,
        "tuned": None if tuned is None else {"fp_batch": tuned["fp_batch"],
                                             "fp_stage": tuned.get("fp_stage", 0),
                                             "upd_planes": tuned["upd_planes"],
                                             "upd_tile": tuned.get("upd_tile", 0),
                                             "fp_ms": tuned.get("fp_ms"),
                                             "update_ms": tuned.get("update_ms")},
        "roofline": {"bound": "hbm", "kernel": dom, "achieved": ach, "peak": peak,
                     "peak_kind": peak_kind, "unit": "GB/s", "frac": ach / peak,
                     "traffic": traffic, "kernels": kern},
    }
    if clk is not None:
        out["clocks"] = clk
    if not args.no_e2e:
        out["e2e"] = e2e_ours(args, cfg, y, b)
    if not args.no_monotone:
        out["monotone"] = monotone_cost(plan, g)
    if rank == 0 and not args.no_cpu_baseline:
        d = plan.section("d").cpu().numpy()
        threads = args.cpu_threads or os.cpu_count() or 1
        dt = np.float64 if args.cpu_dtype == "f64" else np.float32
        times = cpu_port_subiters(cfg, x_true, y, b, d, args.cpu_subiters, threads, dt)
        ncpu, model = cpu_info()
        prec = "FP64 oracle" if dt == np.float64 else "FP32 restatement"
        out["cpu_baseline"] = {"value": len(times) / sum(times), "unit": UNIT, "cores": threads,
                               "kind": "port",
                               "sample": f"{len(times)} sub-iterations of the {cfg.name} workload "
                                         f"({prec}, OpenMP on {threads} of {ncpu} cores), {model}"}
    if not args.no_warm:
        out["warm_start"] = warm_bench(cfg, plan, rank, x_true=x_true)
    if args.batch:
        out["batch"] = batch_bench(args, rank)
    if ws > 1:
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(out), flush=True)


def monotone_cost(plan, g):
    """Wall time of one iteration of the plain loop, of the loop with the
    FP64 objective check per iteration (monotone=True) and with the subset
    objective check per sub-iteration (monotone="subset"), from the same
    start; and of one FP64 objective evaluation."""
    import torch

    stream = torch.cuda.current_stream()
    x0 = torch.zeros(g.n_voxels, device="cuda")
    plan.iterate(x0, 2)  # a start away from zero

    def timed(fn, reps=3):
        best = float("inf")
        for _ in range(reps):
            x = x0.clone()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            fn(x)
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best * 1e3

    plain = timed(lambda x: plan.iterate(x, 1))
    it = timed(lambda x: plan.iterate(x, 1, monotone=True))
    sub = timed(lambda x: plan.iterate(x, 1, monotone="subset"))
    # a whole 50-iteration run with the objective checked every 25 iterations
    # (start, 25, 50) against the plain run
    plain50 = timed(lambda x: plan.iterate(x, 50), reps=1)
    ck25 = timed(lambda x: plan.iterate(x, 50, monotone=True, check_every=25), reps=1)
    obj = timed(lambda x: plan.objective(x))
    a = torch.cuda.Event(enable_timing=True)
    b = torch.cuda.Event(enable_timing=True)
    x = x0.clone()
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    plan.penalty(x, out)
    a.record(stream)
    plan.penalty(x, out)
    b.record(stream)
    b.synchronize()
    return {"plain_iteration_ms": plain, "monotone_iteration_ms": it,
            "monotone_subset_iteration_ms": sub, "objective_ms": obj,
            "penalty_fp64_ms": a.elapsed_time(b),
            "overhead_iteration": it / plain - 1.0, "overhead_subset": sub / plain - 1.0,
            "plain_50_iterations_ms": plain50, "monotone_check_every_25_ms": ck25,
            "overhead_check_every_25": ck25 / plain50 - 1.0,
            "note": "wall time from a start two iterations in; monotone=True adds one FP64 "
                    "objective (all views + penalty) per iteration (per 25 with check_every=25), "
                    "monotone=\"subset\" one projection of the subset's views and one penalty "
                    "per sub-iteration"}


def batch_bench(args, rank):
    """N independent reconstructions of uneven size and view count advanced
    together by shared batched launches (the whole loop one CUDA graph); the
    same cases one after another, each through its own graph, for scale."""
    import torch

    from newrecon_gb300 import ostr, replicas
    from newrecon_gb300.geometry import batch_configs, config
    from newrecon_gb300.phantom import breast_phantom, poisson_counts

    fullres = args.batch_config == "fullres"
    if fullres:
        cfgs = [config("fullres", seed=replicas.case_seed(11, rank) * 100 + k)
                for k in range(args.batch)]
    else:
        cfgs = batch_configs(args.batch, seed=replicas.case_seed(7, rank))
    cases = []
    for c in cfgs:
        g = c.geom
        if fullres:
            x = breast_phantom(g, c.seed, c.n_glandular, c.n_calc, thickness_mm=c.thickness_mm)
        else:
            x = breast_phantom(g, c.seed, 0, c.n_calc, glandular_fraction=c.n_glandular / 100.0)
        ostr.set_geometry(g)
        idx = np.arange(g.n_angles, dtype=np.int32)
        line = torch.zeros(g.n_angles * g.n_bins, device="cuda")
        ostr.fprojectCB_1R_GPU_OSTR_cos(torch.from_numpy(x.ravel()).cuda(), line,
                                        torch.from_numpy(c.angles).cuda(),
                                        torch.from_numpy(idx).cuda(), 0, g.n_angles)
        y = poisson_counts(line.cpu().numpy(), c.I0, c.seed)
        cases.append(dict(geom=g, angles=c.angles, prj=y, blank=np.full_like(y, c.I0),
                          subset_num=c.subset_num, iter_num=c.iter_num, beta=c.beta,
                          delta=c.delta, potential=c.potential))
    bt = ostr.Batch(cases, tune=not args.no_tune)
    stream = torch.cuda.current_stream()
    full = args.batch_steps <= 0 or args.batch_steps >= bt.n_steps
    steps = bt.n_steps if full else args.batch_steps
    subits = sum(min(steps, cs["iter_num"] * cs["subset_num"]) for cs in cases)

    def timed(launch, reset):
        """Best of args.batch_runs replays after one warm-up, each from x = 0."""
        launch()
        best = float("inf")
        for _ in range(max(1, args.batch_runs)):
            reset()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            launch()
            e1.record(stream)
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) / 1e3)
        return best

    def zero_all():
        for xx in bt.x:
            xx.zero_()

    # the batch: steps 0 .. steps-1 (and the finish) captured once as a CUDA graph
    gr = bt.graph(steps)
    t_batch = timed(gr.launch, zero_all)
    bt.check()
    gr.close()
    # the same cases one after another through the single-case kernels: each
    # case's whole iteration loop as its own graph (or, for a partial run, its
    # first sub-iterations launched one by one)
    t_seq = 0.0
    for p, xx, cs in zip(bt.plans, bt.x, cases):
        if full:
            g1 = p.graph(xx, cs["iter_num"])
            t_seq += timed(g1.launch, xx.zero_)
            g1.close()
        else:
            n = min(steps, cs["iter_num"] * cs["subset_num"])
            xo = torch.empty_like(xx)

            def run(p=p, xx=xx, xo=xo, n=n):
                a, b_ = xx, xo
                for k in range(n):
                    s_ = k % p.params.subset_num
                    p.project(a, s_)
                    p.update(a, b_, s_)
                    a, b_ = b_, a
            t_seq += timed(run, xx.zero_)
    vox = sum(cs["geom"].n_voxels for cs in cases)
    return {"cases": len(cases), "steps_timed": steps, "whole_run": full,
            "mode": bt.mode if full else "shared",
            "timing": "CUDA graph replay of " + ("the whole batch (every step and the finish)"
                                                 if full else f"the first {steps} steps"),
            "voxels_total": vox, "seconds": t_batch,
            "subset_iters_per_s": subits / t_batch,
            "projections_per_s": subits / t_batch,
            "volumes_per_hour": len(cases) * 3600.0 / t_batch if full else None,
            "sequential_subset_iters_per_s": subits / t_seq,
            "sequential_volumes_per_hour": len(cases) * 3600.0 / t_seq if full else None,
            "workload": ("full resolution: 2048x1024x70 @0.085x0.085x1mm, 3328x1664 det "
                         "@0.085mm, 15 views +-7.5deg, I0 4e3, hyperbola d=0.002 b=200, "
                         "50 iterations" if fullres else
                         "batch: thickness U(30,80), in-plane U(512,1024)xU(256,512) @0.14mm, "
                         "9/15/25 views over +-U(7.5,25) deg, I0 U(3e3,2e4), gland U(10,50)%, "
                         "hyperbola, 50 iterations"),
            "gpu_memory_gb": torch.cuda.max_memory_allocated() / 1e9}


def warm_bench(cfg, plan, rank, x_true=None, tol=1e-4, early=2):
    """Time to RMSE <= tol (1/mm) against the 50-iteration volume: plain OSTR
    vs the learned warm start (2 iterations, CNN, then iterations), both from
    the scan already resident; the target's two criteria (objective within 1 %
    of plain OSTR's 50-iteration objective gap, RMSE against the phantom within
    1 % of plain OSTR's after 50 iterations); plus the CNN's own throughput on
    this volume.  The network trained for this workload is used when there is
    one (data/warmstart_<workload>.npz), else the batched workload's."""
    import torch

    from newrecon_gb300 import warmstart

    data = os.path.join(HERE, "newrecon_gb300", "data")
    matched = os.path.join(data, f"warmstart_{cfg.name}.npz")
    path = matched if os.path.isfile(matched) else os.path.join(data, "warmstart_params.npz")
    if not os.path.isfile(path):
        return {"unavailable": "no trained parameters"}
    cnn = warmstart.load(path)
    trained_for = cfg.name if path == matched else "batch (hyperbola, delta 0.002, beta 50)"
    g = cfg.geom
    ref = torch.zeros(g.n_voxels, device="cuda")
    plan.iterate(ref, cfg.iter_num)
    stream = torch.cuda.current_stream()

    def rmse(a):
        return float(torch.sqrt(torch.mean((a.double() - ref.double()) ** 2)).item())

    dims = (g.nx, g.ny, g.nz, 1)
    x = torch.zeros(g.n_voxels, device="cuda")
    plan.iterate(x, early)
    cnn.forward(x, dims)  # warm-up (workspace, weight packing)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    xw = cnn.forward(x, dims)
    e1.record(stream)
    torch.cuda.synchronize()
    cnn.check()
    cnn_ms = e0.elapsed_time(e1)
    flops = g.n_voxels * 2 * 27 * (1 * 32 + 4 * 32 * 32 + 32 * 1)
    # equal-work objective check (3 iterations after the warm start vs plain)
    xp = x.clone()
    plan.iterate(xp, 3)
    plan.iterate(xw, 3)
    obj_p, obj_w = plan.total_objective(xp), plan.total_objective(xw)

    cap = cfg.iter_num + 10

    def iters_to_tol(start_warm):
        """Iterations until RMSE <= tol (None if not within cap), untimed."""
        y = torch.zeros(g.n_voxels, device="cuda")
        its = 0
        if start_warm:
            plan.iterate(y, early)
            y = cnn.forward(y, dims)
            its = early
        while its <= cap:
            if rmse(y) <= tol:
                return its, rmse(y)
            plan.iterate(y, 1)
            its += 1
        return None, rmse(y)

    def timed(start_warm, its):
        """Wall time of exactly that work from x = 0 (scan resident, no checks inside)."""
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        y = torch.zeros(g.n_voxels, device="cuda")
        if start_warm:
            plan.iterate(y, early)
            y = cnn.forward(y, dims)
            plan.iterate(y, its - early)
        else:
            plan.iterate(y, its)
        torch.cuda.synchronize()
        return time.perf_counter() - t0

    ip, rp = iters_to_tol(False)
    iw, rw = iters_to_tol(True)
    tp = timed(False, ip) if ip is not None else None
    tw = timed(True, iw) if iw is not None else None
    crit = None
    if x_true is not None:
        pair = warmstart.Pair(cfg, None, None, None, None, x_true)
        crit = warmstart.criteria(cnn, plan, pair, early, full=cfg.iter_num)
    return {"trained_for": trained_for, "criteria": crit,
            "tol_per_mm": tol, "reference": f"{cfg.iter_num}-iteration plain OSTR",
            "plain": {"iterations": ip, "seconds": tp, "rmse": rp},
            "warm": {"iterations": iw, "seconds": tw, "rmse_at_stop": rw,
                     "reached": iw is not None},
            "speedup": (tp / tw) if (tp and tw) else None,
            "objective_after_5_iters": {"plain": obj_p, "warm": obj_w,
                                        "warm_accepted": obj_w <= obj_p},
            "cnn_ms": cnn_ms, "cnn_tflops": flops / (cnn_ms / 1e3) / 1e12,
            "cnn_flops": flops}


def ctypes_ptr(t):
    import ctypes

    return ctypes.c_void_p(t.data_ptr())


def stream_ptr():
    import ctypes

    import torch

    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def e2e_ours(args, cfg, y, b):
    import torch

    from newrecon_gb300 import ostr

    iters = args.e2e_iters or cfg.iter_num
    g = cfg.geom
    y_h = torch.from_numpy(y).pin_memory()
    b_h = torch.from_numpy(b).pin_memory()
    a_h = torch.from_numpy(cfg.angles).pin_memory()
    kw = dict(angles=a_h, subset_num=cfg.subset_num, iter_num=iters, beta=cfg.beta,
              delta=cfg.delta, potential=cfg.potential)
    ostr.reconstruct(g, y_h, b_h, **kw)  # warm-up
    torch.cuda.synchronize()
    ts = []
    phases = []
    vol = None
    for _ in range(args.e2e_runs):
        # the caller is done with the previous volume (its pinned block goes
        # back to torch's host cache, as in a stream of reconstructions)
        vol = None
        ph = {}
        t0 = time.perf_counter()
        vol = ostr.reconstruct(g, y_h, b_h, timing=ph, **kw)
        torch.cuda.synchronize()
        ts.append(time.perf_counter() - t0)
        phases.append(ph)
    assert vol.device.type == "cpu"
    sub = iters * cfg.subset_num
    # device time of each phase (CUDA events inside reconstruct), averaged over
    # the runs; "host_s" is the rest of the call's wall time (plan and
    # workspace creation, Python, launch gaps)
    ph = {k: float(np.mean([p[k] for p in phases]))
          for k in ("upload_s", "setup_s", "iterate_s", "download_s")}
    ph["host_s"] = float(np.mean(ts)) - sum(ph.values())
    ph["iterate_subiters_per_s"] = sub / ph["iterate_s"]
    return {"value": sub / float(np.mean(ts)), "unit": UNIT, "phases": ph,
            "h2d_bytes_per_step": int(y.nbytes + b.nbytes + cfg.angles.nbytes),
            "d2h_bytes_per_step": int(g.n_voxels * 4),
            "step": f"ostr.reconstruct from pinned host buffers: upload, gamma/d setup, "
                    f"{iters} iterations x {cfg.subset_num} subsets (the kernel variants "
                    f"the tuner cached for this geometry, if any), volume download",
            "seconds_per_call": float(np.mean(ts))}


def run_reference(args):
    from newrecon_gb300 import replicas

    ws, rank, local = replicas.env()
    if rank != 0:
        return
    from newrecon_gb300.geometry import config
    from newrecon_gb300.phantom import breast_phantom, poisson_counts
    from oracle import build as obuild
    from oracle.oracle import Oracle

    if not os.path.isfile(obuild.ORACLE_SO):
        obuild.build_oracle().wait()
    cfg = config(args.config, seed=0)
    g = cfg.geom
    threads = os.cpu_count() or 1
    O = Oracle(np.float32)
    O.set_threads(threads)
    x = breast_phantom(g, 0, cfg.n_glandular, cfg.n_calc, thickness_mm=cfg.thickness_mm).ravel()
    idx = np.arange(g.n_angles, dtype=np.int32)
    y = poisson_counts(O.fp_ostr(g, x, cfg.angles, idx, 0, g.n_angles), cfg.I0, 0)
    b = np.full_like(y, cfg.I0)
    # d = SBP(gamma * yry) over all views, as the reference precomputes it
    gam = O.fp_gamma(g, cfg.angles, idx, 0, g.n_angles, "length")
    d = O.bp_sbp(g, O.compute_yry(y) * gam, idx, cfg.angles, 0, g.n_angles)
    times = cpu_port_subiters(cfg, x, y, b, d, args.warmup + args.steps, threads)[args.warmup:]
    elapsed = float(sum(times))
    value = len(times) / elapsed
    ncpu, model = cpu_info()
    out = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": elapsed / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded breast phantom, Poisson counts)",
        "config": {"workload": workload_name(cfg),
                   "step": "1 OSTR sub-iteration on the host cores", "parallelism": "host"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{len(times)} sub-iterations (FP32 restatement of the "
                                   f"reference's gold path, OpenMP), {model}"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out), flush=True)


# ---------------------------------------------------------------------------
# OS-SART on the same workload (--algo ossart): lambda 0.8, cos projector,
# hyperbola prior (beta -0.2, the workload's delta).

SART_METRIC = "OS-SART subset-iterations/s"
SART_KW = dict(lam=0.8, use_cos=True, regularized=True, beta=-0.2)


def sart_line(cfg, y, b):
    import torch

    from newrecon_gb300 import sart

    return sart.line_integrals(torch.from_numpy(y).cuda(), torch.from_numpy(b).cuda())


def cpu_port_ossart(cfg, line, n_sub: int, threads: int):
    """FP32 CPU restatement of the OS-SART sub-iteration (s per sub-iteration):
    SART projection, difference, SART prior, OS-SART back projection."""
    from oracle.oracle import Oracle

    g = cfg.geom
    O = Oracle(np.float32)
    O.set_threads(threads)
    M, A = cfg.subset_num, g.n_angles
    Vs, B = A // M, g.n_bins
    ridx = O.reorder_index(A, M)
    lr = O.regroup(line, A, M)
    x = np.zeros(g.n_voxels, np.float32)
    times = []
    for k in range(n_sub):
        a = k % M
        a0, a1 = a * Vs, (a + 1) * Vs
        t0 = time.perf_counter()
        est, norm = O.fp_sart(g, x, cfg.angles, ridx, a0, a1, SART_KW["use_cos"])
        diff = O.sart_prj_diff(lr[a0 * B:a1 * B], est, norm)
        prior = O.prior_sart(g, x, cfg.delta)
        x = O.bp_ossart(g, x, diff, ridx, cfg.angles, a0, a1, SART_KW["lam"], prior,
                        SART_KW["beta"])
        times.append(time.perf_counter() - t0)
    return times


def run_ossart(args):
    import torch
    import torch.distributed as dist

    from newrecon_gb300 import native, replicas, sart
    from newrecon_gb300.geometry import config

    ws, rank, local = replicas.env()
    if ws > 1:
        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    native.load()
    seed = replicas.case_seed(0, rank)
    cfg = config(args.config, seed=seed)
    g = cfg.geom
    x_true, y, b = make_scan_gpu(cfg, seed=seed)
    line = sart_line(cfg, y, b)
    M = cfg.subset_num
    plan = sart.OSSART(g, subset_num=M, delta=cfg.delta, supersample=args.supersample, **SART_KW)
    plan.setup(cfg.angles, line)
    xa = torch.zeros(g.n_voxels, device="cuda")
    xb = torch.zeros(g.n_voxels, device="cuda")
    stream = torch.cuda.current_stream()

    def step(evs=None):
        nonlocal xa, xb
        for a in range(M):
            if evs is not None:
                evs[0].record(stream)
            plan.project(xa, a)
            if evs is not None:
                evs[1].record(stream)
            plan.update(xa, xb, a)
            if evs is not None:
                evs[2].record(stream)
                evs = evs[3:]
            xa, xb = xb, xa

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    plan.check()
    events = [torch.cuda.Event(enable_timing=True) for _ in range(3 * M * args.steps)]
    clocks = Clocks(local)
    clocks.start()
    if ws > 1:
        dist.barrier()
    torch.cuda.synchronize()
    t_start = torch.cuda.Event(enable_timing=True)
    t_end = torch.cuda.Event(enable_timing=True)
    t_start.record(stream)
    for s in range(args.steps):
        step(events[3 * M * s:3 * M * (s + 1)])
    t_end.record(stream)
    torch.cuda.synchronize()
    if ws > 1:
        dist.barrier()
    clk = clocks.stop()
    elapsed = t_start.elapsed_time(t_end) / 1e3
    elapsed, n_sub = replicas.reduce_timing(elapsed, M * args.steps)
    plan.check()
    fp_ms = np.array([events[3 * k].elapsed_time(events[3 * k + 1]) for k in range(M * args.steps)])
    up_ms = np.array([events[3 * k + 1].elapsed_time(events[3 * k + 2])
                      for k in range(M * args.steps)])
    N, B, Vs = g.n_voxels, g.n_bins, g.n_angles // M
    fp_bytes = 4 * N * Vs + 12 * B * Vs       # x read per view + p, norm read + diff written
    up_bytes = 8 * N + 4 * B * Vs             # x read + x' written + diff read
    peak, peak_kind = measured_peaks()
    kern = {
        "sart_fp_diff": {"avg_ms": float(fp_ms.mean()), "bytes": fp_bytes,
                         "gbs": fp_bytes / (fp_ms.mean() / 1e3) / 1e9},
        "sart_update": {"avg_ms": float(up_ms.mean()), "bytes": up_bytes,
                        "gbs": up_bytes / (up_ms.mean() / 1e3) / 1e9},
    }
    dom = max(kern, key=lambda k: kern[k]["avg_ms"])
    traffic = None
    prof_traffic = os.path.join(HERE, "profiles", "dram_traffic.txt")
    if os.path.isfile(prof_traffic):
        for ln in open(prof_traffic):
            parts = ln.split()
            if len(parts) >= 2 and not ln.startswith("#") and parts[0] == dom:
                traffic = float(parts[1])
    workload = sart_workload_name(cfg, args.supersample)
    out = {
        "metric": SART_METRIC, "value": n_sub / elapsed, "unit": UNIT, "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": elapsed / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded breast phantom, Poisson counts, log transform)",
        "config": {"workload": workload, "step": f"1 OS-SART iteration = {M} sub-iterations",
                   "parallelism": f"replicas x{ws}",
                   "l2": f"inputs larger than L2 (x, x': 2 x {4 * g.n_voxels / 1e6:.0f} MB; "
                         f"p, norm: 2 x {4 * g.n_angles * g.n_bins / 1e6:.0f} MB)"},
        "gpu_launches": 2 * M * args.steps,
        "roofline": {"bound": "hbm", "kernel": dom, "achieved": kern[dom]["gbs"], "peak": peak,
                     "peak_kind": peak_kind, "unit": "GB/s",
                     "frac": kern[dom]["gbs"] / peak, "traffic": traffic, "kernels": kern},
    }
    if clk is not None:
        out["clocks"] = clk
    if not args.no_e2e:
        iters = args.e2e_iters or cfg.iter_num
        l_h = line.cpu().pin_memory()
        a_h = torch.from_numpy(cfg.angles).pin_memory()
        kw = dict(angles=a_h, subset_num=M, iter_num=iters, delta=cfg.delta,
                  supersample=args.supersample, **SART_KW)
        sart.ossart_reconstruct(g, l_h, **kw)
        torch.cuda.synchronize()
        ts = []
        vol = None
        for _ in range(args.e2e_runs):
            vol = None  # the previous volume released, as in ostr's e2e leg
            t0 = time.perf_counter()
            vol = sart.ossart_reconstruct(g, l_h, **kw)
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t0)
        assert vol.device.type == "cpu"
        out["e2e"] = {"value": iters * M / float(np.mean(ts)), "unit": UNIT,
                      "h2d_bytes_per_step": int(l_h.numel() * 4 + cfg.angles.nbytes),
                      "d2h_bytes_per_step": int(g.n_voxels * 4),
                      "step": f"sart.ossart_reconstruct from pinned host line integrals: upload, "
                              f"chord setup, {iters} iterations x {M} subsets, volume download",
                      "seconds_per_call": float(np.mean(ts))}
    if rank == 0 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        times = cpu_port_ossart(cfg, line.cpu().numpy(), args.cpu_subiters, threads)
        ncpu, model = cpu_info()
        out["cpu_baseline"] = {"value": len(times) / sum(times), "unit": UNIT, "cores": threads,
                               "kind": "port",
                               "sample": f"{len(times)} OS-SART sub-iterations of the clinical "
                                         f"workload (FP32 restatement of the reference's SART "
                                         f"kernels, OpenMP), {model}"}
    if ws > 1:
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(out), flush=True)


def run_reference_ossart(args):
    from newrecon_gb300 import replicas

    ws, rank, local = replicas.env()
    if rank != 0:
        return
    from newrecon_gb300.geometry import config
    from newrecon_gb300.phantom import breast_phantom, poisson_counts
    from oracle import build as obuild
    from oracle.oracle import Oracle

    if not os.path.isfile(obuild.ORACLE_SO):
        obuild.build_oracle().wait()
    cfg = config(args.config, seed=0)
    g = cfg.geom
    threads = os.cpu_count() or 1
    O = Oracle(np.float32)
    O.set_threads(threads)
    x = breast_phantom(g, 0, cfg.n_glandular, cfg.n_calc, thickness_mm=cfg.thickness_mm).ravel()
    idx = np.arange(g.n_angles, dtype=np.int32)
    y = poisson_counts(O.fp_ostr(g, x, cfg.angles, idx, 0, g.n_angles), cfg.I0, 0)
    line = O.line_integrals(y, np.full_like(y, cfg.I0))
    times = cpu_port_ossart(cfg, line, args.warmup + args.steps, threads)[args.warmup:]
    elapsed = float(sum(times))
    value = len(times) / elapsed
    ncpu, model = cpu_info()
    print(json.dumps({
        "impl": "reference", "metric": SART_METRIC, "value": value, "unit": UNIT, "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": elapsed / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded breast phantom, Poisson counts, log transform)",
        "config": {"workload": sart_workload_name(cfg, args.supersample),
                   "step": "1 OS-SART sub-iteration on the host cores", "parallelism": "host"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{len(times)} sub-iterations (FP32 restatement of the "
                                   f"reference's SART kernels, OpenMP), {model}"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


# ---------------------------------------------------------------------------
# Dual-energy subtraction (--algo dual-energy): the nine weights of
# syncrecon.m on two clinical-size volumes (1024x512x60), slice-30 entropies.

DE_METRIC = "dual-energy subtracted volumes/s"


def de_volumes(n, seed=0):
    rng = np.random.default_rng(seed)
    he = rng.gamma(2.0, 0.02, size=n).astype(np.float32)
    le = (he * np.float32(1.3) + rng.normal(0, 0.003, n).astype(np.float32)).astype(np.float32)
    return he, le


def run_dual_energy(args):
    import torch

    from newrecon_gb300 import dual_energy, native, replicas
    from newrecon_gb300.geometry import config

    ws, rank, local = replicas.env()
    torch.cuda.set_device(local)
    native.load()
    g = config(args.config).geom
    n = g.n_voxels
    w = list(dual_energy.DEFAULT_WEIGHTS)
    he, le = de_volumes(n)
    h = torch.from_numpy(he).cuda()
    l = torch.from_numpy(le).cuda()
    out = torch.empty((len(w), n), device="cuda")
    kw = dict(slice_shape=(g.nx, g.ny), entropy_slice=g.nz // 2, out=out)
    for _ in range(args.warmup):
        dual_energy.subtract(h, l, w, **kw)
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
           for _ in range(args.steps)]
    clocks = Clocks(local)
    clocks.start()
    for e0, e1 in evs:
        e0.record(stream)
        dual_energy.subtract(h, l, w, **kw)   # includes the slice histograms and their D2H
        e1.record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    ms = np.array([e0.elapsed_time(e1) for e0, e1 in evs])
    nbytes = 8 * n + 4 * len(w) * n          # he, le read once; K volumes written
    peak, peak_kind = measured_peaks()
    gbs = nbytes / (ms.mean() / 1e3) / 1e9
    # e2e: the file-level workflow's device part from pinned host volumes to host d
    h_h = torch.from_numpy(he).pin_memory()
    l_h = torch.from_numpy(le).pin_memory()
    d_h = torch.empty((len(w), n), dtype=torch.float32).pin_memory()
    ts = []
    for _ in range(max(2, args.e2e_runs)):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        hd = h_h.cuda(non_blocking=True)
        ld = l_h.cuda(non_blocking=True)
        dual_energy.subtract(hd, ld, w, **kw)
        d_h.copy_(out, non_blocking=True)
        torch.cuda.synchronize()
        ts.append(time.perf_counter() - t0)
    out_json = {
        "metric": DE_METRIC, "value": 1e3 / ms.mean() * len(w), "unit": "volumes/s",
        "n_gpus": ws, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": float(ms.mean()), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 error-free arithmetic (f64 for undecided near-ties), f32 volumes",
        "data": "synthetic gamma-distributed volumes",
        "config": {"workload": f"{g.nx}x{g.ny}x{g.nz} HE and LE volumes, 9 weights 0.1..0.9, "
                               f"slice-{g.nz // 2} entropies (syncrecon.m)",
                   "step": "nine subtracted volumes + slice histograms + entropies",
                   "l2": "inputs larger than L2 (2 x 126 MB in, 9 x 126 MB out)"},
        "gpu_launches": 2 * args.steps,
        "roofline": {"bound": "hbm", "kernel": "de_subtract", "achieved": gbs, "peak": peak,
                     "peak_kind": peak_kind, "unit": "GB/s", "frac": gbs / peak,
                     "traffic": None},
        "e2e": {"value": len(w) / float(np.mean(ts)), "unit": "volumes/s",
                "h2d_bytes_per_step": int(8 * n), "d2h_bytes_per_step": int(4 * len(w) * n),
                "seconds_per_call": float(np.mean(ts))},
    }
    if clk is not None:
        out_json["clocks"] = clk
    if not args.no_cpu_baseline:
        from oracle import dual_energy_oracle as deo

        m = n // 8   # a bounded sample: one eighth of the volume
        t0 = time.perf_counter()
        deo.subtract(he[:m], le[:m], w)
        dt = time.perf_counter() - t0
        out_json["cpu_baseline"] = {"value": len(w) * m / n / dt, "unit": "volumes/s", "cores": 1,
                                    "kind": "port",
                                    "sample": "NumPy restatement of syncrecon.m on 1/8 of the "
                                              "volumes, scaled"}
    print(json.dumps(out_json), flush=True)


def main():
    args = parse()
    if args.algo == "dual-energy":
        run_dual_energy(args)
        return
    if args.algo == "ossart":
        run_reference_ossart(args) if args.impl == "reference" else run_ossart(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
