#!/usr/bin/env python
"""Throughput benchmark of the B200 MHD step (GAMERA-OP single-domain path).

Workload: the 3-D Cartesian blast wave on a periodic 256^3 grid in FP64
(rho=1, p=0.1 with p=10 inside r<0.1 of the centre, v=0, uniform
B=(1/sqrt2,1/sqrt2,0), gamma=5/3, CFL 0.3).  One step is one AB2 time step of
the whole grid: CFL dt reduction, AB2 predictor, PDM reconstruction, Rusanov
fluxes, edge EMFs, constrained transport, update, ghost fill.  The metric is
cell-updates per second (active cells x steps / device time).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (launched by torchrun) every rank advances its own 256^3 replica
(the path does not shard: no collective on the data path), rank 0 prints the
whole-job rate over the max of the ranks' device times.  ``--impl reference``
times GAMERA-OP's own CPU solver (built from its sources into oracle/_ref) on
this host's cores on a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
for p in (ROOT / "gamera-op_b200", ROOT / "oracle"):
    sys.path.insert(0, str(p))

METRIC = "Mcell-updates/s vs plain FP64 GPU at fixed L1 err; %HBM peak; p50/p99 lat"
UNIT = "Mcell-updates/s"
BYTES_PER_CELL_UPDATE = 216  # algorithmic bytes of one cell-update (FP64)
REF_BUDGET_S = 120  # seconds of timed steps the reference arm may spend
# directions a group covers per step: the bytes and times below are of one
# direction (the three go out in one launch or three, by stage and grid)
GROUP_LAUNCHES = {"ab2": 1, "c2c": 3, "emf": 3, "flux": 3, "update": 1}
# the kernel a group's time is spent in on a large grid
GROUP_KERNEL = {"ab2": "k_ab2", "c2c": "k_c2c", "emf": "k_sweep", "flux": "k_sweep", "update": "k_update_sweep"}
# thread-block shapes the library's autotuner chooses from (gop_autotune)
BLOCK_CANDIDATES = ["32x4x2", "32x8x1", "32x1x8", "32x2x4", "64x2x2", "64x4x1", "64x1x4",
                    "128x2x1", "128x1x2", "32x4x1", "64x2x1", "256x1x1", "8x32x1", "8x4x8",
                    "tma_sweep"]  # index 14 (GOP_TUNE_SWEEP): the tile-staged sweep kernel


def peaks():
    try:
        m = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
        return float(m["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def algorithmic_bytes(group, n, mixed=False, ps_live=False):
    """Compulsory DRAM bytes of one direction of a kernel group (each input
    array element read once, each output written once).  Work arrays are
    FP32 on the mixed path (4 bytes), the state and its AB2 history FP64.
    ps_live False: the entropy channel p_S is identically zero (every
    problem measured here), and the step's kernels leave it out."""
    ni, nj, nk = n
    cells = ni * nj * nk
    ext = (ni + 9) * (nj + 9) * (nk + 9)
    w = 4 if mixed else 8  # element size of the work arrays
    g = 6 if ps_live else 5  # gas fields the step moves
    if group == "flux":   # per direction: Wh g, W g, mags_h 3, mags 3, B_n 1 in; g+3 fluxes, 2 edge velocities out
        return (3 * g + 12) * w * (cells + nj * nk)
    if group == "emf":    # per direction: 2 velocities, 2 B_h, 2 B, rho_h in; E out
        return 8 * w * cells
    if group == "c2c":    # per direction: 2 W_h, 2 W in; 2 edge velocities out (ghost layers)
        return 6 * w * (ni + 1) * 8 * nk
    if group == "update":  # W g, B 3 in and out (FP64); 3 (g+3) fluxes, 3 EMFs in
        return (2 * (g + 3) * 8 + (3 * (g + 3) + 3) * w) * cells
    if group == "ab2":    # W, W_old, B, B_old in (FP64); W_h, mags, mags_h, B_h out (+ W, B copies when mixed)
        return (2 * (g + 3) * 8 + (g + 9 + ((g + 3) if mixed else 0)) * w) * ext
    return 0


def fp64_flop_per_cell_update():
    """FP64 FLOP of one plain cell-update (2 per DFMA, 1 per DADD / DMUL,
    all step kernels) from the committed ncu summary, if any."""
    import re
    f = ROOT / "profiles" / "blast128_fp64_ops.md"
    if not f.exists():
        return None
    m = re.search(r"flop_per_cell_update_fp64=([\d.]+)", f.read_text())
    return float(m.group(1)) if m else None


def ncu_traffic(group, mixed=False):
    """DRAM bytes per launch from the committed ncu summary, if any."""
    import re
    f = ROOT / "profiles" / "blast256_launches.md"
    if not f.exists():
        return None
    key = "mixed" if mixed else "fp64"
    m = re.search(rf"^\|\s*{group}\s*\|.*?\|\s*traffic_per_launch_bytes_{key}=([\d.e+]+)", f.read_text(), re.M)
    return float(m.group(1)) if m else None


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        try:
            self.p = subprocess.Popen(
                ["nvidia-smi", "-i", str(gpu_index), f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None

    def stop(self):
        if self.p is None:
            return None
        self.p.terminate()
        try:
            self.p.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.p.kill()
        self.f.seek(0)
        rows = [r.split(",") for r in self.f.read().strip().splitlines() if r.count(",") >= 8]
        os.unlink(self.f.name)
        if not rows:
            return None
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[t] for r in rows for t in range(4) if "Active" in r[5 + t]
                          and "Not" not in r[5 + t]})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons, "samples": len(rows)}


def host_cores():
    """Physical cores of this host (logical CPUs when it cannot tell)."""
    try:
        seen = set()
        phys = core = None
        for line in open("/proc/cpuinfo"):
            if line.startswith("physical id"):
                phys = line.split(":")[1].strip()
            elif line.startswith("core id"):
                core = line.split(":")[1].strip()
                seen.add((phys, core))
        if seen:
            return len(seen)
    except OSError:
        pass
    return os.cpu_count() or 1


def cpu_model():
    """The host CPU's model name, as /proc/cpuinfo gives it."""
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                return line.split(":", 1)[1].strip()
    except OSError:
        pass
    return "unknown"


def rank_dims(cores, n):
    """The reference's process grid for about `cores` ranks: the largest
    power of two not above it, split over the axes as evenly as the grid
    divides (GAMERA-OP needs every axis divisible by its process count)."""
    r = 1
    while r * 2 <= max(1, cores):
        r *= 2
    dims = [1, 1, 1]
    a = 0
    while r > 1:
        for _ in range(3):
            if n[a] % (dims[a] * 2) == 0 and n[a] // (dims[a] * 2) >= 8:
                dims[a] *= 2
                r //= 2
                a = (a + 1) % 3
                break
            a = (a + 1) % 3
        else:
            break
    return tuple(dims)


def ref_bytes(n, dims):
    """Host memory of a reference run: about 268 doubles per ghost-extended
    point of every rank's block (its state, work and geometry arrays)."""
    pts = 1
    for a in range(3):
        pts *= n[a] // dims[a] + 9
    return 268 * 8 * pts * dims[0] * dims[1] * dims[2]


def mem_available():
    try:
        for line in open("/proc/meminfo"):
            if line.startswith("MemAvailable:"):
                return int(line.split()[1]) * 1024
    except OSError:
        pass
    return 0


def cpu_baseline(n=(128, 128, 128), steps=4):
    """GAMERA-OP's own solver on this host's cores in its README mode (one
    process of one thread per core), a bounded sample of the blast."""
    try:
        import ref_run
        if ref_run.available("cart", "release"):
            dims = rank_dims(host_cores(), n)
            ranks = dims[0] * dims[1] * dims[2]
            r = ref_run.run(n, steps + 1, problem="blast", flavor="release", keep_output=False,
                            threads=1, dims=dims, timeout=900,
                            env={"GOP_BC": "pppppp", "GOP_DOMAIN": "-0.5,0.5,-0.5,0.5,-0.5,0.5"})
            cells = n[0] * n[1] * n[2]
            v = cells * r.wall_steps / r.wall_seconds / 1e6
            return {"value": round(v, 4), "unit": UNIT, "cores": ranks, "kind": "reference",
                    "cpu": cpu_model(),
                    "sample": f"reference Release build, {ranks} ranks x 1 thread "
                              f"(process grid {dims[0]}x{dims[1]}x{dims[2]}), blast {n[0]}^3, "
                              f"{r.wall_steps} timed steps after 1"}
    except Exception:  # reference binary missing or failed: time the oracle port
        pass
    import oracle
    import gop
    m = 32
    x = [gop.grid_uniform(m, -0.5, 0.5) for _ in range(3)]
    W0, B0 = gop.problem_state((m,) * 3, x, gop.PROBLEM_BLAST)
    o = oracle.Oracle((m,) * 3, *x)
    o.set_state(W0, B0)
    o.prepare()
    t = time.perf_counter()
    o.run(4)
    dt = time.perf_counter() - t
    return {"value": round(m ** 3 * 4 / dt / 1e6, 4), "unit": UNIT, "cores": 1, "kind": "port",
            "sample": f"C restatement, blast {m}^3, 4 steps"}


def run_reference(args, rank):
    """GAMERA-OP's own CPU solver (Release build) on this host's cores in its
    README mode, mpirun -n N with one thread per rank, through the fork-based
    MPI stand-in: N = the host's physical cores (rounded down to a power of
    two that divides the grid), on the workload's own grid when the host has
    the memory for it."""
    if rank != 0:
        return
    import ref_run
    line = {"impl": "reference", "metric": METRIC, "unit": UNIT, "higher_is_better": True,
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup}
    if not ref_run.available("cart", "release"):
        line["unavailable"] = "reference binary oracle/_ref/ref_cart_release_* is not built"
        print(json.dumps(line))
        return
    full = (args.n,) * 3
    cores = host_cores()
    n, why = full, None
    need, avail = ref_bytes(full, rank_dims(cores, full)), mem_available()
    if avail and need > 0.8 * avail:
        n = (128, 128, 128)
        why = (f"host RAM: {args.n}^3 needs about {need / 2**30:.0f} GiB, "
               f"{avail / 2**30:.0f} GiB available")
    dims = rank_dims(cores, n)
    ranks = dims[0] * dims[1] * dims[2]
    cells = n[0] * n[1] * n[2]
    # a bounded sample of the K steps: about REF_BUDGET_S seconds of steps at
    # a conservative 0.4 M cell-updates/s per rank
    est = cells / (ranks * 0.4e6)
    steps = max(3, min(args.steps, int(REF_BUDGET_S / est)))
    r = ref_run.run(n, args.warmup + steps + 1, problem="blast", flavor="release",
                    keep_output=False, threads=1, dims=dims,
                    env={"GOP_SHIM_TIMING": "2", "GOP_BC": "pppppp",
                         "GOP_DOMAIN": "-0.5,0.5,-0.5,0.5,-0.5,0.5"}, timeout=3000)
    starts = r.step_starts
    w = args.warmup
    t = starts[w + steps] - starts[w]
    v = cells * steps / t / 1e6
    durs = np.diff(starts[w:w + steps + 1]) * 1e3
    cfg = {"workload": f"blast3d_periodic_{args.n}^3_{args.precision}",
           "grid": list(full),
           "problem": "blast p_in=10 p_out=0.1 r=0.1 B=(1/sqrt2,1/sqrt2,0) gamma=5/3 CFL=0.3",
           "ranks": ranks, "process_grid": list(dims), "threads_per_rank": 1,
           "cpu": cpu_model(), "host_physical_cores": cores,
           "mode": "mpirun -n N, OMP_NUM_THREADS=1 (the reference README's mode), "
                   "through the fork-based MPI stand-in"}
    if n != full:
        cfg["sample_grid"] = list(n)
        cfg["note"] = f"each step timed at {n[0]}^3 instead of {args.n}^3: {why}"
    cfg["timed_steps"] = steps
    line.update({
        "value": round(v, 4), "ms_per_step": round(t / steps * 1e3, 3),
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": cfg,
        "latency_ms": {"p50": round(float(np.percentile(durs, 50)), 3),
                       "p99": round(float(np.percentile(durs, 99)), 3)},
        "cpu_baseline": {"value": round(v, 4), "unit": UNIT, "cores": ranks, "kind": "reference",
                         "sample": f"blast {n[0]}^3, {steps} of the {args.steps} steps timed after "
                                   f"{w} warm-up, {ranks} ranks x 1 thread, Release flags"},
        "e2e": {"value": round(v, 4), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    })
    print(json.dumps(line))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=256)
    ap.add_argument("--precision", default="fp64", choices=["fp64", "mixed"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-mixed", action="store_true",
                    help="default workload: skip the mixed-precision run beside the FP64 one")
    ap.add_argument("--no-batched-sample", action="store_true",
                    help="default workload: skip the bounded batched sample")
    ap.add_argument("--no-ot-sample", action="store_true",
                    help="default workload: skip the Orszag-Tang run to t=0.5")
    ap.add_argument("--workload", default="blast256",
                    choices=["blast256", "batched", "served", "ot", "sphere"],
                    help="blast256: the single 256^3 grid (default); batched: 96 uneven "
                         "OT/blast grids in one batch; served: a Poisson request stream; "
                         "ot: Orszag-Tang 256x256x4 to t=0.5; sphere: field loop on a "
                         "192x128x128 spherical shell for one crossing")
    ap.add_argument("--requests", type=int, default=160, help="served: stream length")
    ap.add_argument("--rate", type=float, default=50.0,
                    help="served: mean arrivals per second (50: the configured stream, about "
                         "ten times one GPU's capacity; a few per second stays below it)")
    ap.add_argument("--members", type=int, default=96, help="batched: number of grids")
    ap.add_argument("--max-live", type=int, default=32, help="served: live request slots")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return

    import torch
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", local),
                                timeout=datetime.timedelta(seconds=300))

    def barrier():
        if dist is not None:
            dist.barrier()

    def max_all(v):
        if dist is None:
            return v
        t = torch.tensor([v], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    import gop
    if args.workload != "blast256":
        fn = {"batched": bench_batched, "served": bench_served, "ot": bench_ot,
              "sphere": bench_sphere}[args.workload]
        line = fn(args, gop, torch, dist, rank, world, local, max_all, barrier)
        if rank == 0:
            print(json.dumps(line))
        if dist is not None:
            dist.destroy_process_group()
        return
    n = (args.n,) * 3
    prec = gop.PREC_MIXED if args.precision == "mixed" else gop.PREC_FP64
    stream = torch.cuda.Stream()
    inst = gop.make(gop.PROBLEM_BLAST, n, precision=prec)
    inst.set_stream(stream.cuda_stream)
    inst.prepare()
    tuned = None if args.no_autotune else inst.autotune(reps=2)
    with torch.cuda.stream(stream):
        inst.step(args.warmup)
        torch.cuda.synchronize()
        clocks = ClockSampler(local)
        time.sleep(0.3)
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
        launches0 = gop.kernel_launches()
        barrier()
        torch.cuda.synchronize()
        evs[0].record(stream)
        for s in range(args.steps):  # each step one replay of the captured step graph
            inst.step(1, sync=False)
            evs[s + 1].record(stream)
        torch.cuda.synchronize()
        barrier()
        launches = gop.kernel_launches() - launches0
        clk = clocks.stop()
        # kernel shares and the dominant kernel's launch time: a separate
        # pass with CUDA events around every kernel group
        inst.set_profiling(True)
        for s in range(min(args.steps, 20)):
            inst.step(1, sync=False)
        torch.cuda.synchronize()
    ms = evs[0].elapsed_time(evs[-1])
    durs = np.array([evs[s].elapsed_time(evs[s + 1]) for s in range(args.steps)])
    prof = inst.profile()
    inst.set_profiling(False)
    st = inst.stats()
    ms_max = max_all(ms)
    cells = n[0] * n[1] * n[2]
    value = world * cells * args.steps / (ms_max / 1e3) / 1e6

    peak, peak_kind = peaks()
    step_s = ms / args.steps / 1e3
    step_gbs = BYTES_PER_CELL_UPDATE * cells / step_s / 1e9
    # dominant kernel group by device time
    groups = {g: v for g, v in prof.items() if g in GROUP_LAUNCHES}
    dom = max(groups, key=lambda g: groups[g][0])
    dom_ms, dom_cnt = groups[dom]
    per_launch_s = dom_ms / 1e3 / (dom_cnt * GROUP_LAUNCHES[dom])
    alg = algorithmic_bytes(dom, n, mixed=prec != 0)
    achieved = alg / per_launch_s / 1e9
    share = {g: round(v[0] / sum(x[0] for x in groups.values()), 4) for g, v in groups.items()}
    tr = ncu_traffic(dom, mixed=prec != 0)

    # the secondary bound: FP64 arithmetic against the measured FP64 peak
    fp64 = None
    if prec == gop.PREC_FP64:
        peak64 = gop.fp64_peak_tflops(stream.cuda_stream)
        flop = fp64_flop_per_cell_update()
        fp64 = {"peak_tflops": round(peak64, 2), "peak_kind": "measured (timed DFMA loop)",
                "flop_per_cell_update": flop}
        if flop:
            ach = value / world * 1e6 * flop / 1e12
            fp64.update({"achieved_tflops": round(ach, 3), "frac": round(ach / peak64, 4)})
    e2e = None
    if not args.no_e2e:
        e2e = measure_e2e(gop, torch, n, prec, args, max_all, barrier, world)
    # the metric's own comparison: the mixed path on the same grid and steps,
    # its rate against this plain FP64 rate and its error against this run
    mixed = None
    if prec == gop.PREC_FP64 and not args.no_mixed:
        mixed = measure_mixed(gop, torch, n, args, inst, value, max_all, barrier, world)
    batched = None
    if prec == gop.PREC_FP64 and not args.no_batched_sample:
        batched = batched_sample(args, gop, torch, dist, rank, world, local, max_all, barrier)
    ot = None
    if prec == gop.PREC_FP64 and not args.no_ot_sample:
        full = bench_ot(args, gop, torch, dist, rank, world, local, max_all, barrier)
        ot = {k: full[k] for k in ("value", "ms_per_step", "steps", "plain_fp64",
                                   "speedup_vs_plain_fp64", "accuracy_vs_fp64",
                                   "fp64_sensitivity")}
        ot["config"] = full["config"]

    line = {
        "metric": METRIC, "value": round(value, 3), "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(ms_max / args.steps, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64" if prec == 0 else "f32+f64",
        "data": "synthetic",
        "config": {"workload": f"blast3d_periodic_{args.n}^3_{args.precision}", "grid": list(n),
                   "problem": "blast p_in=10 p_out=0.1 r=0.1 B=(1/sqrt2,1/sqrt2,0) gamma=5/3 CFL=0.3",
                   "parallelism": f"replicas x{world} (no data-path collective)",
                   "l2": "state 2.4 GB per replica >> 126 MB L2, no flush needed",
                   "precision": args.precision,
                   "block_shapes": ({k: BLOCK_CANDIDATES[v] for k, v in tuned.items()} if tuned else "defaults"),
                   "launch_order": inst.launch_order()},
        "latency_ms": {"p50": round(float(np.percentile(durs, 50)), 4),
                       "p99": round(float(np.percentile(durs, 99)), 4)},
        "roofline": {"bound": "hbm", "kernel": GROUP_KERNEL[dom], "achieved": round(achieved, 2),
                     "peak": peak, "unit": "GB/s", "frac": round(achieved / peak, 4),
                     "traffic": tr, "peak_kind": peak_kind,
                     "algorithmic_bytes_per_launch": alg,
                     "avg_launch_ms": round(per_launch_s * 1e3, 4)},
        "step_roofline": {"bytes_per_cell_update": BYTES_PER_CELL_UPDATE,
                          "achieved_gbs": round(step_gbs, 2), "frac": round(step_gbs / peak, 4),
                          "fp64": fp64},
        "kernel_share": share,
        "gpu_launches": int(launches),
        "final_time": st["time"], "divb_max": st["divb_max"],
    }
    if clk:
        line["clocks"] = clk
    if e2e:
        line["e2e"] = e2e
    if mixed:
        line["mixed"] = mixed
    if batched:
        line["batched_sample"] = batched
    if ot:
        line["ot_to_t05"] = ot
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline()
    if rank == 0:
        print(json.dumps(line))
    inst.close()
    if dist is not None:
        dist.destroy_process_group()


def measure_mixed(gop, torch, n, args, plain, plain_value, max_all, barrier, world):
    """The mixed path (FP32 reconstruction, fluxes and EMFs; FP64 state,
    AB2, update and pressure recovery) on the same blast grid: K steps timed
    after W warm-up steps like the plain run, then stepped on to the plain
    instance's step count and compared with it variable by variable."""
    from gop import accuracy
    mx = gop.make(gop.PROBLEM_BLAST, n, precision=gop.PREC_MIXED)
    stream = torch.cuda.Stream()
    mx.set_stream(stream.cuda_stream)
    mx.prepare()
    if not args.no_autotune:
        mx.autotune(reps=2)
    with torch.cuda.stream(stream):
        mx.step(args.warmup)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier()
        torch.cuda.synchronize()
        a.record(stream)
        mx.step(args.steps, sync=False)
        b.record(stream)
        torch.cuda.synchronize()
        barrier()
    ms = max_all(a.elapsed_time(b))
    cells = n[0] * n[1] * n[2]
    value = world * cells * args.steps / (ms / 1e3) / 1e6
    steps_plain = plain.stats()["steps"]
    extra = steps_plain - mx.stats()["steps"]
    if extra > 0:
        mx.step(extra)
    which = ("gas", "face_b")
    errs = accuracy.rel_l1(n, mx.download(which), plain.download(which))
    worst, var = accuracy.worst(errs)
    st = mx.stats()
    mx.close()
    return {"value": round(value, 3), "unit": UNIT, "ms_per_step": round(ms / args.steps, 4),
            "ratio_vs_plain_fp64": round(value / plain_value, 3),
            "dtype": "f32 reconstruction/flux/EMF, f64 state/AB2/update/p recovery",
            "accuracy_vs_fp64": {"max_rel_l1": worst, "variable": var,
                                 "rel_l1": {k: float(f"{v:.3e}") for k, v in errs.items()},
                                 "steps": int(st["steps"]), "tolerance": 1e-5},
            "divb_max": st["divb_max"]}


def batched_sample(args, gop, torch, dist, rank, world, local, max_all, barrier):
    """A bounded sample of the batched workload inside the default run: the
    first 16 grids of the seeded 96-grid draw, 100 steps each, in one batch
    (mixed) against the same grids one at a time on the plain FP64 path."""
    import copy
    a = copy.copy(args)
    a.members, a.steps = 16, 100
    line = bench_batched(a, gop, torch, dist, rank, world, local, max_all, barrier)
    keep = ("value", "unit", "ms_per_step", "plain_fp64_one_at_a_time", "mixed_one_at_a_time",
            "speedup_vs_plain_fp64", "accuracy_vs_fp64")
    out = {k: line[k] for k in keep if k in line}
    out["config"] = {k: line["config"][k] for k in ("workload", "members", "grids", "cells",
                                                   "steps_per_member", "seed")}
    out["config"]["sample"] = "first 16 grids of the seeded draw of 96, 100 steps each"
    return out


def _accuracy(gop, n, got, want):
    """Largest per-variable relative L1 of a mixed result against FP64
    (vector components normalised by the vector's magnitude)."""
    from gop import accuracy
    return accuracy.worst(accuracy.rel_l1(n, got, want))


def bench_batched(args, gop, torch, dist, rank, world, local, max_all, barrier):
    """96 independent OT / blast grids of uneven size advanced in one batch
    (mixed precision) against the same grids run one at a time on the plain
    FP64 path (gop_step per grid); both with autotuned block shapes."""
    from collections import Counter
    from gop import serve, workloads
    jobs = workloads.batched_uneven(count=args.members, steps=args.steps)
    mine = serve.shard(jobs, rank, world)
    stream = torch.cuda.Stream()
    K, W = args.steps, args.warmup
    cells = sum(j.cells for j in mine)

    def timed(fn):
        barrier()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        fn()
        b.record(stream)
        torch.cuda.synchronize()
        barrier()
        return a.elapsed_time(b)

    # batched mixed path
    members = [workloads.build(j) for j in mine]
    batch = gop.Batch(members)
    batch.set_stream(stream.cuda_stream)
    tuned = batch.autotune(reps=2)
    batch.step([W] * len(members))
    launches0 = gop.kernel_launches()
    clocks = ClockSampler(local)
    ms_batch = timed(lambda: (batch.launch([K] * len(members)), batch.wait()))
    clk = clocks.stop()
    launches = gop.kernel_launches() - launches0

    def serial(prec):
        insts = [workloads.build(j, precision=prec) for j in mine]
        tb = gop.Batch(insts)  # only to give them the same per-class tuning
        tb.autotune(reps=2)
        tb.close()
        for i in insts:
            i.set_stream(stream.cuda_stream)
            i.step(W, sync=False)

        def go():
            for i in insts:
                i.step(K, sync=False)
        return insts, timed(go)

    fp64, ms_fp64 = serial(gop.PREC_FP64)
    worst, divb = (0.0, ""), 0.0
    for m, f, j in zip(members, fp64, mine):
        e = _accuracy(gop, j.n, m.download(("gas", "face_b")), f.download(("gas", "face_b")))
        worst = max(worst, e)
        divb = max(divb, m.stats()["divb_max"])
    for f in fp64:
        f.close()
    mixed1, ms_mixed1 = serial(gop.PREC_MIXED)
    for f in mixed1:
        f.close()
    batch.close()
    for m in members:
        m.close()
    ms_b, ms_f, ms_m = max_all(ms_batch), max_all(ms_fp64), max_all(ms_mixed1)
    total = sum(j.cells for j in jobs) * K
    rate = lambda ms: round(total / (ms / 1e3) / 1e6, 3)
    return {
        "metric": METRIC, "value": rate(ms_b), "unit": UNIT, "n_gpus": world, "steps": K,
        "warmup": W, "ms_per_step": round(ms_b / K, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
        "config": {"workload": f"batched_uneven_{len(jobs)}_mixed", "members": len(jobs),
                   "grids": {"x".join(map(str, k)): v for k, v in sorted(Counter(j.n for j in jobs).items())},
                   "cells": sum(j.cells for j in jobs), "steps_per_member": K, "seed": 20261203,
                   "parallelism": f"members sharded over {world} GPU(s), no data-path collective",
                   "l2": "states total tens of GB >> 126 MB L2, no flush needed",
                   "block_shapes": {k: BLOCK_CANDIDATES[v] for k, v in tuned.items()}},
        "plain_fp64_one_at_a_time": {"value": rate(ms_f), "ms": round(ms_f, 3)},
        "mixed_one_at_a_time": {"value": rate(ms_m), "ms": round(ms_m, 3)},
        "speedup_vs_plain_fp64": round(ms_f / ms_b, 3),
        "accuracy_vs_fp64": {"max_rel_l1": worst[0], "variable": worst[1], "max_divb": divb,
                             "tolerance": 1e-5},
        "gpu_launches": int(launches), "clocks": clk,
    }


def bench_served(args, gop, torch, dist, rank, world, local, max_all, barrier):
    """A Poisson request stream served with continuous batching (mixed
    precision, HBM budget admission) against a one-request-at-a-time plain
    FP64 loop on the same requests; latency is time-to-solution."""
    from collections import Counter
    from gop import serve, workloads
    jobs = workloads.served_stream(count=args.requests, rate=args.rate)
    mine = serve.shard(jobs, rank, world)
    sample = lambda j: j.rid % 8 == 0
    # warm the kernels and the allocator on a small request
    warm = workloads.Job(-1, gop.PROBLEM_BLAST, (32, 32, 32), 10, domain=workloads._domain(2, (32, 32, 32)))
    w_eng = serve.GpuEngine()
    serve.Server(w_eng, 150 * 10 ** 9).run([warm])
    w_eng.close()
    eng = serve.GpuEngine(keep=sample)
    barrier()
    launches0 = gop.kernel_launches()
    clocks = ClockSampler(local)
    rep = serve.Server(eng, 150 * 10 ** 9, max_live=args.max_live, chunk=50,
                       workers=4).run(mine)
    clk = clocks.stop()
    launches = gop.kernel_launches() - launches0
    eng.close()
    served = serve.combine(rep, dist)
    pool = {}
    kept = {o.rid: o.result for o in rep.outcomes if o.rid % 8 == 0}
    worst, divb = (0.0, ""), 0.0

    def run_one(j):
        inst = workloads.build(j, precision=gop.PREC_FP64, device_init=True)
        inst.step(j.steps)
        res = serve.download_result(inst, pool, copy=j.rid in kept)
        inst.close()
        return res

    span = max(j.arrival for j in jobs) - min(j.arrival for j in jobs)
    offered = sum(j.cells * j.steps for j in jobs) / max(span, 1e-9) / 1e6
    base_rep = serve.serial(mine, run_one)
    base = serve.combine(base_rep, dist)
    for o in base_rep.outcomes:
        if o.rid in kept:
            worst = max(worst, _accuracy(gop, next(j.n for j in mine if j.rid == o.rid),
                                         kept[o.rid], o.result))
            divb = max(divb, kept[o.rid]["divb_max"])
    return {
        "metric": METRIC, "value": round(served["mcell_updates_per_s"], 3), "unit": UNIT,
        "n_gpus": world, "steps": sum(j.steps for j in jobs), "warmup": 1,
        "ms_per_step": None, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32+f64", "data": "synthetic",
        "config": {"workload": f"served_poisson{args.rate:g}_{len(jobs)}req_mixed",
                   "requests": len(jobs), "rate_per_s": args.rate, "seed": 5150,
                   "grids": {"x".join(map(str, k)): v for k, v in sorted(Counter(j.n for j in jobs).items())},
                   "steps": "uniform [100, 1000]", "hbm_budget_gb": 150, "max_live": args.max_live,
                   "round_steps": 50, "host_workers": 4, "tolerance": 1e-5,
                   "parallelism": f"requests sharded over {world} GPU(s), no data-path collective",
                   "l2": "live states >> 126 MB L2"},
        "latency_s": {"p50": round(served["p50_s"], 3), "p99": round(served["p99_s"], 3),
                      "what": "time-to-solution: arrival to result on the host"},
        "load": {"offered_mcell_updates_per_s": round(offered, 3),
                 "utilisation": round(offered / served["mcell_updates_per_s"], 3),
                 "what": "work of the stream over its arrival span, against the served "
                         "throughput (above 1: requests queue for the GPU)"},
        "served": {k: (round(v, 4) if isinstance(v, float) else v) for k, v in served.items()},
        "plain_fp64_one_at_a_time": {k: (round(v, 4) if isinstance(v, float) else v) for k, v in base.items()},
        "speedup_vs_plain_fp64": round(served["mcell_updates_per_s"] / base["mcell_updates_per_s"], 3),
        "rounds": rep.rounds, "peak_live": rep.peak_live, "peak_bytes": rep.peak_bytes,
        "host_seconds": {k: round(v, 3) for k, v in rep.seconds.items()},
        "engine": {k: (round(v, 3) if isinstance(v, float) else v) for k, v in eng.stats.items()},
        "accuracy_vs_fp64": {"max_rel_l1": worst[0], "variable": worst[1], "max_divb": divb,
                             "sampled_requests": len(kept), "tolerance": 1e-5},
        "gpu_launches": int(launches), "clocks": clk,
    }


def _run_to(gop, torch, inst, steps, time_stop):
    """Advances an instance on a fresh stream, timed with CUDA events;
    returns (device ms, steps taken)."""
    stream = torch.cuda.Stream()
    inst.set_stream(stream.cuda_stream)
    s0 = inst.stats()["steps"]
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    a.record(stream)
    inst.step(steps, time_stop=time_stop, sync=False)
    b.record(stream)
    torch.cuda.synchronize()
    return a.elapsed_time(b), inst.stats()["steps"] - s0


def _perturbed(gop, make, rel=1e-15, seed=7):
    """An FP64 instance whose initial density differs from make()'s by a
    seeded relative perturbation of about `rel` per cell (round-off level)."""
    inst = make(gop.PREC_FP64)
    d = inst.download(("gas", "face_b"))
    rng = np.random.default_rng(seed)
    gas = d["gas"].copy()
    gas[0] *= 1.0 + rel * rng.uniform(-1.0, 1.0, size=gas[0].shape)
    inst.upload(gas, d["face_b"])
    return inst


def _single_pair(args, gop, torch, local, make, n, t_end, workload, extra):
    """FP64 to t_end, then the mixed path for the same number of steps; the
    mixed result is compared with the FP64 one.  A third run, FP64 again from
    an initial density perturbed at round-off level (1e-15 relative), shows
    how far two FP64 solutions of the same problem drift apart by then: the
    floor below which the mixed path's error is the problem's sensitivity,
    not its precision."""
    from gop import accuracy
    warm = make(gop.PREC_FP64)
    warm.prepare()
    warm.step(max(args.warmup, 3))
    warm.close()
    launches0 = gop.kernel_launches()
    clocks = ClockSampler(local)
    f64 = make(gop.PREC_FP64)
    f64.prepare()
    ms64, steps = _run_to(gop, torch, f64, 10 ** 8, t_end)
    mx = make(gop.PREC_MIXED)
    mx.prepare()
    msmx, steps_mx = _run_to(gop, torch, mx, steps, 1e300)
    clk = clocks.stop()
    launches = gop.kernel_launches() - launches0
    cells = n[0] * n[1] * n[2]
    which = ("gas", "face_b", "mags")
    a, b = mx.download(which), f64.download(which)
    errs = accuracy.rel_l1(n, a, b)
    pt = _perturbed(gop, make)
    pt.prepare()
    _run_to(gop, torch, pt, steps, 1e300)
    c = pt.download(which)
    errs_pt = accuracy.rel_l1(n, c, b)
    sl = tuple(slice(4, 4 + m) for m in n)
    bm = lambda d: np.sqrt(sum(d["mags"][k][sl] ** 2 for k in range(3)))
    ba, bb, bc = bm(a), bm(b), bm(c)
    l1_bmag = float(np.abs(ba - bb).sum() / max(np.abs(bb).sum(), 1e-300))
    l1_bmag_pt = float(np.abs(bc - bb).sum() / max(np.abs(bb).sum(), 1e-300))
    st64, stmx = f64.stats(), mx.stats()
    rate = lambda ms, k: round(cells * k / (ms / 1e3) / 1e6, 3)
    line = {
        "metric": METRIC, "value": rate(msmx, steps_mx), "unit": UNIT, "n_gpus": 1,
        "steps": steps, "warmup": max(args.warmup, 3), "ms_per_step": round(msmx / steps_mx, 4),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
        "data": "synthetic",
        "config": dict(workload=workload, grid=list(n), t_end=t_end,
                       l2="state >> 126 MB L2" if cells >= 2 ** 20 else "state fits L2 (small grid)",
                       **extra),
        "plain_fp64": {"value": rate(ms64, steps), "ms_per_step": round(ms64 / steps, 4),
                       "time": st64["time"], "divb_max": st64["divb_max"]},
        "speedup_vs_plain_fp64": round(rate(msmx, steps_mx) / rate(ms64, steps), 3),
        "accuracy_vs_fp64": {"rel_l1": errs, "l1_bmag": l1_bmag, "l1_rho": errs["rho"],
                             "max_divb_mixed": stmx["divb_max"], "time_mixed": stmx["time"],
                             "tolerance": 1e-5},
        "fp64_sensitivity": {"what": "FP64 from a 1e-15 relative density perturbation vs FP64",
                             "rel_l1": errs_pt, "l1_bmag": l1_bmag_pt, "l1_rho": errs_pt["rho"]},
        "gpu_launches": int(launches), "clocks": clk,
    }
    f64.close()
    mx.close()
    pt.close()
    return line


def bench_ot(args, gop, torch, dist, rank, world, local, max_all, barrier):
    """Orszag-Tang vortex, 256x256x4 periodic, FP64 to t = 0.5 (the last
    step overshoots, as in the reference), mixed for the same steps."""
    n = (256, 256, 4)
    make = lambda prec: gop.make(gop.PROBLEM_OT, n, domain=(0, 1, 0, 1, 0, 1 / 64), precision=prec)
    line = _single_pair(args, gop, torch, local, make, n, 0.5, "orszag_tang_256x256x4_to_t0.5",
                        {"problem": "OT rho=25/(36pi) p=5/(12pi) gamma=5/3 CFL=0.3"})
    # through the C ABI with host buffers, plain FP64: the drop-in's pattern
    e2e = measure_e2e(gop, torch, n, gop.PREC_FP64, args, max_all, barrier, world,
                      problem=gop.PROBLEM_OT, t_end=0.5)
    e2e["vs_device_plain_fp64"] = round(e2e["value"] / line["plain_fp64"]["value"], 3)
    line["plain_fp64"]["e2e"] = e2e
    return line


def bench_sphere(args, gop, torch, dist, rank, world, local, max_all, barrier):
    """Field loop advected through a pole-free spherical shell r in [1,2],
    theta in [pi/4, 3pi/4], phi in [-pi/4, pi/4], 192x128x128, outflow: FP64
    for one crossing (t = 2.1), mixed for the same steps."""
    n = (192, 128, 128)
    make = lambda prec: gop.make(gop.PROBLEM_LOOP_SPH, n, bc="eeeeee", precision=prec)
    return _single_pair(args, gop, torch, local, make, n, 2.1, "field_loop_sphere_192x128x128_one_crossing",
                        {"problem": "loop R=0.15 at (1.5,0,0), A0=1e-3, v=(0,1,0.5), rho=1 p=1"})


def measure_e2e(gop, torch, n, prec, args, max_all, barrier, world, problem=None, t_end=None):
    """The drop-in solve() pattern through the C ABI with host buffers:
    upload the state from pinned memory, prepare, step on the device up to
    the next host event with the simulated time read back there (no dump or
    log falls inside a benchmark run, so one gop_step of K steps, or to
    t_end), download the final state to pinned memory."""
    problem = gop.PROBLEM_BLAST if problem is None else problem
    lo, hi = (-0.5, 0.5) if problem == gop.PROBLEM_BLAST else (0.0, 1.0)
    xs = [gop.grid_uniform(m, lo, hi) for m in n]
    if problem == gop.PROBLEM_OT:
        xs[2] = gop.grid_uniform(n[2], 0.0, 1.0 / 64)
    gas0, fb0 = gop.problem_state(n, xs, problem)
    N = tuple(v + 9 for v in n)
    pin = lambda shape: torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()
    h_gas, h_fb = pin((6,) + N), pin((3,) + N)
    h_gas[...] = gas0
    h_fb[...] = fb0
    o_gas, o_fb = pin((6,) + N), pin((3,) + N)
    inst = gop.Instance(n, *xs, precision=prec)
    stream = torch.cuda.Stream()
    inst.set_stream(stream.cuda_stream)
    # one untimed pass warms the allocator and the kernels
    inst.upload(h_gas, h_fb)
    inst.prepare()
    inst.step(args.warmup)
    barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    inst.upload(h_gas, h_fb)
    inst.prepare()
    if t_end is None:
        inst.step(args.steps, sync=True)
    else:
        inst.step(10 ** 8, time_stop=t_end, sync=True)
    inst.download(("gas", "face_b"), out={"gas": o_gas, "face_b": o_fb})
    torch.cuda.synchronize()
    t = time.perf_counter() - t0
    steps = inst.stats()["steps"]
    barrier()
    t = max_all(t)
    inst.close()
    cells = n[0] * n[1] * n[2]
    state_bytes = 9 * N[0] * N[1] * N[2] * 8
    return {"value": round(world * cells * steps / t / 1e6, 3), "unit": UNIT,
            "h2d_bytes_per_step": int(state_bytes / steps),
            "d2h_bytes_per_step": int(state_bytes / steps + 11 * 8),
            "steps": int(steps),
            "pattern": "upload(pinned) + prepare + gop_step to the next host event (time read "
                       "back there) + download(pinned)"}


if __name__ == "__main__":
    main()
