#!/usr/bin/env python
"""Benchmark of the FDTD time-step engine on the 2D TMz workload.

Workload (default): 2D TMz, 2048 x 2048 cells, dx = 1 nm, Courant 0.5,
32-cell split-field PML on all faces, 40 seeded gold cylinders (Drude +
2 critical points), Ez line source at y=100 (600 nm pulse), line DFT monitors
of Ez and Hx at y=200 (incident / reflected, gated) and y=1948 (transmitted)
with 100 frequencies, 10000 time steps.  Synthetic, seeded geometry.

One bench "step" is one whole job of that workload (10000 time steps from
a fresh state) with its inputs already resident in HBM.  The headline value
is Mcell-updates/s of the FP32 path (FP64 DFT accumulation); the FP64 plain
path, the FP32/FP64 ratio and the FP32 DFT error against the FP64 path are
reported beside it, with the dominant kernel's roofline, an end-to-end
figure through the C ABI with host buffers, and a CPU baseline (the FP64
oracle on the host cores).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
import argparse
import json
import math
import os
import re
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "fortran-mpi-fdtd_gb300")
for _p in (ROOT, PKG):
    if _p not in sys.path:
        sys.path.insert(0, _p)

METRIC = "Mcell-updates/s FP32 vs FP64 plain at <=1e-4 DFT rel err; serve p50/p99 latency"
UNIT = "Mcell-updates/s"
L2_FLUSH_BYTES = 512 << 20


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--nt", type=int, default=10000, help="time steps per job")
    ap.add_argument("--n", type=int, default=2048, help="grid cells per side")
    ap.add_argument("--fp64-steps", type=int, default=3)
    ap.add_argument("--cpu-child", action="store_true", help=argparse.SUPPRESS)
    ap.add_argument("--cpu-threads", type=int, default=0, help=argparse.SUPPRESS)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-configs", action="store_true", help="skip the 3D, graphene and 1D runs")
    ap.add_argument("--serve-jobs", type=int, default=200, help="jobs per arrival rate of the serving sweep (0: none)")
    ap.add_argument("--serve-rates", default="4,8,16,32", help="Poisson arrival rates of the sweep, jobs/s")
    ap.add_argument("--serve-arms-jobs", type=int, default=48,
                    help="jobs of each of the served/sequential x FP32/FP64 arms (0: none)")
    ap.add_argument("--serve-arms-rate", type=float, default=16.0, help="arrival rate of the arms, jobs/s")
    return ap.parse_args()


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)), int(os.environ.get("LOCAL_RANK", 0))


def max_over_ranks(x, device, world):
    """The largest x over all ranks: a replicated job's time is its slowest
    replica's."""
    if world <= 1:
        return float(x)
    import torch
    import torch.distributed as dist
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def aggregate_mcells(world, cells, steps, seconds):
    """Whole-job Mcell-updates/s: every replica updates `cells` cells for
    `steps` time steps in `seconds` (the slowest replica's time)."""
    return world * cells * steps / seconds / 1e6


def workload(n, nt, precision):
    from fdtd_gpu import problems
    spec, meta = problems.config_2d_tmz(precision=precision, n=n, steps=nt)
    return spec, meta


def workload_name(n, nt):
    return f"2d_tmz_{n}x{n}_40cyl_splitpml32_{nt}steps"


# ---- bytes each kernel must move per cell (FP32 / FP64 word size w) --------
# E kernel: read Hx, Hy, Ez, material id; write Ez        -> 4w + 1
# H kernel: read Ez, Hx, Hy; write Hx, Hy                  -> 5w
# whole step, each field read and written once (+ id)      -> 6w + 1
def alg_bytes(kind, w):
    return {"E": 4 * w + 1, "H": 5 * w, "step": 6 * w + 1}[kind]


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def profile_traffic(kernel):
    """dram bytes per launch from the committed ncu summary, if present."""
    name = {"STEP": "step2d_block"}.get(kernel, kernel)
    path = os.path.join(ROOT, "profiles", f"{name}_2d_tmz.md")
    try:
        txt = open(path).read()
    except OSError:
        return None, None
    m = re.search(r"traffic_bytes_per_full_launch:\s*([0-9.eE+]+)", txt)
    return (float(m.group(1)) if m else None), os.path.relpath(path, ROOT)


class Clocks:
    """nvidia-smi sampler for the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-i", str(self.index), "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.t.join(timeout=2)
        sm, smax, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = max(smax, float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": smax, "reasons": sorted(reasons),
                "samples": len(sm)}


def dft_rel_err(ja, jb, nmon):
    """Relative L2 distance of job a's monitor sums from job b's, over all
    monitors together."""
    import numpy as np
    num = den = 0.0
    for q in range(nmon):
        ra, ia = ja.get_monitor(q)
        rb, ib = jb.get_monitor(q)
        num += float(np.sum((ra - rb) ** 2) + np.sum((ia - ib) ** 2))
        den += float(np.sum(rb ** 2) + np.sum(ib ** 2))
    return math.sqrt(num / den) if den > 0 else float("nan")


def pml_cells_by_axes(spec):
    """Cells of a split-PML grid inside the PML of exactly one axis, and of
    two or three."""
    npml = (spec.pml or {}).get("npml", ((0, 0),) * 3)
    inside, outside = [], []
    for a in range(3):
        n = spec.n[a]
        lo, hi = (0, 0) if spec.periodic[a] or n == 1 else npml[a]
        inside.append(lo + hi)
        outside.append(n - lo - hi)
    (ax, ay, az), (bx, by, bz) = inside, outside
    one = ax * by * bz + bx * ay * bz + bx * by * az
    total = spec.cells() - bx * by * bz
    return one, total - one


def config_runs(stream):
    """The other named configurations.  The 3D ones run their whole length
    in FP32 and in FP64 plain (timed with CUDA events on the bench stream
    after a short warm-up), so that the FP32 spectra can be compared with the
    FP64 ones of the same run: Mcell-updates/s, the FP32 DFT error, and the
    step's ideal bytes (each field read and written once, plus the material
    id: 12w+1 per cell in 3D, 4w+1 in 1D) over the measured HBM peak; in 3D
    also the step's algorithmic bytes with the split-PML shell's stored parts
    (in FP32 8w more per cell inside one axis's PML and 12w inside more, 24w
    in FP64) over the same peak."""
    import torch
    from fdtd_gpu import abi, problems
    from fdtd_gpu.job import Job
    peak, _ = measured_peaks()

    def timed(spec, warm, k, per_cell, keep=False, shell=False):
        J = Job(spec)
        J.set_stream(stream.cuda_stream)
        J.step(1, warm)
        J.sync()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        J.step(warm + 1, k)
        J.sync()
        b.record(stream)
        torch.cuda.synchronize()
        ms = a.elapsed_time(b)
        mc = spec.cells() * k / (ms / 1e3) / 1e6
        w = 4 if spec.precision == abi.F32 else 8
        r = {"mcell_updates_per_s": mc, "ms_per_step": ms / k, "timed_steps": k, "tile": J.tile(),
             "step_bytes_frac_of_hbm": mc * 1e6 * per_cell(w) / (peak * 1e9)}
        if shell:
            # the split-PML shell (cells outside the interior box) also reads
            # and writes its stored parts: in FP64 12 per cell; in FP32 one per
            # component that has a PML axis among its two curl axes, so 4 for a
            # cell inside one axis's PML and 6 inside two or three
            nshell = spec.cells() - J.kernel_cells(abi.KERNEL_E)
            n1, n2 = pml_cells_by_axes(spec)
            extra = (4 * n1 + 6 * n2) * 2 * w if w == 4 else (n1 + n2) * 24 * w
            alg = spec.cells() * per_cell(w) + extra
            r["shell_cells"] = nshell
            r["pml_cells_one_axis"], r["pml_cells_more_axes"] = n1, n2
            r["step_alg_bytes"] = alg
            r["step_alg_bytes_frac_of_hbm"] = alg / (ms / k / 1e3) / (peak * 1e9)
        if keep:
            return r, J
        J.close()
        return r

    out = {}
    for name, make, nmon in (("3d_sphere_512^3_splitpml16_64freq", problems.config_3d_sphere, 6),
                             ("3d_graphene_256x256x384_pmlz10_128freq", problems.config_3d_graphene, 1)):
        s32, meta = make(precision=abi.F32)
        s64, _ = make(precision=abi.F64)
        nt, warm = meta["Nt"], 64
        r32, j32 = timed(s32, warm, nt - warm, lambda w: 12 * w + 1, keep=True, shell=True)
        r64, j64 = timed(s64, warm, nt - warm, lambda w: 12 * w + 1, keep=True, shell=True)
        out[name] = {"fp32": r32, "fp64_plain": r64, "time_steps": nt,
                     "fp32_over_fp64": r32["mcell_updates_per_s"] / r64["mcell_updates_per_s"],
                     "dft_rel_err_fp32_vs_fp64": dft_rel_err(j32, j64, nmon)}
        j32.close()
        j64.close()
    o32, _ = problems.config_1d_gold(precision=abi.F32)
    o64, _ = problems.config_1d_gold(precision=abi.F64)
    l32, l64 = timed(o32, 2000, 18000, lambda w: 4 * w + 1), timed(o64, 2000, 18000, lambda w: 4 * w + 1)
    for r in (l32, l64):
        r["steps_per_s"] = 1e3 / r["ms_per_step"]
        r["note"] = "4000 cells: a launch per 32 steps (FP64: 16), latency-bound; the roofline does not apply"
    out["1d_gold_slab_4000"] = {"fp32": l32, "fp64_plain": l64}
    return out


def serve_served(mix):
    """The mix through the library's server (continuous batching, HBM
    admission, packs of small 2D jobs, graph rings): jobs/s, p50/p99 latency
    and the pack statistics."""
    from fdtd_gpu import serve
    S = serve.Server(max_active=16, chunk_steps=256)
    lat, wall = serve.run_mix(S, mix)
    st = S.stats()
    S.close()
    cells = sum(sp.cells() * nst for _, sp, nst in mix)
    return {"jobs": len(mix), "jobs_per_s": len(mix) / wall, "p50_s": serve.percentile(lat, 50),
            "p99_s": serve.percentile(lat, 99), "wall_s": wall, "mcell_updates_per_s": cells / wall / 1e6,
            "hbm_held_max_bytes": st["held_bytes_max"], "packed_rings": st["packed_rings"],
            "pack_builds": st["pack_builds"], "pack_build_s": st["pack_build_s"]}


def serve_sequential(mix):
    """The same arrivals run one job at a time through the plain job API
    (each job created, stepped and its spectra read before the next one)."""
    from fdtd_gpu import serve
    from fdtd_gpu.job import Job
    t0 = time.perf_counter()
    lat = []
    for ta, spec, nst in mix:
        idle = ta - (time.perf_counter() - t0)
        if idle > 0:
            time.sleep(idle)
        J = Job(spec)
        J.step(1, nst)
        for q in range(len(spec.monitors)):
            J.get_monitor(q)
        J.close()
        lat.append(time.perf_counter() - t0 - ta)
    wall = time.perf_counter() - t0
    cells = sum(sp.cells() * nst for _, sp, nst in mix)
    return {"jobs": len(mix), "jobs_per_s": len(mix) / wall, "p50_s": serve.percentile(lat, 50),
            "p99_s": serve.percentile(lat, 99), "wall_s": wall, "mcell_updates_per_s": cells / wall / 1e6}


def serving_run(njobs, rates, arms_jobs, arms_rate):
    """The serving workload: seeded Poisson arrivals of 2D TMz and 3D sphere
    jobs.  For each arrival rate, `njobs` jobs served in FP32; at `arms_rate`,
    `arms_jobs` jobs in four arms -- served and one-at-a-time, each in FP32
    and in FP64 plain -- so that the gain of batching (served vs sequential
    at one precision) is apart from the gain of precision."""
    from fdtd_gpu import abi, serve
    out = {"workload": "Poisson arrivals, numpy default_rng(1): 80% 2D TMz N in {256,512,1024} with 1-20 "
                       "cylinders, 20% 3D spheres N in {128,192,256}; 2000-8000 steps, 32-128 frequencies",
           "latency": "host time from submission (at the Poisson arrival time) to the job's completion",
           "server": {"max_active": 16, "chunk_steps": 256}, "sweep_fp32": []}
    for rate in rates:
        r = serve_served(serve.poisson_mix(njobs, rate, seed=1))
        r["rate_per_s"] = rate
        out["sweep_fp32"].append(r)
    if arms_jobs > 0:
        m32 = serve.poisson_mix(arms_jobs, arms_rate, seed=1)
        m64 = serve.poisson_mix(arms_jobs, arms_rate, seed=1, precision=abi.F64)
        out["arms"] = {"rate_per_s": arms_rate, "jobs": arms_jobs,
                       "served_fp32": serve_served(m32), "sequential_fp32": serve_sequential(m32),
                       "served_fp64_plain": serve_served(m64), "sequential_fp64_plain": serve_sequential(m64)}
        a = out["arms"]
        a["batching_gain_fp32"] = a["served_fp32"]["jobs_per_s"] / a["sequential_fp32"]["jobs_per_s"]
        a["batching_gain_fp64"] = a["served_fp64_plain"]["jobs_per_s"] / a["sequential_fp64_plain"]["jobs_per_s"]
    return out


CPU_SAMPLE_STEPS = 200  # time steps of the workload in one timed CPU sample


def cpu_child(args):
    """Child process of cpu_measure: the FP64 oracle on the host cores, the
    OpenMP threads pinned (OMP_PROC_BIND=close, OMP_PLACES=cores, set by the
    parent before the runtime starts).  Memory is first touched and the
    thread team started by a few untimed steps; then `warm` untimed and `k`
    timed samples of CPU_SAMPLE_STEPS steps each, from one running state.
    Prints one JSON line: the sample times."""
    from fdtd_gpu import abi
    from oracle.pyoracle import OracleJob, build
    build()
    spec, _ = workload(args.n, 10000, abi.F64)
    O = OracleJob(spec, nthreads=args.cpu_threads)
    n = 1
    O.step(n, 4)
    n += 4
    times = []
    for r in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        O.step(n, CPU_SAMPLE_STEPS)
        dt = time.perf_counter() - t0
        n += CPU_SAMPLE_STEPS
        if r >= args.warmup:
            times.append(dt)
    print(json.dumps({"times": times, "cells": spec.cells()}), flush=True)
    return 0


def cpu_measure(n, warm, k):
    """The CPU baseline, the same measurement for the GPU line's
    cpu_baseline and for the reference arm: the FP64 oracle (the reference's
    algorithm restated in C; the Fortran/MPI reference cannot be built
    without gfortran and MPI) on all host cores with pinned threads, the
    median of k samples of CPU_SAMPLE_STEPS time steps of the n x n workload
    after `warm` untimed ones.  Runs in a child process, so that the OpenMP
    runtime starts with the pinning settings and without the GPU process's
    threads."""
    nth = os.cpu_count() or 1
    env = dict(os.environ, OMP_PROC_BIND="close", OMP_PLACES="cores", OMP_NUM_THREADS=str(nth))
    cmd = [sys.executable, os.path.abspath(__file__), "--cpu-child", "--n", str(n), "--warmup", str(warm),
           "--steps", str(k), "--cpu-threads", str(nth)]
    out = subprocess.run(cmd, env=env, capture_output=True, text=True, check=True).stdout
    d = json.loads(out.strip().splitlines()[-1])
    med = statistics.median(d["times"])
    value = d["cells"] * CPU_SAMPLE_STEPS / med / 1e6
    spread = (max(d["times"]) - min(d["times"])) / med
    return {"value": value, "unit": UNIT, "cores": nth, "kind": "port",
            "sample": f"FP64 oracle (the reference's algorithm in C; the Fortran/MPI reference needs gfortran and "
                      f"MPI, absent on this box), median of {k} samples of {CPU_SAMPLE_STEPS} time steps of the "
                      f"{n}x{n} workload after {warm} untimed, {nth} threads pinned "
                      f"(OMP_PROC_BIND=close, OMP_PLACES=cores)",
            "sample_seconds": d["times"], "spread": spread}


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    cb = cpu_measure(args.n, args.warmup, args.steps)
    value = cb["value"]
    ms = 1e3 * statistics.median(cb["sample_seconds"])
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": workload_name(args.n, args.nt),
                                            "note": f"each bench step = a sample of {CPU_SAMPLE_STEPS} time steps "
                                                    f"of the workload (the median sample is reported)"},
            "cpu_baseline": cb,
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def main():
    args = parse()
    if args.cpu_child:
        return cpu_child(args)
    if args.impl == "reference":
        return run_reference(args)
    import numpy as np
    import torch
    from fdtd_gpu import abi
    from fdtd_gpu import job as gj

    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local)
    flush = torch.empty(L2_FLUSH_BYTES, dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream(dev)

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    def timed_jobs(precision, k, warm):
        spec, meta = workload(args.n, args.nt, precision)
        jobs = [gj.Job(spec) for _ in range(warm + k)]
        for j in jobs:
            j.set_stream(stream.cuda_stream)
        for j in jobs[:warm]:
            flush.zero_()
            j.step(1, args.nt)
            j.sync()
        barrier()
        torch.cuda.synchronize()
        evs = []
        launches0 = sum(j.launch_count() for j in jobs[warm:])
        clk = Clocks(local)
        clk.start()
        for j in jobs[warm:]:
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            j.step(1, args.nt)
            j.sync()  # folds the last DFT ring
            b.record(stream)
            evs.append((a, b))
        torch.cuda.synchronize()
        clocks = clk.stop()
        barrier()
        ms = [a.elapsed_time(b) for a, b in evs]
        launches = sum(j.launch_count() for j in jobs[warm:]) - launches0
        # per-kernel device time: the same job once more with an event pair
        # around every launch (eager launches; the timed jobs replay graphs)
        pj = gj.Job(spec)
        pj.set_stream(stream.cuda_stream)
        pj.profile(True)
        flush.zero_()
        pj.step(1, args.nt)
        pj.sync()
        kt = {}
        for kind, name in ((abi.KERNEL_E, "E"), (abi.KERNEL_H, "H"), (abi.KERNEL_EDGE, "EDGE"),
                           (abi.KERNEL_ADE, "ADE"), (abi.KERNEL_DFT, "DFT"), (abi.KERNEL_STEP, "STEP")):
            kt[name] = pj.kernel_time(kind) + (pj.kernel_cells(kind),)
        tile = pj.tile()
        pj.close()
        return spec, meta, jobs[warm:], ms, launches, kt, clocks, tile

    # ---- FP32 (headline) ----
    spec32, meta, jobs32, ms32, launches, kt32, clocks, tile32 = timed_jobs(abi.F32, args.steps, args.warmup)
    t_step = max(ms32) if False else sum(ms32) / len(ms32)
    t_step = max_over_ranks(t_step, dev, world)
    cells = spec32.cells()
    value = aggregate_mcells(world, cells, args.nt, t_step / 1e3)

    # ---- FP64 plain ----
    spec64, _, jobs64, ms64, _, kt64, _, tile64 = timed_jobs(abi.F64, args.fp64_steps, 1)
    t64 = max_over_ranks(sum(ms64) / len(ms64), dev, world)
    value64 = aggregate_mcells(world, cells, args.nt, t64 / 1e3)

    # ---- DFT error FP32 vs FP64 (same job, same steps) ----
    dft_err = dft_rel_err(jobs32[0], jobs64[0], len(spec32.monitors))

    # ---- roofline of the dominant kernel (FP32) ----
    # with the block-step kernel (the tuner's usual choice here) one launch takes
    # every cell eight steps on; otherwise the interior (core) E and H kernels
    # update nearly all cells, with the edge and dispersive-cell kernels as
    # parallel branches
    if kt32["STEP"][0] > 0:
        dom, kname, per = "STEP", "step2d_block (TMz, FP32)", "step"
        note = ("algorithmic bytes = grid cells x (6w+1) per launch of eight steps: Ez, Hx, Hy read and written once "
                "and the material id read; the kernel is bound by its instructions, not by these bytes")
    else:
        dom = "E" if kt32["E"][1] >= kt32["H"][1] else "H"
        kname, per = f"{dom.lower()}2d_core<float,TM,4>", dom
        note = ("algorithmic bytes = core cells x (4w+1) for E, 5w for H; the working set (~0.1 GB) is "
                "L2-resident between steps (129 MB L2), so the frac can exceed 1 against HBM")
    cnt, tot, dcells = kt32[dom]
    avg_s = (tot / cnt) / 1e3
    bpl = dcells * alg_bytes(per, 4)
    achieved = bpl / avg_s / 1e9
    peak, peak_kind = measured_peaks()
    traffic, tr_src = profile_traffic(dom)
    roof = {"bound": "hbm", "kernel": kname, "achieved": achieved, "peak": peak,
            "unit": "GB/s", "frac": achieved / peak, "traffic": traffic, "peak_source": peak_kind,
            "alg_bytes_per_launch": bpl, "cells_per_launch": dcells, "avg_launch_us": avg_s * 1e6,
            "note": note}
    if tr_src:
        roof["traffic_source"] = tr_src
    step_bw = cells * alg_bytes("step", 4) / (t_step / 1e3 / args.nt) / 1e9

    # ---- end to end through the C ABI with host buffers ----
    # the spectra land in pinned host buffers allocated (and touched) before
    # the timed region, as the inputs of a streamed job would come from one
    from fdtd_gpu import spec as gspec
    spec_bufs = []
    for m in spec32.monitors:
        nc, nf, ncell = gspec.monitor_shape(m)
        spec_bufs.append(tuple(torch.zeros(nc * nf * ncell, dtype=torch.float64, pin_memory=True).numpy()
                               for _ in range(2)))
    e2e_runs = 2
    t_e2e, h2d, d2h = [], 0, 0
    for _ in range(e2e_runs):
        torch.cuda.synchronize()
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        J = gj.Job(spec32)              # host geometry -> device
        J.step(1, args.nt)
        outs = [J.get_monitor(q, out=spec_bufs[q]) for q in range(len(spec32.monitors))]  # spectra -> host
        t_e2e.append(time.perf_counter() - t0)
        h2d, d2h = J.transfer_bytes()
        J.close()
    e2e_value = aggregate_mcells(world, cells, args.nt, max_over_ranks(sum(t_e2e) / len(t_e2e), dev, world))

    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": t_step, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": workload_name(args.n, args.nt), "cells": cells, "time_steps_per_job": args.nt,
                   "bench_step": "one job of the workload from a fresh state",
                   "launch": ("CUDA graph per 32-step ring: the block-step kernels per eight steps, "
                              "the DFT fold per ring" if kt32["STEP"][0] > 0 else
                              "CUDA graph per 32-step ring (E, H and DFT fold kernels)"),
                   "tile": tile32,
                   "l2": f"{L2_FLUSH_BYTES >> 20} MiB buffer written between timed jobs",
                   "parallelism": f"replicas x{world}"},
        "fp64_plain": {"value": value64, "ms_per_step": t64, "steps": len(ms64), "tile": tile64},
        "fp32_over_fp64": value / value64,
        "dft_rel_err_fp32_vs_fp64": dft_err,
        "step_bandwidth_gbs": step_bw,
        "roofline": roof,
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "clock": ("host wall clock around create+commit (geometry from pageable host memory), all time "
                          "steps and the spectra download into pinned host buffers allocated before the clock starts")},
        "gpu_launches": launches,
        "kernel_ms_fp32": {k: {"launches": v[0], "ms": v[1], "cells": v[2]} for k, v in kt32.items()},
        "kernel_ms_fp64": {k: {"launches": v[0], "ms": v[1], "cells": v[2]} for k, v in kt64.items()},
        "clocks": clocks,
    }
    if rank == 0 and not args.no_configs:
        out["configs"] = config_runs(stream)
    if rank == 0 and args.serve_jobs > 0:
        out["serving"] = serving_run(args.serve_jobs, [float(x) for x in args.serve_rates.split(",") if x],
                                     args.serve_arms_jobs, args.serve_arms_rate)
    if rank == 0 and not args.no_cpu:
        out["cpu_baseline"] = cpu_measure(args.n, 1, 5)
    if rank == 0:
        print(json.dumps(out), flush=True)
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
