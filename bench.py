#!/usr/bin/env python
"""FP64 zone-updates/s of the moving-mesh RK2 step on B200.

A step is one timestep_rk2 of a disk (two substeps: face list, PLM,
HLL/HLLC + viscous fluxes, sources, mesh motion, boundaries).  A zone-update
is one non-ghost cell advanced by one full step.  Default workload: the
circumbinary disk (400 log annuli, r in [0.4, 20], 258,078 cells, equal-mass
binary, alpha = 0.1 viscosity, HLLC, outer damping zone).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Under torchrun (N > 1) every rank advances its own replica of the disk (the
single-disk step does not shard without a radial domain split): per-GPU work is fixed, the
reported value is the sum over ranks, timed as the maximum over ranks.
Prints one JSON line (rank 0).
"""
from __future__ import annotations

import argparse
import ctypes as C
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

METRIC = "FP64 zone-updates/s"
UNIT = "zone-updates/s"
PEAKS_FILE = os.path.join(HERE, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6650.0

# Algorithmic DRAM bytes per zone-update (one interior cell advanced by one RK2
# step): 5 conserved values and 1 phi edge, FP64, read and written across the
# two stages -- stage 1 reads U^n (48 B) and writes U^1 (48 B), stage 2 reads
# U^1 and U^n and writes U^(n+1) (144 B).  Everything else (prims, slopes,
# faces, w, dt) is recomputable within the step.
STEP_ALG_BYTES = 240
# The kernel that reads and writes the state carries those bytes: per interior
# cell, (substep 1, substep 2).  No other kernel of the step has a share.
STATE_SHARE = {"update": (96, 144), "sweep": (96, 144)}
PROFILE_SUMMARY = {"sweep": "profiles/sweep_circumbinary.md", "prep": "profiles/sweep_circumbinary.md",
                   "update": "profiles/step_kernels_circumbinary.md"}


def workload_params(name: str):
    from disco2_b200 import configs
    if name == "circumbinary":
        return configs.circumbinary(), ("circumbinary disk: equal-mass binary, 400 log annuli "
                                        "r in [0.4, 20], aspect 1, alpha=0.1, HLLC, PLM 1.5, "
                                        "outer damping r>16")
    if name == "kepler_ring":
        return configs.kepler_ring(), ("viscous Keplerian ring: 256 log annuli r in [0.5, 4], "
                                       "nu=1e-3, HLL")
    if name == "gresho":
        return configs.gresho(), ("Gresho vortex: 96 uniform annuli r in [0.1, 1], rigidly "
                                  "rotating mesh, HLLC")
    raise SystemExit(f"unknown workload {name}")


def profiled_traffic(kernel: str):
    """DRAM bytes per launch of a kernel (dram__bytes_read.sum +
    dram__bytes_write.sum) as recorded in the committed ncu summary of the
    same workload, and that file's name; (None, None) when there is none."""
    import re
    rel = PROFILE_SUMMARY.get(kernel)
    if rel is None:
        return None, None
    try:
        text = open(os.path.join(HERE, rel)).read()
    except OSError:
        return None, None
    m = re.search(r"dram_bytes_per_launch:([^`\n]*)", text)
    if not m:
        return None, None
    for tok in m.group(1).split():
        k, _, v = tok.partition("=")
        if k == "k_" + kernel:
            return float(v), rel
    return None, None


def load_peaks():
    try:
        with open(PEAKS_FILE) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """nvidia-smi sampling of SM clocks and throttle reasons while running."""

    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_id: str | None):
        self.proc = None
        self.path = None
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            cmd = ["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits", "-lms", "50"]
            if gpu_id:
                cmd += ["-i", gpu_id]
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(cmd, stdout=self.out, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.out.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        with open(self.path) as f:
            for line in f:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) < 8:
                    continue
                try:
                    sm.append(float(parts[0]))
                    smax.append(float(parts[1]))
                except ValueError:
                    continue
                for nm, v in zip(names, parts[4:8]):
                    if v.lower().startswith("active"):
                        reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        busy = [s for s in sm if s > 0.5 * max(sm)] or sm
        return {"sm_mhz": statistics.median(busy), "sm_max_mhz": max(smax), "samples": len(sm),
                "reasons": sorted(reasons)}


def cpu_baseline_run(par_text: str, steps: int, warmup: int):
    """Time the reference build (or the C restatement) on the host cores."""
    sys.path.insert(0, os.path.join(HERE, "oracle"))
    import oracle  # noqa: E402  (CPU baseline leg only)
    exe, kind = (oracle.REF_BIN, "reference") if oracle.have_ref() else (oracle.PORT_BIN, "port")
    if not os.path.exists(exe):
        try:
            oracle.build(ref=False, port=True)
        except Exception:
            pass
        exe, kind = oracle.PORT_BIN, "port"
    if not os.path.exists(exe):
        return None
    with tempfile.TemporaryDirectory() as td:
        par = os.path.join(td, "w.par")
        with open(par, "w") as f:
            f.write(par_text)
        r = subprocess.run([exe, "run", par, str(steps), os.path.join(td, "o.bin"), "--warmup",
                            str(warmup)], capture_output=True, text=True, check=True)
    wall = None
    for line in r.stderr.splitlines():
        if line.startswith("steps_wall_s"):
            wall = float(line.split()[1])
    return wall, kind


def cpu_batch_baseline(par_texts, nins, steps: int):
    """The sweep on the host: one reference (or restatement) process per disk,
    as many at once as there are host cores, each timing `steps` RK2 steps
    after its set-up.  Aggregate zone-updates/s = the steps' work over the
    core-seconds they took, times the cores used."""
    from concurrent.futures import ThreadPoolExecutor
    try:
        cores = len(os.sched_getaffinity(0))
    except AttributeError:
        cores = os.cpu_count() or 1
    cores = max(1, min(cores, len(par_texts)))
    with ThreadPoolExecutor(max_workers=cores) as ex:
        res = list(ex.map(lambda t: cpu_baseline_run(t, steps, 0), par_texts))
    if any(r is None for r in res):
        return None
    core_s = sum(w for w, _ in res)
    work = sum(n * steps for n in nins)
    return {"value": work / core_s * cores, "unit": UNIT, "cores": cores, "kind": res[0][1],
            "sample": f"{steps} RK2 step(s) of each of the {len(par_texts)} disks, one process "
                      f"per disk, {cores} at a time ({core_s:.1f} core-seconds of steps)"}


def interior_cells(sim) -> int:
    N_p, _ = sim.grid()
    ngmin = 1
    ngmax = int(sim.param("ng"))
    return int(N_p[ngmin:len(N_p) - ngmax].sum())


def reference_grid(par_text: str):
    """The state header of a workload from the reference build's own set-up (a
    0-step run dumps N_p and the cell count), so the reference arm never loads
    this package's library."""
    sys.path.insert(0, os.path.join(HERE, "oracle"))
    import oracle  # noqa: E402  (reference arm only)
    exe = oracle.REF_BIN if oracle.have_ref() else oracle.PORT_BIN
    with tempfile.TemporaryDirectory() as td:
        par = os.path.join(td, "w.par")
        with open(par, "w") as f:
            f.write(par_text)
        out = os.path.join(td, "o.bin")
        subprocess.run([exe, "run", par, "0", out], capture_output=True, check=True)
        st = oracle.read_state(out)
    return st


def run_reference(args, rank, world):
    """The reference build on every host core at once. Without MPI it is
    single-threaded, so each core runs its own copy of the disk; the value is
    the sum of the copies' zone-updates/s over a bounded sample of the steps."""
    if rank != 0:
        return
    from concurrent.futures import ThreadPoolExecutor
    from disco2_b200 import configs
    p, desc = workload_params(args.workload)
    text = configs.parfile_text(p)
    try:
        st = reference_grid(text)
    except Exception as e:  # no oracle binary could be built or run
        print(json.dumps({"impl": "reference", "unavailable": f"reference build did not run: {e}"}))
        return
    ng = int(p["ng"])
    nin = int(st.N_p[1:st.NR - ng].sum())
    # the reference needs ~2 s per step here: time a bounded sample of the K steps
    steps = max(1, min(args.steps, args.ref_max_steps))
    warm = max(0, min(args.warmup, 3))
    try:
        cores = len(os.sched_getaffinity(0))
    except AttributeError:
        cores = os.cpu_count() or 1
    with ThreadPoolExecutor(max_workers=cores) as ex:
        res = list(ex.map(lambda _: cpu_baseline_run(text, steps, warm), range(cores)))
    if any(r is None for r in res):
        print(json.dumps({"impl": "reference", "unavailable": "no oracle binary could be built"}))
        return
    walls = [w for w, _ in res]
    kind = res[0][1]
    value = sum(nin * steps / w for w in walls)
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": world,
        "steps": steps, "warmup": warm, "ms_per_step": 1e3 * sum(walls) / len(walls) / steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic", "config": {"workload": desc, "cells": int(st.N),
                                        "interior_cells": nin, "annuli": int(st.NR),
                                        "parallelism": f"{cores} independent copies, one per host core"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": kind,
                         "sample": f"{steps} of the {args.steps} requested RK2 steps of the same "
                                   f"disk, after {warm} warm-up step(s), in {cores} processes at "
                                   f"once (the reference is single-threaded without MPI); "
                                   f"ms_per_step is the mean over the processes"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def run_batched(args, rank, world, flush, barrier, max_over_ranks):
    """The 48-disk circumbinary sweep (q, alpha, h/r, N_r, R_out drawn from seed 3)
    advanced in one context, against the same disks advanced one context at a time;
    disks are split over ranks (no exchange)."""
    import torch
    from disco2_b200 import configs, lib, replicas
    sweep = configs.circumbinary_sweep(48, seed=3)
    sims_all = [lib.Sim(p) for p in sweep]
    part = replicas.partition([s.num_cells for s in sims_all], world)[rank]
    sims = [sims_all[k] for k in part]
    nin = [interior_cells(s) for s in sims]
    k_steps = max(3, min(args.steps, args.batch_steps))
    stream = torch.cuda.Stream()

    def timed(ctx):
        if args.tune_steps > 0:
            ctx.autotune(args.tune_steps)
        ctx.step(2, sync=True)  # warm-up, graph capture
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
              for _ in range(k_steps)]
        L = lib.load()
        for s, e in ev:
            with torch.cuda.stream(stream):
                flush.zero_()
                s.record(stream)
                L.dgpu_step_rk2(ctx.handle, 1)
                e.record(stream)
        ctx.synchronize()
        torch.cuda.synchronize()
        return sum(s.elapsed_time(e) for s, e in ev)

    ctx = lib.Context(sims, device=int(os.environ.get("LOCAL_RANK", "0")), stream=stream.cuda_stream)
    if args.fused:
        ctx.set_fused(True)
    for k in range(len(sims)):
        ctx.init_state(k)
    barrier()
    ms_b = max_over_ranks(timed(ctx))
    ctx.close()
    ms_seq = 0.0
    for s in sims:
        c1 = lib.Context(s, device=int(os.environ.get("LOCAL_RANK", "0")), stream=stream.cuda_stream)
        if args.fused:
            c1.set_fused(True)
        c1.init_state(0)
        ms_seq += timed(c1)
        c1.close()
    ms_seq = max_over_ranks(ms_seq)
    tot = sum(nin)
    if world > 1:
        t = torch.tensor([float(tot)], dtype=torch.float64, device="cuda")
        torch.distributed.all_reduce(t)
        tot = t.item()
    v_b = tot * k_steps / (ms_b / 1e3)
    v_s = tot * k_steps / (ms_seq / 1e3)
    cpu = None
    if world == 1 and not args.no_cpu and args.batch_cpu_steps > 0:
        cpu = cpu_batch_baseline([configs.parfile_text(p) for p in sweep],
                                 [interior_cells(s) for s in sims_all], args.batch_cpu_steps)
    return {"workload": "48 independent circumbinary disks from seed 3: q log-uniform [0.01,1], "
                        "alpha [0.01,0.1], h/r [0.05,0.1], N_r [128,512], R_out [10,30]",
            "cells": int(sum(s.num_cells for s in sims_all)), "interior_cells": int(tot),
            "steps": k_steps, "value": v_b, "unit": UNIT, "ms_per_step": ms_b / k_steps,
            "sequential_value": v_s, "batched_over_sequential": v_b / v_s,
            "how": "one context holding every disk of the rank vs one context per disk run (each autotuned) "
                   "back to back, same steps, L2 flushed before each step",
            "cpu_baseline": cpu}


def run_adjoint(args):
    """Cost of the gradient against the forward it differentiates: the
    circumbinary disk at 192 annuli, 500 RK2 steps, both objectives averaged
    over steps 251-500; forward = dgpu_objective (graph-replayed steps plus the
    objective after each step of its window), plain = the same number of dgpu_step_rk2
    steps with no objective, adjoint = dgpu_adjoint (forward sweep with a
    checkpoint every 25 steps, then each segment replayed and reversed),
    tangent = dgpu_tangent along q.  Wall time of the synchronous calls."""
    from disco2_b200 import configs, lib
    n, w0, K = args.adj_steps, args.adj_steps // 2, 25
    s = lib.Sim(configs.circumbinary(num_r=192))
    ctx = lib.Context(s, device=int(os.environ.get("LOCAL_RANK", "0")))
    ctx.init_state(0)
    ctx.objective(4, 2)          # graph capture, buffers
    ctx.init_state(0)
    ctx.adjoint(4, 2, ckpt_every=2)
    ctx.init_state(0)
    ctx.tangent(4, 2, dq=1.0)
    ctx.init_state(0)
    ctx.step(2)                  # the plain step's graph
    res = {}
    for name, fn in (("forward", lambda: ctx.objective(n, w0)),
                     ("plain", lambda: ctx.step(n)),
                     ("adjoint", lambda: ctx.adjoint(n, w0, ckpt_every=K)),
                     ("tangent", lambda: ctx.tangent(n, w0, dq=1.0))):
        best = None
        for _ in range(2):
            ctx.init_state(0)
            ctx.synchronize()
            t0 = time.perf_counter()
            fn()
            ctx.synchronize()
            dt = time.perf_counter() - t0
            best = dt if best is None else min(best, dt)
        res[name] = best
    ctx.close()
    return {"workload": f"circumbinary disk, 192 annuli ({s.num_cells} cells), {n} steps, objectives "
                        f"averaged over steps {w0 + 1}-{n}, checkpoints every {K} steps",
            "forward_s": res["forward"], "plain_steps_s": res["plain"], "adjoint_s": res["adjoint"],
            "tangent_s": res["tangent"],
            "adjoint_over_forward": res["adjoint"] / res["forward"],
            "adjoint_over_plain_steps": res["adjoint"] / res["plain"],
            "tangent_over_forward": res["tangent"] / res["forward"],
            "how": "wall time of the synchronous library calls, best of 2, same initial state"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="circumbinary")
    ap.add_argument("--ref-max-steps", type=int, default=12)
    ap.add_argument("--cpu-steps", type=int, default=10)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-batched", action="store_true")
    ap.add_argument("--no-alt", action="store_true", help="skip timing the other substep form")
    ap.add_argument("--no-3d", action="store_true", help="skip timing the 3-D torus")
    ap.add_argument("--batch-steps", type=int, default=20)
    ap.add_argument("--batch-cpu-steps", type=int, default=1,
                    help="RK2 steps per disk of the sweep's host baseline (0: skip it)")
    ap.add_argument("--tune-steps", type=int, default=3,
                    help="steps per launch-shape candidate for the autotuner (0: built-in shapes)")
    ap.add_argument("--no-adjoint", action="store_true")
    ap.add_argument("--adj-steps", type=int, default=500)
    ap.add_argument("--fused", action="store_true",
                    help="time the fused substep (k_prep + k_sweep) instead of the eight kernels")
    args = ap.parse_args()

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return

    import torch
    import torch.distributed as dist
    from disco2_b200 import configs, lib

    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))

    def barrier():
        if world > 1:
            dist.barrier()

    def max_over_ranks(x: float) -> float:
        if world == 1:
            return x
        t = torch.tensor([x], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    p, desc = workload_params(args.workload)
    sim = lib.Sim(p)
    nin = interior_cells(sim)
    stream = torch.cuda.Stream()
    ctx = lib.Context(sim, device=local, stream=stream.cuda_stream)
    if args.fused:
        ctx.set_fused(True)
    ctx.init_state(0)
    L = lib.load()
    # launch shapes of the heavy kernels timed on this disk (state restored)
    tuned = ctx.autotune(args.tune_steps) if args.tune_steps > 0 else None

    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device="cuda")
    uuid = None
    try:
        uuid = "GPU-" + str(torch.cuda.get_device_properties(local).uuid)
    except Exception:
        pass

    # warm-up (also captures the step graph)
    with torch.cuda.stream(stream):
        ctx.step(args.warmup, sync=False)
    ctx.synchronize()
    sampler = ClockSampler(uuid)
    # keep the GPU busy ~0.3 s before timing so the clock samples see load
    t_end = time.time() + 0.3
    while time.time() < t_end:
        ctx.step(20, sync=False)
        ctx.synchronize()
    barrier()
    torch.cuda.synchronize()
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    for k in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
            starts[k].record(stream)
            L.dgpu_step_rk2(ctx.handle, 1)
            ends[k].record(stream)
    ctx.synchronize()
    torch.cuda.synchronize()
    barrier()
    clocks = sampler.stop()
    ms = sum(s.elapsed_time(e) for s, e in zip(starts, ends))
    ms = max_over_ranks(ms)
    value = nin * args.steps * world / (ms / 1e3)

    # per-kernel device times (same steps launched kernel by kernel, L2 flushed between steps)
    kern = {}
    nprof = max(3, min(args.steps, 50))
    for k in range(nprof):
        with torch.cuda.stream(stream):
            flush.zero_()
        torch.cuda.synchronize()
        for nm, (t1, t2) in ctx.step_timed(1).items():
            a, b = kern.get(nm, (0.0, 0.0))
            kern[nm] = (a + t1, b + t2)
    kern = {nm: (a / nprof, b / nprof) for nm, (a, b) in kern.items()}  # ms per launch, substep 1 / 2
    per_kernel = {nm: (a + b) / 2 for nm, (a, b) in kern.items()}
    # the roofline's kernel: the one that reads and writes the state, the only one with a share of
    # the algorithmic bytes (k_flux_r takes as long)
    dom = max((nm for nm in per_kernel if nm in STATE_SHARE), key=per_kernel.get)
    slowest = max(per_kernel, key=per_kernel.get)
    fl = ctx.face_list(0)
    nfaces = int(len(fl["L"]))
    ncell = sim.num_cells
    peak, peak_kind = load_peaks()
    # its share of the algorithmic bytes, over its two launches of a step
    s1, s2 = STATE_SHARE[dom]
    alg_bytes_step = (s1 + s2) * nin
    achieved = alg_bytes_step / ((kern[dom][0] + kern[dom][1]) * 1e-3) / 1e9
    traffic, traffic_src = profiled_traffic(dom) if args.workload == "circumbinary" else (None, None)
    fused = ctx.fused
    # beside the substeps' kernels: k_ring_mean of a rigid mesh, in both substeps, and k_dt, in
    # the eight-kernel step of more than two waves of cells (dgpu_ctx.c: few_waves)
    rigid = p["w_numeric_type"] == 2
    with_dt = not fused and sim.num_cells > 2 * 148 * 4 * 256
    launches_per_step = 2 * (len(ctx.kernels) + (rigid and not fused)) + with_dt

    # end to end through the C ABI: host (pinned) state in, one step, host state out
    n = sim.num_cells
    prim_h = torch.empty((n, 5), dtype=torch.float64, pin_memory=True)
    tiph_h = torch.empty(n, dtype=torch.float64, pin_memory=True)
    dphi_h = torch.empty(n, dtype=torch.float64, pin_memory=True)
    dp = C.POINTER(C.c_double)
    P_prim = C.cast(prim_h.data_ptr(), dp)
    P_tiph = C.cast(tiph_h.data_ptr(), dp)
    P_dphi = C.cast(dphi_h.data_ptr(), dp)
    rc = L.dgpu_get_state(ctx.handle, 0, P_prim, None, P_tiph, P_dphi)
    assert rc == 0, L.dgpu_last_error(ctx.handle)
    h2d = (5 + 2) * 8 * n
    d2h = (5 + 2) * 8 * n
    ke = max(3, min(args.steps, 50))
    for _ in range(2):  # warm
        L.dgpu_set_state(ctx.handle, 0, P_prim, P_tiph, P_dphi)
        L.dgpu_step_rk2(ctx.handle, 1)
        L.dgpu_get_state(ctx.handle, 0, P_prim, None, P_tiph, P_dphi)
    barrier()
    t0 = time.perf_counter()
    for _ in range(ke):
        rc = L.dgpu_set_state(ctx.handle, 0, P_prim, P_tiph, P_dphi)
        rc |= L.dgpu_step_rk2(ctx.handle, 1)
        rc |= L.dgpu_get_state(ctx.handle, 0, P_prim, None, P_tiph, P_dphi)
        assert rc == 0, L.dgpu_last_error(ctx.handle)
    e2e_s = max_over_ranks(time.perf_counter() - t0)
    e2e = nin * ke * world / e2e_s

    ctx.close()

    # the other substep form on the same disk (informational): the fused
    # k_prep + k_sweep when the line is the eight-kernel graph, and back
    alt = None
    if world == 1 and not args.no_alt:
        actx = lib.Context(sim, device=local, stream=stream.cuda_stream)
        actx.set_fused(not fused)
        actx.init_state(0)
        if args.tune_steps > 0:
            actx.autotune(args.tune_steps)
        with torch.cuda.stream(stream):
            actx.step(args.warmup, sync=False)
        actx.synchronize()
        ka = max(3, min(args.steps, 100))
        a_s = [torch.cuda.Event(enable_timing=True) for _ in range(ka)]
        a_e = [torch.cuda.Event(enable_timing=True) for _ in range(ka)]
        for k in range(ka):
            with torch.cuda.stream(stream):
                flush.zero_()
                a_s[k].record(stream)
                L.dgpu_step_rk2(actx.handle, 1)
                a_e[k].record(stream)
        actx.synchronize()
        torch.cuda.synchronize()
        a_ms = sum(x.elapsed_time(y) for x, y in zip(a_s, a_e))
        alt = {"substep": "eight kernels" if fused else "fused (k_prep + k_sweep)", "steps": ka,
               "ms_per_step": a_ms / ka, "value": nin * ka / (a_ms / 1e3), "unit": UNIT,
               "how": "same disk and timing as the line (autotuned, L2 flushed before each step)"}
        actx.close()

    # the reference's torus.par (3-D, 80 x 80 annuli and layers), informational
    three_d = None
    if world == 1 and not args.no_3d:
        from disco2_b200 import configs as _cf
        tsim = lib.Sim(_cf.torus_3d())
        tctx = lib.Context(tsim, device=local, stream=stream.cuda_stream)
        tctx.init_state(0)
        if args.tune_steps > 0:
            tctx.autotune(args.tune_steps)
        with torch.cuda.stream(stream):
            tctx.step(args.warmup, sync=False)
        tctx.synchronize()
        kt = max(3, min(args.steps, 100))
        t_s = [torch.cuda.Event(enable_timing=True) for _ in range(kt)]
        t_e = [torch.cuda.Event(enable_timing=True) for _ in range(kt)]
        for k in range(kt):
            with torch.cuda.stream(stream):
                flush.zero_()
                t_s[k].record(stream)
                L.dgpu_step_rk2(tctx.handle, 1)
                t_e[k].record(stream)
        tctx.synchronize()
        torch.cuda.synchronize()
        t_ms = sum(x.elapsed_time(y) for x, y in zip(t_s, t_e))
        tin = interior_cells(tsim) * int(tsim.param("NumZ"))  # non-ghost annuli of the non-ghost layers
        three_d = {"workload": f"torus.par: 3-D torus, 80 annuli x 80 layers, periodic z ({tsim.num_cells} cells, "
                               f"{tin} interior)", "steps": kt, "ms_per_step": t_ms / kt,
                   "value": tin * kt / (t_ms / 1e3), "unit": UNIT,
                   "how": "autotuned, L2 flushed before each step, CUDA events on the library's stream"}
        tctx.close()

    batched = None
    if not args.no_batched:
        batched = run_batched(args, rank, world, flush, barrier, max_over_ranks)

    adjoint = None
    if world == 1 and not args.no_adjoint:
        adjoint = run_adjoint(args)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        res = cpu_baseline_run(configs.parfile_text(p), args.cpu_steps, 1)
        if res is not None:
            wall, kind = res
            cpu = {"value": nin * args.cpu_steps / wall, "unit": UNIT, "cores": 1, "kind": kind,
                   "sample": f"{args.cpu_steps} RK2 steps of the same disk on one host core, "
                             f"after 1 warm-up step ({wall:.1f} s)"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "cells": ncell, "interior_cells": nin,
                       "annuli": sim.num_annuli, "r_faces": nfaces,
                       "l2": "flushed between timed steps (256 MiB write outside the events)",
                       "parallelism": f"replicas x{world}" if world > 1 else "single disk",
                       "blocks_per_sm": tuned},
            "roofline": {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": peak,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / peak,
                         "traffic": traffic,
                         "alg_bytes_per_launch": alg_bytes_step / 2,
                         "alg_bytes": f"{s1} B (substep 1) and {s2} B (substep 2) per interior cell: "
                                      "the conserved state and phi edge the kernel reads and writes",
                         "ms_per_launch": per_kernel[dom],
                         "slowest_kernel": slowest, "slowest_ms_per_launch": per_kernel[slowest],
                         "traffic_source": (f"copied from {traffic_src} (ncu dram__bytes_read.sum + "
                                            "dram__bytes_write.sum, one launch of the same workload); "
                                            "not measured in this run") if traffic_src else None},
            "step_roofline": {"alg_bytes_per_zone_update": STEP_ALG_BYTES,
                              "achieved_gbs": value / world * STEP_ALG_BYTES / 1e9,
                              "frac": value / world * STEP_ALG_BYTES / 1e9 / peak},
            "kernel_ms": {nm: {"substep1": a, "substep2": b} for nm, (a, b) in kern.items()},
            "step_kernels": "fused: k_prep + k_sweep per substep" if fused else
                            "eight kernels per substep",
            "gpu_launches": launches_per_step * args.steps,
            "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "steps": ke, "how": "dgpu_set_state from pinned host prim/tiph/dphi, "
                                        "dgpu_step_rk2(1), dgpu_get_state to pinned host, per step"},
            "cpu_baseline": cpu,
            "clocks": clocks,
            "alt_substep": alt,
            "three_d": three_d,
            "batched": batched,
            "adjoint": adjoint,
        }
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
