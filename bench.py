#!/usr/bin/env python
"""Benchmark of the B200 gradient-domain Poisson solver.

Default workload (one GPU): tone-mapping-style Neumann integration of a
4096 x 4096 x 3 radiance map (16.8 MP per channel, three channels solved as
one batched plan), mixed precision (FP32 V-cycle, FP64 residual refresh and
accumulator) to a true relative residual of 1e-8.  The plan's sweeps and kernel
geometry come from the project's autotuner, run on the plan's own right-hand
sides before the measurement (``--no-tune``: ``--sweeps`` and the default
geometry; the choice is in ``config.autotuned``).  One step = one batched
solve of the three channels from x0 = 0.  ``value`` is whole-job Mpix/s
(channels x pixels / step time, device-timed, inputs resident in HBM);
``e2e`` repeats the measurement through the public API with pinned host
buffers, including both copies of every step, with several steps in flight
(three, ``solve_neumann_batch_async``; ``e2e.one_call_at_a_time`` is the same with
each call finished before the next); the FP64 MGPCG on the same plan shape is
timed for the mixed-vs-FP64 ratio.

    python bench.py [--gpus N --steps K --warmup W] [--impl reference]
    python bench.py --config composite|batch|serve|smoother|autotune|dct

Under torchrun each rank solves its own replica (no collective on the data
path; ``scaling`` = weak) and rank 0 prints one JSON line with the max over
ranks of the device time.
"""

from __future__ import annotations

import argparse
import dataclasses
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "Mpix/s to 1e-8 rel. residual, mixed vs FP64 MGPCG; served p50/p99 latency"
FALLBACK_HBM_GBS = 6650.0

# Algorithmic bytes per grid cell of each kernel kind (FP32 vectors of the
# mixed plan; the FP64 plan doubles the FP32 terms).  Level kernels count the
# cells of the level they work on; coarse arrays are a quarter of that.
BYTES_PER_CELL_MIXED = {
    "down0": 4 + 4 + 1, "down": 4 + 4 + 1,          # read b; write pre-smoothed w, coarse b
    "up0": 4 + 4 + 1 + 4, "up": 4 + 4 + 1 + 4,      # read b, w, coarse e; write u
    "pupdate": 4 + 4 + 4,                   # read z, p; write p
    "cgupdate": 12 + 8,                     # read p, d, r; write d, r
    "resid": 8 + 4 + 8 + 8 + 4,             # read x, d, f; write x + d, r (refresh iterations)
    "init": 8 + 8 + 4,                      # read f twice (its mean, then r); write r; x = 0
    "mean": 8 + 8,                          # read the solution; write x, mean subtracted
}


def bytes_per_cell(kind: str, fp64: bool) -> float:
    b = BYTES_PER_CELL_MIXED.get(kind, 0.0)
    if not fp64:
        return b
    fp32_part = {"down0": 9, "down": 9, "up0": 13, "up": 13, "pupdate": 12, "cgupdate": 20,
                 "resid": 8, "init": 4, "mean": 0}.get(kind, 0)
    return b + fp32_part


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as fh:
            data = json.load(fh)
        return float(data["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle sampling while the timed region runs."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.lines: list[str] = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "50"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except Exception:
            self.proc = None
            return
        # nvidia-smi takes a moment to start: begin the timed region once it samples
        t0 = time.perf_counter()
        while not self.lines and time.perf_counter() - t0 < 5.0:
            time.sleep(0.01)
        self.first = len(self.lines)

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        # at least one sample taken after the timed region began (a short region can end
        # between two samples; the GPU is still at its load clock just after)
        t0 = time.perf_counter()
        while len(self.lines) <= getattr(self, "first", 0) and time.perf_counter() - t0 < 2.0:
            time.sleep(0.01)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        during = self.lines[getattr(self, "first", 0):] or self.lines
        for line in during:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": float(max(smax)) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_setup():
    from gradient_domain_b200 import replicas
    return replicas.rank_env()


def cpu_baseline_tonemap(rhs: np.ndarray, budget_s: float = 20.0) -> dict:
    """Time the oracle's DCT Neumann solve (the reference's CPU path) on host cores."""
    from oracle import solvers as osolvers
    cores = os.cpu_count() or 1
    n_ch, h, w = rhs.shape
    t0 = time.perf_counter()
    done = 0
    while done < n_ch and (time.perf_counter() - t0) < budget_s:
        osolvers.solve_neumann(rhs[done], workers=cores)
        done += 1
    dt = time.perf_counter() - t0
    # the same solve on one core (one fft worker; the NumPy steps are single-threaded)
    t1 = time.perf_counter()
    osolvers.solve_neumann(rhs[0], workers=1)
    dt1 = time.perf_counter() - t1
    return {"value": done * h * w / dt / 1e6, "unit": "Mpix/s", "cores": cores, "kind": "port",
            "sample": f"{done} of {n_ch} channels of {h}x{w}, scipy DCT solve_neumann "
                      f"restatement, {cores} fft workers, {dt:.2f} s",
            "single_core": {"value": h * w / dt1 / 1e6, "unit": "Mpix/s", "cores": 1,
                            "sample": f"1 channel of {h}x{w}, 1 fft worker, {dt1:.2f} s"}}


def reference_arm(args) -> None:
    """`--impl reference`: the reference's CPU algorithm for this path on host cores."""
    world, rank, _ = dist_setup()
    if rank != 0:
        return
    from gradient_domain_b200 import workloads
    from oracle import solvers as osolvers
    rhs = workloads.tonemap_rhs(args.size, seed=1)
    cores = os.cpu_count() or 1
    n_ch, h, w = rhs.shape
    for _ in range(args.warmup):
        osolvers.solve_neumann(rhs[0], workers=cores)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        for c in range(n_ch):
            osolvers.solve_neumann(rhs[c], workers=cores)
    dt = (time.perf_counter() - t0) / args.steps
    value = n_ch * h * w / dt / 1e6
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "Mpix/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": f"tonemap-neumann {args.size}x{args.size}x3", "tolerance": "exact"},
        "cpu_baseline": {"value": value, "unit": "Mpix/s", "cores": cores, "kind": "port",
                         "sample": f"full workload per step ({n_ch} channels), scipy DCT "
                                   f"restatement of solve_neumann, {cores} fft workers"},
        "e2e": {"value": value, "unit": "Mpix/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


E2E_DEPTH = 3  # steps in flight in the end-to-end leg


def ours(args) -> None:
    import torch

    from gradient_domain_b200 import replicas, workloads
    from gradient_domain_b200.plan import Instance, PoissonPlan, SolveParams
    from gradient_domain_b200.solvers import solve_neumann_batch, solve_neumann_batch_async

    world, rank, local = dist_setup()
    torch.cuda.set_device(local)
    replicas.init(world)

    dev = torch.device("cuda", local)
    size = args.size
    rhs_np = workloads.tonemap_rhs(size, seed=replicas.replica_seed(1, rank),
                                   channels=args.channels)
    n_ch = rhs_np.shape[0]
    cells = n_ch * size * size
    f = torch.as_tensor(rhs_np).to(dev)
    x = torch.empty_like(f)
    insts = [Instance(size, size, "neumann", zero_mean=True) for _ in range(n_ch)]
    # every solve starts from zero (as the reference's solve_neumann); x is only written
    params = SolveParams(precision="mixed", tolerance=args.tol, sweeps=args.sweeps,
                         reliable_delta=args.delta, zero_start=True)
    tuning = None
    if not args.no_tune:
        # the plan's sweeps and kernel geometry come from the autotuner, timed on this
        # plan's own right-hand sides before the measurement (untimed)
        from gradient_domain_b200 import autotune
        t0 = time.perf_counter()
        params = autotune.tune(insts, params, rhs=list(f), reps=3, force=True, scale=-1.0)
        tuning = {name: getattr(params, name) for name, _ in autotune.SPACE}
        tuning["seconds"] = round(time.perf_counter() - t0, 2)
    plan = PoissonPlan(insts, params)
    stream = torch.cuda.current_stream()

    def step(p):
        return p.solve(list(f), list(x), scale=-1.0)

    def barrier():
        replicas.barrier(world)

    def max_over_ranks(v: float) -> float:
        return replicas.max_over_ranks(v, world, dev)

    for _ in range(args.warmup):
        results = step(plan)
    if args.solve_only:
        for _ in range(args.steps):
            results = step(plan)
        torch.cuda.synchronize()
        if rank == 0:
            print(json.dumps({"solve_only": True, "iterations": [r.iterations for r in results],
                              "relative_residual": max(r.relative_residual for r in results)}))
        plan.close()
        return
    clocks = ClockSampler(local)
    clocks.start()
    barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        results = step(plan)
    e1.record(stream)
    torch.cuda.synchronize()
    barrier()
    clock = clocks.stop()
    ms = max_over_ranks(e0.elapsed_time(e1) / args.steps)
    # Per-kernel CUDA-event durations: the same steps again with an event pair around
    # every launch.  Graphs are bypassed while profiling, so this pass runs on direct
    # launches with host polls and is a little slower than the headline pass.
    plan.set_profiling(True)
    barrier()
    torch.cuda.synchronize()
    e0.record(stream)
    for _ in range(args.steps):
        step(plan)
    e1.record(stream)
    torch.cuda.synchronize()
    ms_prof = max_over_ranks(e0.elapsed_time(e1) / args.steps)
    ktimes = plan.kernel_times()
    plan.set_profiling(False)
    value = replicas.aggregate_rate(cells, world, ms / 1e3) / 1e6
    its = [r.iterations for r in results]
    resid = max(r.relative_residual for r in results)
    converged = all(r.converged for r in results)

    # accuracy against the FP64 oracle (DCT) and CPU baseline, rank 0 only
    extra = {}
    sol = (x.cpu().numpy())
    if rank == 0 and not args.no_cpu:
        from oracle import solvers as osolvers
        t0 = time.perf_counter()
        errs = []
        for c in range(n_ch):
            ref = osolvers.solve_neumann(rhs_np[c], workers=os.cpu_count())
            errs.append(float(np.linalg.norm(sol[c] - ref) / np.linalg.norm(ref)))
        extra["rel_l2_err_vs_fp64_oracle"] = errs
        extra["oracle_seconds"] = time.perf_counter() - t0

    # FP64 MGPCG on the same workload (the precision baseline)
    plan64 = PoissonPlan(insts, dataclasses.replace(params, precision="fp64"))
    for _ in range(2):  # the second solve builds the plan's graph
        step(plan64)
    barrier()
    torch.cuda.synchronize()
    e0.record(stream)
    k64 = max(3, args.steps)
    for _ in range(k64):
        r64 = step(plan64)
    e1.record(stream)
    torch.cuda.synchronize()
    ms64 = max_over_ranks(e0.elapsed_time(e1) / k64)
    value64 = replicas.aggregate_rate(cells, world, ms64 / 1e3) / 1e6
    del plan64

    # the literal GPU port of the reference mgcg (vertex-centred V-cycle, one kernel per
    # operation, FP64, scalars read back every iteration) against the B200 solver on the
    # same 4096^2 Dirichlet manufactured problem (the reference mgcg is Dirichlet-only);
    # both device-resident: right-hand side on the device, solution left there
    port = None
    if rank == 0 and not args.no_port:
        from gradient_domain_b200 import benchmark as gbench
        from gradient_domain_b200.solvers import _ref_pcg_dev
        bm, _ = gbench.manufactured_problem((size, size), seed=0)
        bmd = torch.as_tensor(bm).to(dev)
        _ref_pcg_dev(bmd, 1.0, args.tol, 2000, "vcycle")  # warm-up: allocations, kernel loads
        torch.cuda.synchronize()
        t_port = []
        for _ in range(2):
            t0 = time.perf_counter()
            _, it_port, ok_port = _ref_pcg_dev(bmd, 1.0, args.tol, 2000, "vcycle")
            torch.cuda.synchronize()
            t_port.append(time.perf_counter() - t0)
        t_port = min(t_port)
        pd = PoissonPlan([Instance(size, size, "dirichlet")],
                         SolveParams(precision="mixed", tolerance=args.tol, sweeps=args.sweeps,
                                     reliable_delta=args.delta, zero_start=True))
        fd = torch.as_tensor(bm).to(dev)
        xd = torch.empty_like(fd)
        for _ in range(2):  # the second solve captures the plan's graph
            pd.solve([fd], [xd], scale=-1.0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(3):
            (rd,) = pd.solve([fd], [xd], scale=-1.0)
        torch.cuda.synchronize()
        t_ours = (time.perf_counter() - t0) / 3
        pd.close()
        # three instances (the channel count of the headline): the port solves them one
        # after another, the B200 solver as one batched plan
        pd3 = PoissonPlan([Instance(size, size, "dirichlet")] * 3,
                          SolveParams(precision="mixed", tolerance=args.tol, sweeps=args.sweeps,
                                      reliable_delta=args.delta, zero_start=True))
        xd3 = [torch.empty_like(fd) for _ in range(3)]
        for _ in range(2):
            pd3.solve([fd] * 3, xd3, scale=-1.0)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(3):
            pd3.solve([fd] * 3, xd3, scale=-1.0)
        torch.cuda.synchronize()
        t_ours3 = (time.perf_counter() - t0) / 3
        pd3.close()
        port = {"workload": f"dirichlet manufactured {size}x{size}x1, tolerance {args.tol}",
                "port_ms": t_port * 1e3, "port_iterations": it_port, "port_converged": ok_port,
                "port_mpix_s": size * size / t_port / 1e6,
                "b200_mixed_ms": t_ours * 1e3, "b200_mixed_iterations": rd.iterations,
                "b200_mixed_mpix_s": size * size / t_ours / 1e6,
                "speedup_over_port": t_port / t_ours,
                "note": "one instance is the B200 solver's weakest case: its latency-bound "
                        "coarse levels are not shared with other instances",
                "three_instances": {"port_ms": 3 * t_port * 1e3, "b200_mixed_ms": t_ours3 * 1e3,
                                    "speedup_over_port": 3 * t_port / t_ours3}}

    # the exact DCT Neumann solver (solvers.py:224-262 on the device) on the same workload
    dct = None
    if rank == 0:
        from gradient_domain_b200.solvers import DctPlan
        dplan = DctPlan(size, size)
        ud = torch.empty_like(f)
        for _ in range(2):
            for c in range(n_ch):
                dplan.solve(f[c], ud[c])
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(args.steps):
            for c in range(n_ch):
                dplan.solve(f[c], ud[c])
        e1.record(stream)
        torch.cuda.synchronize()
        ms_dct = e0.elapsed_time(e1) / args.steps
        dct = {"ms_per_step": ms_dct, "mpix_s": cells / (ms_dct / 1e3) / 1e6,
               "note": "exact transform solve (the reference's solve_neumann algorithm), "
                       "this library's FFT kernels: rows, columns with the eigenvalue division, rows"}
        if not args.no_cpu:
            from oracle import solvers as osolvers
            ref0 = osolvers.solve_neumann(rhs_np[0], workers=os.cpu_count())
            # laplacian(u) = b here; the MGPCG plan solves A x = -b, the same zero-mean u
            dct["rel_l2_err_vs_fp64_oracle_channel0"] = float(
                np.linalg.norm(ud[0].cpu().numpy() - ref0) / np.linalg.norm(ref0))
        del dplan

    # end to end through the public API, pinned host buffers, copies timed
    host_in = torch.as_tensor(rhs_np).pin_memory()
    host_out = torch.empty_like(host_in).pin_memory()
    for _ in range(max(2, args.warmup)):  # the second call captures the per-channel graphs
        solve_neumann_batch(host_in, tolerance=args.tol, out=host_out)
    barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e0.record(stream)
    for _ in range(args.steps):
        solve_neumann_batch(host_in, tolerance=args.tol, out=host_out)
    e1.record(stream)
    torch.cuda.synchronize()
    wall = (time.perf_counter() - t0) / args.steps
    ms_e2e_sync = max_over_ranks(max(e0.elapsed_time(e1) / args.steps, wall * 1e3))
    # the same calls with E2E_DEPTH steps in flight (solve_neumann_batch_async): a
    # step's uploads overlap earlier steps' solves and downloads; every step still
    # copies its right-hand sides up and its solutions down inside the timed region,
    # through E2E_DEPTH alternating sets of pinned buffers
    host_in2 = [host_in] + [torch.as_tensor(rhs_np).pin_memory() for _ in range(E2E_DEPTH - 1)]
    host_out2 = [host_out] + [torch.empty_like(host_in).pin_memory()
                              for _ in range(E2E_DEPTH - 1)]
    for _ in range(2):
        futs = [solve_neumann_batch_async(host_in2[j], host_out2[j], tolerance=args.tol)
                for j in range(E2E_DEPTH)]
        for fut in futs:
            fut.result()
    barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e0.record(stream)
    pending = []
    for k in range(args.steps):
        j = k % E2E_DEPTH
        pending.append(solve_neumann_batch_async(host_in2[j], host_out2[j], tolerance=args.tol))
        if len(pending) == E2E_DEPTH:
            pending.pop(0).result()
    for fut in pending:
        fut.result()
    e1.record(stream)
    torch.cuda.synchronize()
    wall = (time.perf_counter() - t0) / args.steps
    ms_e2e = max_over_ranks(max(e0.elapsed_time(e1) / args.steps, wall * 1e3))
    e2e_value = replicas.aggregate_rate(cells, world, ms_e2e / 1e3) / 1e6

    # roofline of the dominant kernel (live CUDA-event durations)
    hbm, peak_kind = peaks()
    kinds = {k: v for k, v in ktimes.items() if v["launches"] > 0}
    dom = max(kinds, key=lambda k: kinds[k]["ms"])
    d = kinds[dom]
    per_launch_ms = d["ms"] / d["launches"]
    per_launch_cells = d["cells"] / d["launches"]
    algo_bytes = bytes_per_cell(dom, False) * per_launch_cells
    achieved = algo_bytes / (per_launch_ms / 1e3) / 1e9
    traffic = None
    tpath = os.path.join(ROOT, "profiles", "traffic_per_cell.json")
    if os.path.exists(tpath):
        with open(tpath) as fh:
            tpc = json.load(fh).get(dom)
        if not isinstance(tpc, (int, float)):
            tpc = None
        if tpc:
            traffic = tpc * per_launch_cells
    total_ms = sum(v["ms"] for v in kinds.values())
    # launches in the headline pass: per solve the two init kernels, per executed iteration
    # the iteration's kernels without the refresh, one refresh kernel per refresh that ran,
    # then the solution kernel (the zero-start plan's refreshes leave the mean, so no mean
    # kernel; the device loop runs exactly max(iterations) iterations)
    iter_kinds = [k for k in kinds if k not in ("init", "mean", "resid")]
    per_iter = sum(kinds[k]["launches"] for k in iter_kinds) / max(kinds["pupdate"]["launches"], 1)
    refreshes = max(r.refreshes for r in results)
    launches = args.steps * (2 + max(its) * per_iter + refreshes + 1)

    smoother = smoother_gate(size, hbm, kinds, params.sweeps) if rank == 0 else None

    line = {
        "metric": METRIC, "value": value, "unit": "Mpix/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "fp32/fp64-mixed", "data": "synthetic",
        "config": {"workload": f"tonemap-neumann {size}x{size}x{n_ch}", "tolerance": args.tol,
                   "sweeps": params.sweeps, "autotuned": tuning, "reliable_delta": args.delta,
                   "instances_per_gpu": n_ch,
                   "l2": "inputs larger than L2 (3 x 134 MB rhs + solution + hierarchy)",
                   "parallelism": f"replicas x{world}"},
        "clocks": clock,
        "e2e": {"value": e2e_value, "unit": "Mpix/s", "ms_per_step": ms_e2e,
                "h2d_bytes_per_step": int(host_in.numel() * 8),
                "d2h_bytes_per_step": int(host_out.numel() * 8),
                "api": f"solve_neumann_batch_async, {E2E_DEPTH} steps in flight, pinned FP64 "
                       "host buffers",
                "pcie_bound_note": "402 MB up and 402 MB down per step at about 50 GB/s each "
                                   "way (full duplex): about 8.1 ms per step",
                "one_call_at_a_time": {
                    "value": replicas.aggregate_rate(cells, world, ms_e2e_sync / 1e3) / 1e6,
                    "ms_per_step": ms_e2e_sync, "api": "solve_neumann_batch(host_in, out=host_out)"}},
        "gpu_launches": int(launches),
        "iterations": its, "relative_residual": resid, "converged": converged,
        "port_equivalent_fp64": port,
        "dct_neumann": dct,
        "smoother": smoother,
        "fp64_mgpcg": {"value": value64, "ms_per_step": ms64,
                       "iterations": [r.iterations for r in r64],
                       "mixed_over_fp64": value / value64},
        "roofline": {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": hbm,
                     "unit": "GB/s", "frac": achieved / hbm, "peak_source": peak_kind,
                     "traffic": traffic, "algorithmic_bytes_per_launch": algo_bytes,
                     "avg_launch_ms": per_launch_ms},
        "kernel_share": {k: round(v["ms"] / total_ms, 4) for k, v in kinds.items()},
        "kernel_ms_per_step": {k: v["ms"] / args.steps for k, v in kinds.items()},
        "profiled_pass_ms_per_step": ms_prof,
    }
    line.update(extra)
    if rank == 0 and not args.no_serve:
        line["serving"] = serving_1mp(args)
    if rank == 0 and world == 1 and not args.no_cpu:
        line["cpu_baseline"] = cpu_baseline_tonemap(rhs_np)
    if rank == 0:
        print(json.dumps(line), flush=True)
    plan.close()
    replicas.finish(world)


def serving_1mp(args) -> dict:
    """Served latency of 1 MP requests: ready 1024 x 1024 Neumann systems (blob
    gradient fields) from pinned host memory at 100 req/s, open-loop Poisson
    arrivals, through the continuous-batching server; latency from the scheduled
    arrival to the solution on the host (upload, solve to 1e-8, download)."""
    from gradient_domain_b200 import loadgen
    from gradient_domain_b200.serving import GpuBackend, PoissonServer
    with PoissonServer(GpuBackend(sweeps=args.sweeps), workers=3) as server:
        r = loadgen.latency_1mp(server, requests=args.requests_1mp, rate=100.0)
        server.backend.pool.clear()
    return {"workload": "1024x1024x1 Neumann systems, 100 req/s open-loop Poisson arrivals",
            "requests": r.requests, "p50_ms": r.p50_ms, "p99_ms": r.p99_ms,
            "solves_per_s": r.solves_per_s, "converged": r.converged, "batches": r.batches,
            "latency": "scheduled arrival to the solution on the host: pinned upload, "
                       "solve to a 1e-8 true relative residual, download",
            "target_p99_ms": 5.0}


def serve_main(args) -> None:
    """`--config serve`: the open-loop serving benchmark.  `--requests` requests per
    offered load (default 20000), each built from its own seed (kind uniform over
    composite / flatten / tone-map, side log-uniform in [256, 4096]); p50 / p99
    latency and solves/s per load, plans built, the 1 MP latency, and the plain
    per-request FP64 GPU solve (exact-size plan per request, no reuse) on a sample
    of the same stream."""
    import torch

    from gradient_domain_b200 import loadgen
    from gradient_domain_b200.serving import GpuBackend, PoissonServer
    torch.cuda.set_device(0)
    t0 = time.perf_counter()
    cv = loadgen.Canvases(side=4096, seed=41).build()

    def stream(base):
        return lambda i: loadgen.build(loadgen.describe(base + i, cv.side), cv)

    out = {"metric": "served p50/p99 latency", "unit": "ms", "config": {
        "workload": "open-loop Poisson arrivals; per-request seeds: kind uniform over "
                    "composite / flatten / tone-map, side log-uniform 256-4096",
        "requests_per_rate": args.requests, "rates": args.rates, "hbm_fraction": 0.8,
        "canvas_seconds": round(time.perf_counter() - t0, 2)}}
    with PoissonServer(GpuBackend(sweeps=args.sweeps), workers=3) as server:
        out["budget_gb"] = round(server.budget / 1e9, 1)
        warm = loadgen.run_load(server, stream(10 ** 8), args.warm_requests, 100.0, seed=1)
        out["warm_up"] = {"requests": warm.requests, "plans_built": warm.extra.get("plans_built")}
        loads = []
        for k, rate in enumerate(args.rates):
            r = loadgen.run_load(server, stream((k + 1) * 10 ** 7), args.requests, rate,
                                 seed=int(rate))
            loads.append(r.__dict__)
            print(json.dumps({"load": r.__dict__}), flush=True)
        out["loads"] = loads
        r1 = loadgen.latency_1mp(server, requests=args.requests_1mp, rate=100.0)
        out["one_mp"] = r1.__dict__
        server.backend.pool.clear()
    # the plain per-request FP64 GPU solve: one worker, one request per batch, a plan of
    # the request's exact size built, solved once and freed, no graph
    sample = [loadgen.build(loadgen.describe(10 ** 7 + i, cv.side), cv)
              for i in range(args.baseline_requests)]
    with PoissonServer(GpuBackend(sweeps=args.sweeps, precision="fp64", resident=False),
                       workers=1, max_batch_requests=1) as base:
        t0 = time.perf_counter()
        res = [base.submit(r).result() for r in sample]
        dt = time.perf_counter() - t0
    out["fp64_per_request"] = {"requests": len(sample), "solves_per_s": len(sample) / dt,
                               "converged": sum(r.converged for r in res),
                               "note": "sequential; the first requests of the rated streams"}
    print(json.dumps(out), flush=True)


def smoother_gate(n: int, hbm: float, kinds: dict, sweeps: int, reps: int = 20) -> dict:
    """The smoother against HBM: ``gd_rbgs_smooth`` (FP32, red-black Gauss-Seidel,
    multigrid.py:147-165) on an n x n grid, 1 and 2 sweeps per launch.  A launch reads u
    and b and writes the result once, 12 B/cell whatever the sweeps, so the sweep rate is
    12 k B/cell per launch time.  The fused level-0 V-cycle kernels run `sweeps` sweeps
    each inside the solve; their sweep rate is given the same way."""
    import torch

    from gradient_domain_b200 import _lib

    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(7)
    u = torch.randn((n, n), device=dev, generator=g)
    b = torch.randn((n, n), device=dev, generator=g)
    v = torch.empty_like(u)
    stream = torch.cuda.current_stream()
    fn, sh = _lib.lib().gd_rbgs_smooth, stream.cuda_stream

    def launch(i, k):
        src, dst = (u, v) if i % 2 == 0 else (v, u)
        _lib.check(fn(src.data_ptr(), dst.data_ptr(), b.data_ptr(), n, n, n, 0, 1.0, k, sh),
                   "gd_rbgs_smooth")

    out = {"kernel": "k_rbgs<float>", "grid": f"{n}x{n}", "bytes_per_cell": 12,
           "l2": "u, b and the result: 3 x 67 MB per launch, above the 126 MB L2"}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for k in (1, 2):
        for i in range(4):
            launch(i, k)
        torch.cuda.synchronize()
        e0.record(stream)
        for i in range(reps):
            launch(i, k)
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / reps
        gbs = 12 * n * n / (ms / 1e3) / 1e9
        out[f"sweeps_{k}"] = {"ms": ms, "achieved_gbs": gbs, "frac": gbs / hbm,
                              "sweep_gbs": k * gbs, "sweep_frac": k * gbs / hbm}
    fused = {}
    for kind in ("down0", "up0"):
        d = kinds.get(kind)
        if d and d["launches"]:
            t = d["ms"] / d["launches"] / 1e3
            cells_l = d["cells"] / d["launches"]
            fused[kind] = {"sweeps": sweeps, "sweep_gbs": 12 * sweeps * cells_l / t / 1e9,
                           "sweep_frac": 12 * sweeps * cells_l / t / 1e9 / hbm}
    out["fused_level0"] = fused
    return out


def dct_main(args) -> None:
    """`--config dct`: the exact DCT Neumann solve (solvers.py:224-262 on the device, this
    library's FFT kernels) on the tone-mapping workload, size x size x channels; device time
    per step (all channels), the passes' bytes against HBM, error vs the scipy oracle."""
    import torch

    from gradient_domain_b200 import workloads
    from gradient_domain_b200.solvers import DctPlan
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    rhs = workloads.tonemap_rhs(args.size, seed=1, channels=args.channels)
    n_ch, h, w = rhs.shape
    f = torch.as_tensor(rhs).to(dev)
    u = torch.empty_like(f)
    plan = DctPlan(h, w)
    stream = torch.cuda.current_stream()

    def step():
        for c in range(n_ch):
            plan.solve(f[c], u[c])

    for _ in range(max(args.warmup, 1)):
        step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        step()
    e1.record(stream)
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    hbm, peak_kind = peaks()
    cells = n_ch * h * w
    line = {"config": {"workload": f"dct-neumann {h}x{w}x{n_ch}", "kernels": "k_rows_*, "
                       "k_cols_*, k_irows_* (three passes per channel)"},
            "ms_per_step": ms, "mpix_s": cells / (ms / 1e3) / 1e6,
            "bytes_per_cell": {"algorithmic": 16, "passes": 48},
            "hbm_frac_of_passes": 48 * cells / (ms / 1e3) / 1e9 / hbm, "peak_gbs": hbm,
            "peak_source": peak_kind}
    if not args.no_cpu:
        from oracle import solvers as osolvers
        ref = osolvers.solve_neumann(rhs[0], workers=os.cpu_count())
        line["rel_l2_err_vs_fp64_oracle_channel0"] = float(
            np.linalg.norm(u[0].cpu().numpy() - ref) / np.linalg.norm(ref))
    print(json.dumps({"dct": line}), flush=True)


def autotune_main(args) -> None:
    """Tune the headline plan (size x size x channels Neumann) from its defaults on its own
    right-hand sides, into a cache file of its own, and print the search."""
    import tempfile

    import torch

    from gradient_domain_b200 import autotune, workloads
    from gradient_domain_b200.plan import Instance, SolveParams

    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    rhs_np = workloads.tonemap_rhs(args.size, seed=1, channels=args.channels)
    rhs = [torch.as_tensor(r).to(dev) for r in rhs_np]
    insts = [Instance(args.size, args.size, "neumann", True) for _ in range(len(rhs))]
    params = SolveParams(tolerance=args.tol, sweeps=args.sweeps, reliable_delta=args.delta)
    path = os.path.join(tempfile.mkdtemp(), "autotune.json")
    t0 = time.perf_counter()
    tuned = autotune.tune(insts, params, rhs=rhs, reps=max(args.steps, 3), path=path,
                          force=True, scale=-1.0)
    with open(path) as fh:
        entry = json.load(fh)[autotune.tune_key(insts, params)]
    print(json.dumps({"autotune": {
        "workload": f"tonemap-neumann {args.size}x{args.size}x{len(rhs)}", "key":
        autotune.tune_key(insts, params), "default_ms": entry["default_ms"], "tuned_ms": entry["ms"],
        "choice": {k: getattr(tuned, k) for k, _ in autotune.SPACE}, "trials": entry["trials"],
        "seconds": time.perf_counter() - t0}}), flush=True)


def _timed_steps(step, steps, warmup, world, dev):
    """Warm up, then device-time exactly `steps` calls of step() (max over ranks)."""
    import torch
    from gradient_domain_b200 import replicas
    for _ in range(warmup):
        out = step()
    replicas.barrier(world)
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        out = step()
    e1.record(stream)
    torch.cuda.synchronize()
    return replicas.max_over_ranks(e0.elapsed_time(e1) / steps, world, dev), out


def composite(args) -> None:
    """Masked seamless compositing, 2048 x 2048 x 3, star-polygon selection, tolerance 1e-8."""
    import torch
    from gradient_domain_b200 import replicas
    world, rank, local = dist_setup()
    torch.cuda.set_device(local)
    replicas.init(world)
    import gradient_domain_b200 as gd
    from gradient_domain_b200 import workloads
    from gradient_domain_b200.plan import Instance, PoissonPlan, SolveParams
    dev = torch.device("cuda", local)
    size = args.size if args.size != 4096 else 2048
    src, tgt, mask = workloads.composite_case(size, seed=replicas.replica_seed(2, rank))
    f_np, unk_np, win = workloads.masked_system(src, tgt, mask)
    n_ch, hb, wb = f_np.shape
    unknowns = int(unk_np.sum())
    f = torch.as_tensor(f_np).to(dev)
    x = torch.empty_like(f)
    unk = torch.as_tensor(unk_np.astype(np.uint8)).to(dev)
    plan = PoissonPlan([Instance(hb, wb, "masked") for _ in range(n_ch)],
                       SolveParams(tolerance=args.tol, sweeps=args.sweeps,
                                   reliable_delta=args.delta, zero_start=True))

    def step():
        for k in range(n_ch):
            plan.set_mask(k, unk)
        plan.prepare()
        return plan.solve(list(f), list(x), scale=1.0)

    ms, res = _timed_steps(step, args.steps, args.warmup, world, dev)
    # per-kernel event durations from a second pass on direct launches
    plan.set_profiling(True)
    ms_prof, _ = _timed_steps(step, args.steps, 0, world, dev)
    kt = plan.kernel_times()
    plan.set_profiling(False)
    value = replicas.aggregate_rate(unknowns * n_ch, world, ms / 1e3) / 1e6
    # end to end: the public seamless_clone from host arrays (field, RHS and copies included);
    # the warm-up calls build the cached plan and its graph and fill the pinned-memory cache
    for _ in range(args.warmup):
        gd.seamless_clone(src, tgt, mask, (0, 0), domain="mask", tolerance=args.tol)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e2e_steps = max(1, args.steps // 2)
    for _ in range(e2e_steps):
        out, reps = gd.seamless_clone(src, tgt, mask, (0, 0), domain="mask", tolerance=args.tol)
    e2e_ms = (time.perf_counter() - t0) / e2e_steps * 1e3

    line = {
        "metric": METRIC, "value": value, "unit": "Mpix/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "fp32/fp64-mixed", "data": "synthetic",
        "config": {"workload": f"composite-masked {size}x{size}x{n_ch}", "unknowns": unknowns,
                   "grid": [hb, wb], "tolerance": args.tol, "sweeps": args.sweeps,
                   "unit_note": "Mpix/s counts unknown pixels x channels"},
        "iterations": [r.iterations for r in res],
        "relative_residual": max(r.relative_residual for r in res),
        "converged": all(r.converged for r in res),
        "e2e": {"value": unknowns * n_ch / (e2e_ms / 1e3) / 1e6, "unit": "Mpix/s",
                "ms_per_step": e2e_ms, "h2d_bytes_per_step": int(src.nbytes + tgt.nbytes + mask.nbytes),
                "d2h_bytes_per_step": int(tgt.nbytes)},
        "kernel_ms_per_step": {k: v["ms"] / args.steps for k, v in kt.items() if v["launches"]},
        "profiled_pass_ms_per_step": ms_prof,
    }
    if rank == 0 and world == 1 and not args.no_cpu:
        from oracle import poisson as op
        # CPU baseline and oracle: the reference's SuperLU masked solve on one channel
        field, placed, target = op.clone_field(src[..., :1], tgt[..., :1], mask, (0, 0), "import")
        t0 = time.perf_counter()
        ref, _ = op.solve_masked(field, target[..., 0], placed)
        dt = time.perf_counter() - t0
        got = out[..., 0]
        inner = np.zeros_like(mask)
        inner[1:-1, 1:-1] = mask[1:-1, 1:-1]
        err = float(np.linalg.norm(got[inner] - ref[inner]) / np.linalg.norm(ref[inner]))
        line["rel_l2_err_vs_splu_oracle_channel0"] = err
        line["cpu_baseline"] = {"value": unknowns / dt / 1e6, "unit": "Mpix/s", "cores": 1,
                                "kind": "port",
                                "sample": f"1 channel, SuperLU factorisation + solve of "
                                          f"{unknowns} unknowns (restated solve_masked), {dt:.1f} s"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    plan.close()
    replicas.finish(world)


def batch(args) -> None:
    """256 uneven images (1 or 3 channels; Neumann blobs or masked polygons) in one plan."""
    import torch
    from gradient_domain_b200 import replicas
    world, rank, local = dist_setup()
    torch.cuda.set_device(local)
    replicas.init(world)
    from gradient_domain_b200 import workloads
    from gradient_domain_b200.plan import Instance, PoissonPlan, SolveParams
    dev = torch.device("cuda", local)
    items = workloads.batch_instances(args.count, seed=replicas.replica_seed(3, rank))
    insts, fs, xs, masks = [], [], [], []
    for it in items:
        c, h, w = it["f"].shape
        for k in range(c):
            insts.append(Instance(h, w, it["boundary"], it["boundary"] == "neumann"))
            fs.append(torch.as_tensor(np.ascontiguousarray(it["f"][k])).to(dev))
            masks.append(torch.as_tensor(it["unknown"].astype(np.uint8)).to(dev)
                         if it["boundary"] == "masked" else None)
    xs = [torch.empty_like(t) for t in fs]
    cells = sum(t.numel() for t in fs)
    plan = PoissonPlan(insts, SolveParams(tolerance=args.tol, sweeps=args.sweeps,
                                          reliable_delta=args.delta, zero_start=True))
    for k, m in enumerate(masks):
        if m is not None:
            plan.set_mask(k, m)
    plan.prepare()

    def step():
        return plan.solve(fs, xs, scale=1.0)

    ms, res = _timed_steps(step, args.steps, args.warmup, world, dev)
    value = replicas.aggregate_rate(cells, world, ms / 1e3) / 1e6
    its = [r.iterations for r in res]

    line = {
        "metric": METRIC, "value": value, "unit": "Mpix/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "fp32/fp64-mixed", "data": "synthetic",
        "config": {"workload": f"batch {args.count} images / {len(insts)} instances, "
                               f"sides 64-2048, neumann + masked", "cells": cells,
                   "tolerance": args.tol, "graph": True},
        "iterations": {"min": min(its), "max": max(its), "mean": float(np.mean(its))},
        "converged": sum(r.converged for r in res), "instances": len(res),
        "max_relative_residual": max(r.relative_residual for r in res),
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    plan.close()
    replicas.finish(world)


def main():
    ap = argparse.ArgumentParser(description=__doc__.splitlines()[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--size", type=int, default=4096)
    ap.add_argument("--tol", type=float, default=1e-8)
    ap.add_argument("--sweeps", type=int, default=2)
    ap.add_argument("--delta", type=float, default=1e-4,
                    help="residual drop between FP64 refreshes (mixed precision)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the oracle and CPU baseline")
    ap.add_argument("--no-port", action="store_true",
                    help="skip the literal GPU port of the reference mgcg")
    ap.add_argument("--no-tune", action="store_true",
                    help="headline plan with --sweeps and default geometry instead of the "
                         "autotuner's choice")
    ap.add_argument("--channels", type=int, default=3)
    ap.add_argument("--solve-only", action="store_true",
                    help="only the mixed-precision solves (small profiling runs): no FP64 plan, "
                         "no end-to-end leg, no oracle")
    ap.add_argument("--config", choices=["tonemap", "composite", "batch", "serve", "smoother",
                                         "autotune", "dct"],
                    default="tonemap", help="workload (default: the headline tone-mapping case)")
    ap.add_argument("--count", type=int, default=256, help="images in the batch workload")
    ap.add_argument("--rates", type=float, nargs="+", default=[200.0, 1000.0, 5000.0],
                    help="serving: offered loads in requests per second")
    ap.add_argument("--requests", type=int, default=20000, help="serving: requests per load")
    ap.add_argument("--requests-1mp", type=int, default=300,
                    help="serving: 1 MP requests for the latency target")
    ap.add_argument("--warm-requests", type=int, default=300,
                    help="serving: warm-up requests before the rated loads")
    ap.add_argument("--baseline-requests", type=int, default=60,
                    help="serving: requests of the per-request FP64 baseline")
    ap.add_argument("--no-serve", action="store_true",
                    help="skip the 1 MP serving latency of the default line")
    ap.add_argument("--autotune-cache", default=None,
                    help="autotuner cache file for plans built with unset knobs (default: a "
                         "fresh empty file, so no earlier tuning changes the measured plans)")
    args = ap.parse_args()
    os.environ["GD_AUTOTUNE_CACHE"] = args.autotune_cache or os.path.join(
        tempfile.mkdtemp(prefix="gd_autotune_bench_"), "autotune.json")
    if args.impl == "reference":
        reference_arm(args)
    elif args.config == "composite":
        composite(args)
    elif args.config == "batch":
        batch(args)
    elif args.config == "autotune":
        autotune_main(args)
    elif args.config == "dct":
        dct_main(args)
    elif args.config == "smoother":
        import torch
        torch.cuda.set_device(0)
        hbm, peak_kind = peaks()
        line = smoother_gate(args.size, hbm, {}, args.sweeps, reps=max(args.steps, 1))
        line["peak_source"] = peak_kind
        print(json.dumps({"smoother": line}), flush=True)
    elif args.config == "serve":
        serve_main(args)
    else:
        ours(args)


if __name__ == "__main__":
    main()
