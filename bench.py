"""Benchmark of the 2DENSE hot path on GB300: FP64 WENO5-RK3 cell-updates per second.

Workload (default): double Mach reflection, 1920x480 cells, characteristic-wise AdaWENO with
Roe eigenvectors and GLF splitting (scheme 105, delta 0.5), TVD-RK3 at CFL 0.5, FP64 -- the
configuration the headline metric is quoted on. A "step" is one full TVD-RK3 time step (three
right-hand-side evaluations and stage updates) of the whole grid; one cell-update is one interior
cell advanced one step.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--workload ...]

Reported on one JSON line (rank 0):
  value        cell-updates/s with the state resident in HBM, each timed step bracketed by CUDA
               events on the solver's own stream, L2 flushed (256 MiB write) between steps;
  e2e          the same metric through the C ABI with host buffers: every step uploads the state
               from pinned host memory (dense_upload), advances one step (dense_steps) and reads
               the state back (dense_download);
  roofline     the dominant kernel (the xi-direction flux sweep) against the FP64 peak measured
               live on this GPU (dense_measure_fp64, an FMA-throughput probe): achieved = the
               reference algorithm's FLOPs for that sweep per launch / its mean CUDA-event time (no
               bound: the reconstructions are done in integers);
  cpu_baseline the CPU oracle (a line-faithful C++ restatement of the reference, OpenMP) on
               this host's cores, on a bounded sample of the same workload.
With --impl reference the CPU restatement of the reference (the Fortran itself cannot be built
without a Fortran compiler) is timed on all host threads instead, on the same workload.
N > 1 (torchrun) runs independent replicas, one per GPU: the path has no exchange step.
"""
from __future__ import annotations

import argparse
import ctypes
import importlib
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOADS = {
    # name: (benchmark, splitting, recon, ni, nj, description, flop key)
    "dmr": (5, 105, 0, 1920, 480, "double Mach reflection 1920x480, AdaWENO (105), CFL 0.5",
            "C2 DMR 1920x480 AdaWENO"),
    "ivc": (11, 101, 253, 200, 200, "isentropic vortex 200x200 periodic, LLF + WENO-JS5, CFL 0.5",
            "C1 IVC 200x200 LLF+WENO-JS5"),
    "rt": (13, 104, 0, 256, 1024, "Rayleigh-Taylor 256x1024 reflective sides, characteristic "
           "WENO-Z + GLF (104), CFL 0.5", "C3 RT 256x1024 CH"),
}
METRIC = "FP64 WENO5-RK3 cell-updates/s"
UNIT = "cell-updates/s"
# what the profiles show the sweeps to be bound by; "peak" and "frac" are the FP64 pipe's
BOUND = "integer pipes and issue"


def dist_info():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def load_flops(key):
    with open(os.path.join(ROOT, "tests", "golden", "flop_counts.json")) as f:
        return json.load(f)["bench"][key]


class Clocks:
    """nvidia-smi sampling of SM clock and throttle reasons during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.out = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (OSError, FileNotFoundError):
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.out = self.proc.communicate(timeout=5)[0]
            except subprocess.TimeoutExpired:
                self.proc.kill()
                self.out = self.proc.communicate()[0]

    def summary(self):
        if not self.out:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.out.strip().splitlines():
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = float(parts[2])
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        busy = [s for s in sm if smax and s > 0.5 * smax] or sm
        return {"sm_mhz": statistics.median(busy) if busy else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


def max_over_ranks(x: float) -> float:
    """Max of x over the ranks of the default process group (x itself when there is none): the
    timed region of N replicas ends when the slowest rank ends."""
    import torch
    import torch.distributed as dist
    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return x
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_value(cells: int, steps: int, world: int, total_ms: float) -> float:
    """Whole-job cell-updates/s of `world` replicas, each advancing `cells` cells `steps` steps,
    over the slowest rank's time."""
    return cells * steps * world / (total_ms * 1e-3)


def wl_t_start(args) -> float:
    """Start time of the timed steps: the midpoint (t = 0.1) of the reference's double Mach
    reflection run to t = 0.2 for the AdaWENO workload, whose cost depends on the flow; t = 0
    for the others, whose cost does not."""
    if args.t_start >= 0:
        return args.t_start
    return 0.1 if args.workload == "dmr" else 0.0


def wl_config(args, wl) -> dict:
    """The workload as both arms name it (the same dict in the GPU line and the reference arm's
    line): grid, scheme, the nominal start time of the timed steps and how each arm treats L2."""
    bench, split, recon, ni, nj, desc, _ = wl
    return {"workload": desc, "benchmark": bench, "splitting": split, "recon": recon,
            "ni": ni, "nj": nj, "cells": ni * nj, "t_start": wl_t_start(args),
            "start": "the setup advanced by the solver under test to t_start (untimed), then the "
                     "warm-up steps",
            "l2": "GPU arm: flushed between timed steps (256 MiB write); CPU arm: not applicable"}


def parity_check(cfg_tuple, state, gpu_cons) -> dict:
    """Relative L-inf error per conserved field (density, momentum vector, energy; the largest
    of the three) of one GPU step against one step of the CPU oracle's parity build from the same
    state bits."""
    from oracle import oracle as orc
    bench, split, recon, ni, nj, desc, _ = cfg_tuple
    cfg = orc.default_config(ni=ni, nj=nj, benchmark=bench, splitting=split, recon=recon, cfl=0.5,
                             var_eps=5.0, var_xc=5.0, var_yc=5.0)
    o = orc.OracleSolver(cfg)
    cons, prim, t, step, dt = state
    o.set_state(cons, prim)
    o.set_time(t, step, dt)
    o.steps(1)
    ref = o.get_state()[0][4:-4, 4:-4]
    got = gpu_cons[4:-4, 4:-4]
    errs = []
    for fields in ([0], [1, 2], [3]):
        d = np.sqrt(sum((got[..., v] - ref[..., v]) ** 2 for v in fields))
        n = np.sqrt(sum(ref[..., v] ** 2 for v in fields))
        errs.append(float(d.max() / max(n.max(), 1e-300)))
    return {"rel_linf": max(errs), "tolerance": 1e-12, "pass": max(errs) <= 1e-12,
            "what": "one step of the timed kernels from the first timed step's start state against "
                    "the CPU oracle (parity build) from the same bits"}


def cpu_baseline(cfg_tuple, steps: int, state=None, t_start: float = 0.0, one_thread_steps: int = 0,
                 warmup: int = 1):
    """Time the CPU oracle (OpenMP, all host threads) on the workload, from `state`
    (cons, prim, t, step, dt) when given, else from the setup advanced to t_start and then
    `warmup` steps."""
    from oracle import oracle as orc
    bench, split, recon, ni, nj, desc, _ = cfg_tuple
    cfg = orc.default_config(ni=ni, nj=nj, benchmark=bench, splitting=split, recon=recon, cfl=0.5,
                             var_eps=5.0, var_xc=5.0, var_yc=5.0)
    o = orc.OracleSolver(cfg, timed=True)
    if state is not None:
        cons, prim, t, step, dt = state
        o.set_state(cons, prim)
        o.set_time(t, step, dt)
    elif t_start > 0:
        o.steps(10 ** 7, t_end=t_start)
    o.steps(max(1, warmup))  # warm-up
    t_exact = o.scalars()["time"]
    t0 = time.perf_counter()
    o.steps(steps)
    el = time.perf_counter() - t0
    lib = orc.load(True)
    threads = lib.oracle_threads()
    out = {"value": ni * nj * steps / el, "unit": UNIT, "cores": threads, "kind": "port",
           "sample": f"{desc}: {steps} step(s) of the C++ restatement of the reference "
                     f"(OpenMP, {threads} threads, gcc -O2), after {max(1, warmup)} warm-up step(s)",
           "seconds": el, "t_start_exact": t_exact}
    if one_thread_steps > 0:  # the same code on one core, a shorter sample of the same state
        lib.oracle_set_threads(1)
        t0 = time.perf_counter()
        o.steps(one_thread_steps)
        el1 = time.perf_counter() - t0
        lib.oracle_set_threads(threads)
        out["one_thread"] = {"value": ni * nj * one_thread_steps / el1, "unit": UNIT, "cores": 1,
                             "steps": one_thread_steps}
    return out


def run_reference_arm(args, wl):
    rank, world, _ = dist_info()
    if rank != 0:
        return
    steps = max(1, args.steps)
    warmup = max(0, args.warmup)
    # the oracle first advances itself (untimed) to the start time of the GPU arm's timed steps,
    # then takes the same warm-up and timed steps as the GPU arm
    cb = cpu_baseline(wl, steps=steps, t_start=wl_t_start(args), warmup=warmup)
    line = {"impl": "reference", "metric": METRIC, "value": cb["value"], "unit": UNIT,
            "n_gpus": args.gpus, "steps": steps, "warmup": warmup,
            "ms_per_step": 1e3 * cb["seconds"] / steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": wl_config(args, wl), "t_start_exact": cb["t_start_exact"],
            "cpu_baseline": {k: cb[k] for k in ("value", "unit", "cores", "kind", "sample")},
            "e2e": {"value": cb["value"], "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "note": "the reference is Fortran; no Fortran compiler exists on this image or the GPU "
                    "box, so the reference arm times its line-faithful C++ restatement"}
    print(json.dumps(line), flush=True)


def batched_configs(dense, n: int = 512, seed: int = 2024, nmin: int = 64, nmax: int = 512):
    """The batched workload: n square periodic instances, N drawn uniformly from
    {nmin, nmin+32, ..., nmax} (64..512 by default); even instances a translating vortex with
    strength U[1,5] and centre offset U[-1,1]^2, odd ones a Mach 1.2 shock into a density-3
    interface of amplitude U[0.01,0.05]; LLF + WENO-Z5, CFL 0.5, each with its own CFL time step."""
    rng = np.random.default_rng(seed)
    sizes = list(range(nmin, nmax + 1, 32))
    cfgs = []
    for k in range(n):
        N = int(rng.choice(sizes))
        if k % 2 == 0:
            cfgs.append(dense.config_default(ni=N, nj=N, benchmark=11, splitting=101, recon=255, cfl=0.5,
                                             var_eps=float(rng.uniform(1, 5)),
                                             var_xc=5 + float(rng.uniform(-1, 1)),
                                             var_yc=5 + float(rng.uniform(-1, 1))))
        else:
            cfgs.append(dense.config_default(ni=N, nj=N, benchmark=14, splitting=101, recon=255, cfl=0.5,
                                             var_amp=float(rng.uniform(0.01, 0.05))))
    return cfgs


def run_batched(args, dense, lib):
    """Batched form vs looped plain solves of the same instances on the same GPU."""
    import torch
    at = importlib.import_module("2dense_gb300.autotune")
    n = args.batch
    cfgs = batched_configs(dense, n, seed=args.seed, nmin=args.batch_nmin, nmax=args.batch_nmax)
    setups = [dense.init_general(c) for c in cfgs]
    cfgs = [s[0] for s in setups]
    cells = sum(c.ni * c.nj for c in cfgs)
    sched, info = at.tune(cfgs, setups=setups, steps=2, reps=2)
    if args.batch_mode != "auto":
        sched = tuple(sched[:3]) + (1 if args.batch_mode == "persistent" else 0,)
    b = dense.BatchSolver(cfgs)
    for i, (c, cons, prim, x, y) in enumerate(setups):
        b.upload(i, cons, prim, x, y)
    b.set_schedule(*sched)
    b.steps(args.warmup)
    stream = torch.cuda.ExternalStream(b.stream())
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    launches0 = b.launch_count()
    torch.cuda.synchronize()
    wall0 = time.perf_counter()
    with Clocks(0) as clk:
        ev0.record(stream)
        b.steps(args.steps, wait=False)
        ev1.record(stream)
        torch.cuda.synchronize()
    wall = time.perf_counter() - wall0
    ms = ev0.elapsed_time(ev1)
    launches = b.launch_count() - launches0
    value = cells * args.steps / (ms * 1e-3)
    status = b.status()
    # Looped plain solves of the same instances, each its own handle advanced in turn through the
    # same warm-up and timed steps (the timed steps of all instances summed), and every instance's
    # final state compared bit for bit with the batch's.
    loop_s, same = 0.0, 0
    for i, (c, cons, prim, x, y) in enumerate(setups):
        with dense.Solver(c) as s:
            s.upload(cons, prim, x, y)
            s.steps(args.warmup)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            s.steps(args.steps)
            loop_s += time.perf_counter() - t0
            if np.array_equal(s.download(False), b.download(i)):
                same += 1
    b.close()
    loop_steps = args.steps
    looped = cells * loop_steps / loop_s
    fl = json.load(open(os.path.join(ROOT, "tests", "golden", "flop_counts.json")))["schemes"]["LLF+WENO-Z5"]
    peak = ctypes.c_double()
    lib.dense_measure_fp64(0, ctypes.byref(peak))
    sizes = sorted(c.ni for c in cfgs)
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"batched: {n} periodic instances, N in {args.batch_nmin}..{args.batch_nmax} "
                                   f"(seed {args.seed}), "
                                   "vortex / Richtmyer-Meshkov, LLF + WENO-Z5, CFL 0.5",
                       "instances": n, "cells": cells, "n_min": sizes[0], "n_max": sizes[-1],
                       "l2": "inputs larger than L2 (about 1.7 GB per state copy)"},
            "batched": {"schedule": {"xi_variant": sched[0], "eta_variant": sched[1], "order": sched[2],
                                     "launch": "one persistent launch per step" if sched[3] == 1
                                     else "one launch per phase"},
                        "autotune": {"cached": info["cached"], "trials_s": info["trials"]}},
            "looped_plain": {"value": looped, "unit": UNIT, "steps_per_instance": loop_steps,
                             "api": "one dense_create handle per instance, dense_steps in turn; "
                                    "host wall time of the timed steps, summed over instances"},
            "speedup_vs_looped": value / looped,
            "identical_results": {"checked": n, "bitwise_equal": same,
                                  "what": "every instance's state after the warm-up and timed steps, "
                                          "batched against its own plain solve"},
            "gpu_launches": launches,
            "roofline": {"bound": BOUND, "achieved": fl["flops_per_cell_update"] * value / 1e12,
                         "peak": peak.value / 1e12, "unit": "TFLOP/s",
                         "frac": fl["flops_per_cell_update"] * value / peak.value,
                         "flops_per_cell_update": fl["flops_per_cell_update"], "traffic": None},
            "clocks": clk.summary(), "status_flags": status, "wall_s_timed_region": wall}
    print(json.dumps(line), flush=True)


FD_CRITERION = ("Richardson-extrapolated central differences (h = 1e-6, 2e-6) within 1e-6 relative of the "
                "adjoint in every direction, with the cells of the wave-speed maxima unchanged")
# AdaWENO switches each (face, sign) between two reconstructions at theta = delta: the discrete
# loss is smooth only between switches, and over a 400-step run a 1e-6 step in a parameter flips
# some of its hundreds of millions of decisions, whose jumps dominate a central difference. The
# adjoint is the derivative with the switches held (like the time step's maxima), checked
# against autograd with the same switches (tests/test_gpu_adjoint.py); the differences are
# reported, not judged.
FD_NOT_A_CRITERION_105 = ("not a criterion for AdaWENO (105): its per-face switch makes the loss piecewise "
                          "smooth, and a 1e-6 step flips some of the run's switches; the gradient is checked "
                          "against autograd with the switches held")
# the adjoint workload's schemes: (splitting, recon, name, FLOP-count key)
ADJ_SCHEMES = {"llf-js": (101, 253, "LLF + WENO-JS5", "LLF+WENO-JS5"),
               "char": (104, 0, "characteristic WENO-Z + GLF (104)", "CH (104)"),
               "adaweno": (105, 0, "AdaWENO + GLF (105), DELTA 0.5", "AdaWENO (105) smooth vortex")}


def run_adjoint(args, dense, lib):
    """Gradient of a vortex run through the discrete adjoint: 256x256 periodic vortex, LLF +
    WENO-JS5 (or the characteristic scheme 104 / AdaWENO 105: --adj-scheme char / adaweno), CFL 0.4, 400 steps,
    checkpoints every 20. Loss 1/2 ||rho(T) - rho_target||^2, the
    target from the unperturbed vortex (eps 5, centre (5,5)); the run starts from that vortex plus
    a seeded Gaussian density perturbation of amplitude 1e-3. Gradients w.r.t. the perturbation
    field and (eps, xc, yc), checked against central differences (h = 1e-6) of the CUDA forward."""
    import torch
    adjm = importlib.import_module("2dense_gb300.adjoint")
    ni = args.ni or 256
    nj = args.nj or 256
    n, k = args.adj_steps, 20
    split, recon, scheme, fl_key = ADJ_SCHEMES[args.adj_scheme]
    cfg = dense.init_general(dense.config_default(ni=ni, nj=nj, benchmark=11, splitting=split, recon=recon,
                                                  cfl=0.4, var_eps=5.0, var_xc=5.0, var_yc=5.0))[0]
    adj = adjm.Adjoint(cfg, checkpoint_every=k)
    Step = adjm.AdjointStep
    gen = torch.Generator().manual_seed(args.seed)
    drho_h = (1e-3 * torch.randn(nj, ni, generator=gen, dtype=torch.float64)).pin_memory()
    drho0 = drho_h.cuda()
    target = adj.forward(adjm.vortex_state(cfg, 5.0, 5.0, 5.0), n)[0].clone()
    theta0 = torch.tensor([5.0, 5.0, 5.0], dtype=torch.float64, device="cuda")

    def loss_fn(theta, drho):
        uT = Step.apply(adjm.vortex_state(cfg, theta[0], theta[1], theta[2], drho), adj, n)
        return 0.5 * ((uT[0] - target) ** 2).sum()

    def grads(theta, drho):
        th = theta.detach().clone().requires_grad_(True)
        dr = drho.detach().clone().requires_grad_(True)
        loss = loss_fn(th, dr)
        g_th, g_dr = torch.autograd.grad(loss, [th, dr])
        return float(loss.detach()), g_th, g_dr

    for _ in range(max(1, args.warmup)):
        grads(theta0, drho0)
    torch.cuda.synchronize()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    reps = max(1, args.steps)
    fwd_ms, bwd_ms = [], []
    launches0 = adj.launch_count()
    with Clocks(0) as clk:
        for _ in range(reps):
            th = theta0.clone().requires_grad_(True)
            dr = drho0.clone().requires_grad_(True)
            ev[0].record()
            loss = loss_fn(th, dr)
            ev[1].record()
            g_th, g_dr = torch.autograd.grad(loss, [th, dr])
            ev[2].record()
            torch.cuda.synchronize()
            fwd_ms.append(ev[0].elapsed_time(ev[1]))
            bwd_ms.append(ev[1].elapsed_time(ev[2]))
    launches = (adj.launch_count() - launches0) // reps
    fwd, bwd = statistics.median(fwd_ms), statistics.median(bwd_ms)
    # the plain solver over the same steps, no checkpoints
    c, cons, prim, x, y = dense.init_general(cfg)
    with dense.Solver(c) as s:
        s.upload(cons, prim, x, y)
        s.steps(2)
        stream = torch.cuda.ExternalStream(s.stream())
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(stream)
        s.steps_async(n)
        e1.record(stream)
        torch.cuda.synchronize()
        plain_ms = e0.elapsed_time(e1)
    # end to end: the perturbation from pinned host memory, forward, backward, gradients to host
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    dr = drho_h.cuda(non_blocking=True).requires_grad_(True)
    th = theta0.clone().requires_grad_(True)
    g1, g2 = torch.autograd.grad(loss_fn(th, dr), [th, dr])
    g_host = g2.cpu(), g1.cpu()
    e2e_s = time.perf_counter() - t0
    # central differences in eps, xc, yc and along a smooth direction of the perturbation field
    # (a Gaussian bump): FD(h) at h = 1e-6, FD(2h), and their Richardson extrapolation
    # (4 FD(h) - FD(2h))/3, which removes the h^2 term (the larger step keeps the rounding noise
    # of the 400-step runs, about 1e-12 of the loss, below the bar). Valid where the cells of the
    # wave-speed maxima do not change between the runs (dt = cfl/(max/dx + max/dy) has a kink
    # there).
    loss0, g_th, g_dr = grads(theta0, drho0)
    trace0 = adj.argmax().copy()
    xs = (torch.arange(ni, dtype=torch.float64, device="cuda") + 0.5) * 10.0 / ni
    ys = (torch.arange(nj, dtype=torch.float64, device="cuda") + 0.5) * 10.0 / nj
    Yg, Xg = torch.meshgrid(ys, xs, indexing="ij")
    bump = torch.exp(-((Xg - 3.0) ** 2 + (Yg - 6.0) ** 2))
    h = 1e-6
    fd = {}
    for name, (dth, ddr, exact) in {
            "eps": ((1, 0, 0), None, float(g_th[0])), "xc": ((0, 1, 0), None, float(g_th[1])),
            "yc": ((0, 0, 1), None, float(g_th[2])),
            "drho_bump": ((0, 0, 0), bump, float((g_dr * bump).sum()))}.items():
        same, est = True, {}
        for hh in (h, 2 * h):
            vals = []
            for sgn in (1.0, -1.0):
                th = theta0 + sgn * hh * torch.tensor(dth, dtype=torch.float64, device="cuda")
                dr = drho0 + (sgn * hh * ddr if ddr is not None else 0.0)
                lv, _, _ = grads(th, dr)
                vals.append(lv)
                same = same and np.array_equal(adj.argmax(), trace0)
            est[hh] = (vals[0] - vals[1]) / (2 * hh)
        rich = (4 * est[h] - est[2 * h]) / 3
        rel = lambda x: abs(x - exact) / max(abs(exact), 1e-300)
        fd[name] = {"adjoint": exact, "fd_h": est[h], "fd_2h": est[2 * h], "richardson": rich,
                    "rel_err_fd_h": rel(est[h]), "rel_err_richardson": rel(rich),
                    "max_cells_unchanged": bool(same)}
    status = 0
    cells = ni * nj
    fl = json.load(open(os.path.join(ROOT, "tests", "golden", "flop_counts.json")))["schemes"][fl_key]
    peak = ctypes.c_double()
    lib.dense_measure_fp64(0, ctypes.byref(peak))
    value = cells * n / ((fwd + bwd) * 1e-3)
    line = {"metric": METRIC + " (forward + adjoint)", "value": value, "unit": UNIT, "n_gpus": 1, "steps": reps,
            "warmup": args.warmup, "ms_per_step": (fwd + bwd) / n, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"adjoint: vortex {ni}x{nj} periodic, {scheme}, CFL 0.4, {n} steps, "
                                   f"checkpoint every {k}; loss 1/2||rho(T)-rho_target||^2",
                       "ni": ni, "nj": nj, "nsteps": n, "checkpoint_every": k,
                       "l2": "state (2 MB) fits in L2; no flush: each timed rep is a 400-step chain"},
            "adjoint": {"forward_ms": fwd, "backward_ms": bwd, "plain_forward_ms": plain_ms,
                        "backward_over_forward": bwd / fwd, "backward_over_plain_forward": bwd / plain_ms,
                        "loss": loss0, "fd_check": fd, "fd_h": h,
                        "max_rel_err_fd_h": max(v["rel_err_fd_h"] for v in fd.values()),
                        "max_rel_err_richardson": max(v["rel_err_richardson"] for v in fd.values()),
                        "fd_criterion": FD_CRITERION if split != 105 else FD_NOT_A_CRITERION_105,
                        "fd_pass": None if split == 105 else
                        all(v["rel_err_richardson"] <= 1e-6 and v["max_cells_unchanged"] for v in fd.values())},
            "e2e": {"value": cells * n / e2e_s, "unit": UNIT, "h2d_bytes_per_step": drho_h.numel() * 8,
                    "d2h_bytes_per_step": (g_host[0].numel() + g_host[1].numel()) * 8,
                    "note": "perturbation field from pinned host memory, forward, backward, gradients to host"},
            "gpu_launches": launches,
            "roofline": {"bound": BOUND, "achieved": fl["flops_per_cell_update"] * cells * n / (plain_ms * 1e-3) / 1e12,
                         "peak": peak.value / 1e12, "unit": "TFLOP/s",
                         "frac": fl["flops_per_cell_update"] * cells * n / (plain_ms * 1e-3) / peak.value,
                         "of": "the plain forward's reference FLOPs", "traffic": None},
            "clocks": clk.summary(), "status_flags": status}
    adj.close()
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=None,
                    help="timed steps (default 100; 200 for the batched workload, its specified run)")
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="dmr", choices=sorted(WORKLOADS) + ["batched", "adjoint"])
    ap.add_argument("--strict", type=int, default=0)
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--cpu-steps", type=int, default=20)
    ap.add_argument("--ni", type=int, default=0, help="override the grid (smaller profiling cases)")
    ap.add_argument("--nj", type=int, default=0)
    ap.add_argument("--t-start", type=float, default=-1.0,
                    help="flow time the timed steps start from (default: 0.1 for dmr, 0 otherwise)")
    ap.add_argument("--save-state", default="", help="write the start state (npz) before warm-up")
    ap.add_argument("--load-state", default="", help="start from a state written by --save-state")
    ap.add_argument("--batch", type=int, default=512, help="instances of the batched workload")
    ap.add_argument("--seed", type=int, default=2024)
    ap.add_argument("--batch-nmin", type=int, default=64, help="smallest instance size of the batched workload")
    ap.add_argument("--batch-nmax", type=int, default=512, help="largest instance size of the batched workload")
    ap.add_argument("--batch-mode", choices=("auto", "phases", "persistent"), default="auto",
                    help="launch mode of the batched workload: the autotuner's pick, one launch per "
                         "phase, or one persistent launch per step (tiles and order tuned either way)")
    ap.add_argument("--adj-steps", type=int, default=400, help="time steps of the adjoint workload's run")
    ap.add_argument("--adj-scheme", default="llf-js", choices=sorted(ADJ_SCHEMES),
                    help="the adjoint workload's scheme: LLF + WENO-JS5 (101 + 253), characteristic (104) "
                         "or AdaWENO (105)")
    args = ap.parse_args()
    if args.steps is None:
        args.steps = 200 if args.workload == "batched" else 100
    if args.workload == "adjoint":
        if args.impl == "reference":
            rank, _, _ = dist_info()
            if rank == 0:
                print(json.dumps({"impl": "reference", "unavailable": "the reference has no derivatives; "
                                  "there is no adjoint to time"}))
            return
        import torch
        torch.cuda.set_device(0)
        dense = importlib.import_module("2dense_gb300")
        return run_adjoint(args, dense, dense.load_library())
    if args.workload == "batched":
        if args.impl == "reference":
            rank, _, _ = dist_info()
            if rank == 0:
                print(json.dumps({"impl": "reference", "unavailable": "the reference advances one block per "
                                  "process; it has no batched form to time"}))
            return
        import torch
        torch.cuda.set_device(0)
        dense = importlib.import_module("2dense_gb300")
        return run_batched(args, dense, dense.load_library())
    wl = WORKLOADS[args.workload]
    if args.ni and args.nj:
        full = f"{wl[3]}x{wl[4]}"
        wl = wl[:3] + (args.ni, args.nj, wl[5].replace(full, f"{args.ni}x{args.nj} (the {full} workload's "
                                                               f"scheme on a reduced grid)"), wl[6])
    if args.impl == "reference":
        return run_reference_arm(args, wl)

    import torch
    rank, world, local = dist_info()
    torch.cuda.set_device(local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl" if torch.cuda.is_available() else "gloo")
    dense = importlib.import_module("2dense_gb300")
    lib = dense.load_library()

    bench, split, recon, ni, nj, desc, fkey = wl
    cfg = dense.config_default(ni=ni, nj=nj, benchmark=bench, splitting=split, recon=recon,
                               cfl=0.5, strict=args.strict)
    c, cons, prim, x, y = dense.init_general(cfg)
    cells = ni * nj
    s = dense.Solver(c)
    s.upload(cons, prim, x, y)
    sp = ctypes.c_void_p()
    lib.dense_get_stream(s.h, ctypes.byref(sp))
    stream = torch.cuda.ExternalStream(sp.value)

    # The timed steps start from a developed state at t_start, produced by this solver before the
    # warm-up (AdaWENO's cost depends on how much of the flow is non-smooth).
    t_start = wl_t_start(args)
    if args.load_state:
        z = np.load(args.load_state)
        s.upload(z["cons"], z["prim"], x, y)
        s.current_time, s.current_step = float(z["t"]), int(z["step"])
        t_start = s.current_time
    while s.current_time < t_start:
        s.steps(200, t_end=t_start)
    if args.save_state:
        sc_, sp_ = s.download()
        np.savez(args.save_state, cons=sc_, prim=sp_, t=s.current_time, step=s.current_step)
    # warm-up (also builds the step graph)
    s.steps(args.warmup)
    lib.dense_set_time(s.h, s.current_time, s.current_step)
    # the state the timed steps start from, replayed below to count the work they did
    snap_cons, snap_prim = s.download()
    snap_t, snap_step, snap_dt = s.current_time, s.current_step, s.dt

    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    launches0 = s.launch_count()
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
           for _ in range(args.steps)]
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    wall0 = time.perf_counter()
    with Clocks(local) as clk:
        for k in range(args.steps):
            stream.synchronize()
            flush.fill_(float(k))  # L2 flush between timed steps (outside the events)
            torch.cuda.current_stream().synchronize()
            evs[k][0].record(stream)
            rc = lib.dense_steps_async(s.h, 1, float("inf"), 2**31 - 1)
            if rc:
                raise RuntimeError(lib.dense_last_error(s.h))
            evs[k][1].record(stream)
        torch.cuda.synchronize()
    wall = time.perf_counter() - wall0
    step_ms = [a.elapsed_time(b) for a, b in evs]
    launches = s.launch_count() - launches0
    total_ms = max_over_ranks(sum(step_ms))
    value = replica_value(cells, args.steps, world, total_ms)
    status = s.status()

    # per-kernel times of the stage, for the roofline of the dominant kernel
    prof = np.zeros((3, 4))
    reps = 5
    for r in range(reps):
        for irk in (1, 2, 3):
            ms = (ctypes.c_float * 4)()
            if lib.dense_profile_stage(s.h, irk, ms):
                raise RuntimeError(lib.dense_last_error(s.h))
            prof[irk - 1] += np.array(list(ms)) / reps
    fl = load_flops(fkey)
    peak = ctypes.c_double()
    lib.dense_measure_fp64(0, ctypes.byref(peak))
    div_rate = ctypes.c_double()
    lib.dense_measure_fp64(1, ctypes.byref(div_rate))
    xi_ms = prof[:, 1].mean()
    eta_ms = prof[:, 2].mean()
    stage_ms = prof.sum(axis=1).mean()
    # Reference-algorithm FLOPs of the timed steps. AdaWENO's work depends on the data only
    # through the branch each (interface, sign) takes: replay the timed steps from the same
    # state with the branch counters on and price each branch with the oracle's counts.
    branches = None
    if split == 105:
        ada = fl["adaweno"]
        s.upload(snap_cons, snap_prim, x, y)
        lib.dense_set_time(s.h, snap_t, snap_step)
        lib.dense_count_branches(s.h, 1)
        lib.dense_steps_async(s.h, args.steps, float("inf"), 2**31 - 1)
        cnt = (ctypes.c_ulonglong * 8)()
        lib.dense_get_branch_counts(s.h, cnt)
        lib.dense_count_branches(s.h, 0)
        cnt = [int(v) for v in cnt]
        S, C = ada["smooth_branch_flops"], ada["char_branch_flops"]
        nsteps = args.steps
        step_flops = (ada["base_per_cell_update"] * cells
                      + (S * (cnt[0] + cnt[4]) + C * (cnt[1] + cnt[5])) / nsteps)
        xi_flops = ada["base_xi_per_cell_update"] / 3.0 * cells + (S * cnt[0] + C * cnt[1]) / (3 * nsteps)
        branches = {"smooth": cnt[0] + cnt[4], "char": cnt[1] + cnt[5],
                    "char_fraction": (cnt[1] + cnt[5]) / max(1, sum(cnt[0:2]) + sum(cnt[4:6])),
                    "warps_with_char_fraction": (cnt[3] + cnt[7]) / max(1, cnt[2] + cnt[6]),
                    "smooth_branch_flops": S, "char_branch_flops": C,
                    "base_flops_per_cell_update": ada["base_per_cell_update"]}
    else:
        step_flops = fl["flops_per_cell_update"] * cells
        xi_flops = fl["flux_xi_per_cell_update"] / 3.0 * cells
    achieved = xi_flops / (xi_ms * 1e-3) / 1e12
    kname = {104: "k_flux_char<0,false>", 105: "k_flux_char<0,true>"}.get(split, "k_flux_cw<0,...>")
    roofline = {"bound": BOUND, "kernel": f"xi flux sweep ({kname})",
                "achieved": achieved, "peak": peak.value / 1e12, "unit": "TFLOP/s",
                "frac": achieved * 1e12 / peak.value,
                "frac_note": "the reference's FP64 operations over the FP64 peak, which is no bound: the default "
                             "kernels do the reconstructions in 64-bit integers beside that pipe, so it can exceed 1",
                "peak_source": "measured live: dense_measure_fp64 FMA-throughput probe on this GPU "
                               "(MEASURED_PEAKS.json has no FP64 figure)",
                "traffic": None,
                "traffic_note": "DRAM bytes need an ncu capture, which this run does not take; "
                                "the committed ncu summaries of this kernel give them",
                "whole_step": {"achieved_tflops": step_flops * value / cells / world / 1e12,
                               "frac": step_flops * value / cells / world / peak.value,
                               "flops_per_cell_update": step_flops / cells},
                "flops_per_xi_launch": xi_flops,
                "adaweno_branches": branches,
                "kernel_ms": {"bc": prof[:, 0].mean(), "flux_xi": xi_ms, "flux_eta": eta_ms,
                              "update": prof[:, 3].mean()},
                "kernel_share": {"bc": prof[:, 0].mean() / stage_ms, "flux_xi": xi_ms / stage_ms,
                                 "flux_eta": eta_ms / stage_ms, "update": prof[:, 3].mean() / stage_ms},
                "hbm": {"algorithmic_bytes_per_cell_update": 256,
                        "achieved_gbs": 256 * value / world / 1e9},
                "fp64_div_per_s": div_rate.value}

    # end to end through the C ABI with pinned host buffers
    e2e_steps = max(3, min(args.steps, 20))
    nip, njp = ni + 8, nj + 8
    pin = torch.empty(nip * njp * 4, dtype=torch.float64, pin_memory=True)
    host = pin.numpy().reshape((nip, njp, 4), order="F")
    host[...] = snap_cons
    xs, ys = np.asfortranarray(x), np.asfortranarray(y)
    dp = ctypes.POINTER(ctypes.c_double)
    hp = host.ctypes.data_as(dp)
    with dense.Solver(c) as s2:
        s2.upload(host, snap_prim, xs, ys)
        s2.current_time, s2.current_step = snap_t, snap_step
        s2.steps(1)
        tcur, scur = ctypes.c_double(s2.current_time), ctypes.c_int(s2.current_step)
        t0 = time.perf_counter()
        for k in range(e2e_steps):
            rc = lib.dense_upload(s2.h, hp, None, xs.ctypes.data_as(dp), ys.ctypes.data_as(dp))
            rc = rc or lib.dense_steps(s2.h, 1, float("inf"), 2**31 - 1, ctypes.byref(tcur),
                                       ctypes.byref(scur), None)
            rc = rc or lib.dense_download(s2.h, hp, None)
            if rc:
                raise RuntimeError(lib.dense_last_error(s2.h))
        e2e_s = time.perf_counter() - t0
    e2e = {"value": cells * e2e_steps * world / e2e_s, "unit": UNIT,
           "h2d_bytes_per_step": nip * njp * 4 * 8 + (2 * ni + nj) * 8,
           "d2h_bytes_per_step": nip * njp * 4 * 8,
           "steps": e2e_steps,
           "api": "dense_upload(cons from pinned host) + dense_steps(1) + dense_download(cons)"}

    cpu = None
    parity = None
    if rank == 0 and world == 1 and not args.no_cpu:
        snap = (snap_cons, snap_prim, snap_t, snap_step, snap_dt)
        cpu = cpu_baseline(wl, args.cpu_steps, state=snap, one_thread_steps=max(1, args.cpu_steps // 10))
        cpu.pop("seconds", None)
        cpu.pop("t_start_exact", None)
        # the timed kernels' first step from the same start state, against the oracle
        s.upload(snap_cons, snap_prim, x, y)
        s.current_time, s.current_step, s.dt = snap_t, snap_step, snap_dt
        s.steps(1)
        parity = parity_check(wl, snap, s.download(False))

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": wl_config(args, wl), "t_start_exact": snap_t, "strict": args.strict,
            "parallelism": f"replicas x{world}" if world > 1 else "single GPU",
            "e2e": e2e, "gpu_launches": launches, "roofline": roofline, "cpu_baseline": cpu,
            "parity_checked": parity,
            "clocks": clk.summary(), "status_flags": status, "wall_s_timed_region": wall}
    if rank == 0:
        print(json.dumps(line), flush=True)
    s.close()
    if world > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
