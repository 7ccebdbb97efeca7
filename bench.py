#!/usr/bin/env python
"""Benchmark of the EU3D reacting-Euler timestep on B200.

Workload: the 3-D reacting shock-bubble case, 256 x 128 x 128 nodes over
64 x 32 x 32 mm (4,194,304 cells), H2_JA919 kinetics (9 species, 19 reactions),
Mach 2.83 shock in N2 at 101.325 kPa / 300 K hitting a perturbed 2H2+O2 sphere
(radius 8 mm, centred 16 mm downstream of the shock, seed 3), fixed dt from the
reference's CFL rule at 0.25 on the initial state, 500 steps in all. Synthetic
inputs built by eu3d_cases.shock_bubble.

A step is one full timestep: RSBI ghost fill, MUSCL/AUSM flux divergence in x,
y, z with the explicit update, state recovery with Newton temperature
inversion, Nchem prediction and the adaptive trapezoid kinetics.

The timed window: each arm advances the case untimed for WINDOW_START steps,
until the shock has entered the bubble (it reaches the bubble's upstream
surface after about 160 steps and runs through the bubble gas from then on),
then warms up and times --steps steps there, then runs on to step 500. The
learned + mixed arm and the plain FP64 arm each run their own trajectory from
step 0, and their difference is stated at the end of the window and at step 500.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One JSON line on rank 0 (see the keys below). Multi-GPU runs (torchrun, one
rank per GPU) decompose one grid along x, one block of 256 x 128 x 128 nodes
per rank (the reference's MPI layout: neighbouring blocks share a node, so N
ranks hold N x 255 + 1 nodes along x over N x 64 mm): every step exchanges the
blocks' halo planes over NCCL before it runs, dt is the minimum of the blocks'
CFL steps, and per-GPU work is fixed ("scaling": "weak").

--impl reference times the reference's own CPU timestep (oracle/_ref, built from
its unmodified sources) on the same grid, cut into independent sub-boxes of
64 x 64 x 64 nodes (one host process per sub-box), and never loads this
library.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "eu3d-gpu_b200"))

import eu3d_cases as cases  # noqa: E402  (numpy only; never loads the library)

METRIC = "Mcell-steps/s reacting, learned+mixed vs plain FP64 on same B200 at ≤1e-3 Y err"
GRID = (256, 128, 128)
EXTENT = (0.0, 0.064, 0.0, 0.032, 0.0, 0.032)
# The reference's CFL rule (dx, dy only) at 0.25: its forward-Euler MUSCL/AUSM
# step goes non-finite on this case at 0.5 once the shock runs into the bubble
# (steps 120-130, FP64 and mixed alike) and at 0.35 by step 240-280; at 0.25 it
# runs the 500 steps.
CFL = 0.25
# the 1-D ZND and 2-D ODW cases run at the reference's usual 0.5
CFL_THIN = 0.5
# the config's run length, and the step at which the timed window starts (the
# shock inside the bubble)
TOTAL_STEPS = 500
WINDOW_START = 250
# Algorithmic bytes per cell-step of the flux + update kernel: 16 primitives
# read, 13 conserved read and written (FP64); FP32 primitives in mixed mode.
FLUX_BYTES = {"fp64": (16 + 26) * 8, "mixed": 16 * 4 + 26 * 8}
# DRAM bytes per cell of one launch of each flux kernel, from its ncu capture
# (dram__bytes_read.sum + dram__bytes_write.sum over the cells of the captured
# 256 x 128 x 64-node grid; the traffic scales with the cells, so it is scaled
# to the benchmark grid).
FLUX_TRAFFIC_PER_CELL = {"mixed": 274.4}  # (the FP64 kernel has no capture at that grid)
# FLOPs per row of the learned ensemble (3 members x 2 (12 256 + 256 256 + 256 256 + 256 10)).
MLP_FLOP_PER_ROW = 820224
# FP64 flops per cell-substep of the stiff kinetics (rates, trapezoid update,
# state rebuild with its temperature Newton), counted on the oracle over the
# thin RSBI case by oracle/flop_count.cpp.
F_SUB = 6017
# FP64 vector peak of a B200 (datasheet; no measured FP64 figure is available).
FP64_PEAK_TFLOPS = 37.0
# Nchem histogram bins (upper edges, inclusive)
NCHEM_BINS = (0, 1, 2, 4, 8, 16, 64, 256, 1 << 30)
# The reference arm's sub-boxes (nodes per side) tiling the grid.
REF_BOX = (64, 64, 64)


def env_int(name, default):
    try:
        return int(os.environ.get(name, default))
    except ValueError:
        return default


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return d.get("hbm_gbs", 6650.0), d.get("bf16_tflops", 1590.0), "measured"
    return 6650.0, 1590.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index):
        self.idx = str(device_index)
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(prefix="eu3d_clocks_", suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-i", self.idx, "-lms", "100"], stdout=open(self.path, "w"),
                                         stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[q] for r in rows for q in range(4) if r[5 + q].lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


# ------------------------------------------------------------------ workload

def full_axes(grid=GRID, extent=EXTENT):
    """Node coordinates (with ghosts) of the whole grid along x, y, z."""
    return tuple(cases.node_coordinates(n, extent[2 * a], extent[2 * a + 1]) for a, n in enumerate(grid))


def bubble_field(x, y, z, mw, ns, grid=GRID, extent=EXTENT, seed=3):
    """The shock-bubble primitives on the nodes x, y, z: the whole grid's
    nodes or any sub-box of them (the bubble centre is the whole grid's, so a
    sub-box gets exactly its part of the field)."""
    _, yf, zf = full_axes(grid, extent)
    scale = extent[1] / 0.064
    return cases.shock_bubble(x, y, z, mw, ns, radius=8e-3 * scale, shock_x=4e-3 * scale, standoff=16e-3 * scale,
                              center_yz=(0.5 * (yf[2] + yf[-3]), 0.5 * (zf[2] + zf[-3])), seed=seed)


def build_workload(grid):
    import eu3d
    x, y, z = full_axes(grid)
    mech = eu3d.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = bubble_field(x, y, z, mech["mw"], mech["ns"], grid=grid)
    p, cs, T, E = eu3d.initial_state(mech, *grid, *prim)
    dt = cases.cfl_dt(x, y, p[0], p[1], p[2], p[3], p[6], CFL)
    return mech, prim, (p, cs, T, E), dt


def state_dict(st):
    p, cs, T, E = st
    return {"CS": cs, "T": T, "E": E, "P": p[0], "D": p[1], "U": p[2], "V": p[3], "W": p[4], "H": p[5],
            "Gamma": p[6], "Yi": p[7:]}


def snapshot(s):
    """The handle's whole state as host arrays (the set_state dictionary)."""
    out = {k: s.get(k) for k in ("CS", "T", "E", "P", "D", "U", "V", "W", "H", "Gamma", "Yi")}
    for k in ("T", "E", "P", "D", "U", "V", "W", "H", "Gamma"):
        out[k] = out[k][0]
    return out


def interior(a, bc=2):
    return a[..., bc:-bc, bc:-bc, bc:-bc]


def species_error(a, b, bc=2):
    """Mean over cells of sum_s |Y_a - Y_b| (all cells; and cells holding any
    reactive species)."""
    ya, yb = interior(a, bc), interior(b, bc)
    l1 = np.abs(ya - yb).sum(axis=0)
    reactive = yb[:8].sum(axis=0) > 1e-9
    return float(l1.mean()), float(l1[reactive].mean()) if reactive.any() else 0.0


def rel_linf(a, b, bc=2):
    """max |a - b| / max |b| per plane (interior nodes), as a list."""
    ai, bi = interior(a, bc), interior(b, bc)
    n = ai.shape[0]
    d = np.abs(ai - bi).reshape(n, -1).max(1)
    s = np.abs(bi).reshape(n, -1).max(1)
    return [float(v) for v in d / np.where(s > 0, s, 1.0)]


def shock_shift(p, p_ref, p0=101325.0, bc=2):
    """Largest |difference| (cells) over the (j, k) columns of the leading
    shock's position: the largest x node whose pressure exceeds 1.5 p0."""
    a, b = interior(p, bc)[0] > 1.5 * p0, interior(p_ref, bc)[0] > 1.5 * p0
    n = a.shape[0]
    ia = np.where(a.any(axis=0), n - 1 - a[::-1].argmax(axis=0), -1)
    ib = np.where(b.any(axis=0), n - 1 - b[::-1].argmax(axis=0), -1)
    return int(np.abs(ia - ib).max())


def nchem_histogram(nchem, bc=2):
    """Cells per Nchem bin: {"<=0": .., "1": .., "2": .., "3-4": .., ...}."""
    v = interior(nchem, bc).ravel()
    out, lo = {}, None
    for hi in NCHEM_BINS:
        sel = (v <= hi) if lo is None else ((v > lo) & (v <= hi))
        key = "<=0" if lo is None else (str(hi) if hi == lo + 1 else
                                        (f">{lo}" if hi >= 1 << 30 else f"{lo + 1}-{hi}"))
        out[key] = int(sel.sum())
        lo = hi
    return out


def window_composition(st, bc=2):
    """What the window's cells hold: cells carrying reactants (Y_H2 + Y_O2 >
    1e-9, the cells whose kinetics the plain FP64 path integrates with
    non-zero rates), the peak temperature among them, and the shock-heated
    ones (T > 400 K)."""
    Y = interior(st["Yi"], bc)
    T = interior(st["T"][None], bc)[0]
    fuel = (Y[cases.S_H2] + Y[cases.S_O2]) > 1e-9
    return {"fuel_cells": int(fuel.sum()), "shocked_fuel_cells": int((fuel & (T > 400.0)).sum()),
            "peak_T_fuel_K": round(float(T[fuel].max()), 1) if fuel.any() else None,
            "peak_T_K": round(float(T.max()), 1), "peak_H2O": float(Y[cases.S_H2O].max()),
            "peak_OH": float(Y[3].max())}


# ---------------------------------------------------------------- distribution

def dist_setup(args):
    world = env_int("WORLD_SIZE", 1)
    rank = env_int("RANK", 0)
    local = env_int("LOCAL_RANK", 0)
    dist = None
    if world > 1:
        import torch
        import torch.distributed as dist
        from datetime import timedelta
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        if backend == "nccl":
            torch.cuda.set_device(local)
        dist.init_process_group(backend, timeout=timedelta(seconds=300))
    return world, rank, local, dist


def reduce_max(dist, value, device):
    if dist is None:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(dist, device):
    if dist is not None:
        if device.startswith("cuda"):
            dist.barrier(device_ids=[int(device.split(":")[1])])
        else:
            dist.barrier()


# ---------------------------------------------------------------- reference arm

def ref_boxes(grid=GRID, box=REF_BOX):
    """The sub-boxes tiling the grid: (first node i, j, k) of each."""
    return [(i, j, k) for i in range(0, grid[0], box[0]) for j in range(0, grid[1], box[1])
            for k in range(0, grid[2], box[2])]


def _ref_box(oracle, origin, box=REF_BOX):
    """A RefOracle holding sub-box `origin` of the workload: the same node
    spacing and positions, the field of the whole grid cut to the box."""
    xf, yf, zf = full_axes()
    lo = [origin[a] + 2 for a in range(3)]
    ext = (xf[lo[0]], xf[lo[0] + box[0] - 1], yf[lo[1]], yf[lo[1] + box[1] - 1], zf[lo[2]], zf[lo[2] + box[2] - 1])
    ref = oracle.RefOracle.from_grid(*box, ext, cases.MECH_JA919, cases.THERMO)
    x, y, z = ref.nodes()
    ref.set_primitive(*bubble_field(x, y, z, ref.mechanism().mw, ref.ns))
    return ref


def _ref_worker(task):
    """One host process: the reference's own CPU timestep on its sub-boxes,
    one after the other. Returns the seconds of the timed steps."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    origins, steps, warmup, dt = task
    secs = 0.0
    for origin in origins:
        ref = _ref_box(oracle, origin)
        if warmup:
            ref.step(warmup, dt)
        t0 = time.perf_counter()
        ref.step(steps, dt)
        secs += time.perf_counter() - t0
        ref.close()
    return secs


def reference_dt(oracle):
    """The workload's dt by the reference's CFL rule at CFL (cases.cfl_dt),
    with density and gamma from the NASA polynomials in numpy, on the whole
    grid's nodes of the sub-box holding the shock: the smallest CFL step of
    the grid is in the uniform shocked N2 behind it. (The reference reads grid
    extents to six significant digits, so its own sub-box nodes sit up to 4e-8
    m off the workload's and its CFL step differs in the sixth digit; this is
    the workload's, equal to the library's to rounding.)"""
    ref = oracle.RefOracle.from_grid(2, 2, 2, (0.0, 1e-3, 0.0, 1e-3, 0.0, 1e-3), cases.MECH_JA919, cases.THERMO)
    m = ref.mechanism()
    ref.close()
    xf, yf, zf = full_axes()
    x, y, z = xf[:REF_BOX[0] + 4], yf[:REF_BOX[1] + 4], zf[:REF_BOX[2] + 4]
    P, T, U, V, _, Y = bubble_field(x, y, z, m.mw, m.ns)
    a = np.where((T < 1000.0)[None, None], m.coeff_lo[:, :, None, None, None], m.coeff_hi[:, :, None, None, None])
    r_s = (8.31434 / m.mw)[:, None, None, None]
    cp_s = r_s * (a[0] * T ** -2 + a[1] / T + a[2] + a[3] * T + a[4] * T ** 2 + a[5] * T ** 3 + a[6] * T ** 4)
    cp, r = (Y * cp_s).sum(0), (Y * r_s).sum(0)
    return cases.cfl_dt(x, y, P, P / (r * 1000.0 * T), U, V, cp / (cp - r), CFL)


def reference_arm(args):
    """--impl reference: the reference's CPU timestep (oracle/_ref) on the
    whole 256 x 128 x 128 grid, cut into 16 sub-boxes of 64^3 nodes, one host
    process per box; the aggregate of independent single-rank runs, no halo
    exchange between the boxes. With fewer than 16 host cores each step is a
    bounded sample: one box per core, spread over the grid. Rank 0 alone runs
    it; the other ranks exit without work."""
    world, rank = env_int("WORLD_SIZE", 1), env_int("RANK", 0)
    if rank != 0:
        return 0
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import multiprocessing as mp

    import oracle
    if not os.path.exists(oracle.REF_LIB):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libeu3d_ref.so not built"}))
        return 0
    ncores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    boxes = ref_boxes()
    nproc = max(1, min(ncores, len(boxes)))
    chosen = [boxes[r * len(boxes) // nproc] for r in range(nproc)]
    dt = reference_dt(oracle)
    steps, warmup = max(1, args.steps), max(0, args.warmup)
    tasks = [([b], steps, warmup, dt) for b in chosen]
    ctx = mp.get_context("spawn")
    with ctx.Pool(nproc) as pool:
        secs = max(pool.map(_ref_worker, tasks))
    cells = nproc * REF_BOX[0] * REF_BOX[1] * REF_BOX[2]
    value = cells * steps / secs / 1e6
    whole = nproc == len(boxes)
    sample = (f"reference CPU timestep (oracle/_ref, unmodified sources, -O3) on "
              f"{'the whole ' if whole else ''}{GRID[0]}x{GRID[1]}x{GRID[2]} grid as "
              f"{'all ' if whole else ''}{nproc} of its {len(boxes)} independent {REF_BOX[0]}^3-node sub-boxes, "
              f"one host process each, {steps} timed steps after {warmup} warm-up from the initial field; the "
              f"reference integrates every cell's kinetics with Nchem = 1 both here and in the timed window (the "
              f"GPU FP64 run's substeps per cell there: plain_fp64.substeps_per_cell)")
    line = {"metric": METRIC, "value": round(value, 6), "unit": "Mcell-steps/s", "n_gpus": world,
            "steps": steps, "warmup": warmup, "ms_per_step": round(secs / steps * 1e3, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "impl": "reference",
            "config": {"workload": "3-D reacting shock-bubble, 256x128x128 nodes over 64x32x32 mm, H2_JA919 "
                                   "(9 species, 19 reactions), Mach 2.83 in N2, seed 3",
                       "grid": list(GRID), "dt": dt, "chemistry": "stiff", "precision": "fp64",
                       "decomposition": f"{len(boxes)} sub-boxes of {REF_BOX[0]}x{REF_BOX[1]}x{REF_BOX[2]} nodes"},
            "cpu_baseline": {"value": round(value, 6), "unit": "Mcell-steps/s", "cores": nproc,
                             "kind": "reference", "sample": sample},
            "e2e": {"value": round(value, 6), "unit": "Mcell-steps/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------- our arm

def cpu_baseline(dt):
    """The reference's CPU timestep on one core, on a bounded sample: the
    64^3-node sub-box holding the bubble's upstream half."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    try:
        import oracle
        if not os.path.exists(oracle.REF_LIB):
            return None
    except ImportError:
        return None
    steps = 6
    secs = _ref_worker(([(64, 0, 0)], steps, 1, dt))
    cells = REF_BOX[0] * REF_BOX[1] * REF_BOX[2]
    return {"value": round(cells * steps / secs / 1e6, 6), "unit": "Mcell-steps/s", "cores": 1,
            "kind": "reference",
            "sample": f"reference CPU timestep (oracle/_ref) on the {REF_BOX[0]}^3-node sub-box of the workload at "
                      f"nodes (64, 0, 0) (the bubble's upstream half), {steps} steps after 1 warm-up, single thread "
                      f"({secs:.1f} s)"}


def mlp_roofline(model, rows=1 << 18, reps=5):
    """The fused inference kernel on `rows` feature rows drawn inside the
    model's input box, launched back to back with no host synchronisation
    between launches: FLOPs of the 3-member ensemble per second, against the
    measured BF16 dense peak."""
    import torch
    import learned
    z = np.load(learned.CHECKPOINT)
    lo, hi = z["box_lo"].astype(np.float32), z["box_hi"].astype(np.float32)
    g = torch.Generator(device="cuda").manual_seed(7)
    X = (torch.from_numpy(lo).cuda() + torch.rand(rows, lo.size, device="cuda", generator=g) *
         torch.from_numpy(hi - lo).cuda()).contiguous()
    members = int(z["shape"][4])
    out = torch.empty(members, rows, int(z["shape"][3]), device="cuda")
    ms = model.time_fused_queue(X, out, reps=reps)
    _, bf16, kind = measured_peaks()
    tf = MLP_FLOP_PER_ROW * rows / (ms / 1e3) / 1e12
    return {"kernel": "mlp_fused", "bound": "tensor", "rows": rows, "ms": round(ms, 4), "achieved": round(tf, 2),
            "peak": bf16, "unit": "TFLOP/s", "frac": round(tf / bf16, 4), "peak_source": f"{kind} bf16_tflops",
            "note": "CUDA events on the model's stream around back-to-back launches (eu_mlp_predict_fused_async)"}


def reacting_block(args, model, gate, local, dt=2e-8):
    """The kinetics-dominated case: a quiescent 48 x 32 x 32 block of hot
    2H2+O2/N2 (eu3d_cases.hot_reacting_block, 1300-2600 K, 0.1-1 MPa) at
    dt = 2e-8 s, stepped by the plain FP64 stiff path and by the learned +
    mixed path from the same state. Reports both throughputs, the substeps of
    the last step, the learned/fallback split and the species L1 difference
    (mean over cells of sum_s |dY_s|) after warm-up + steps. The block ignites:
    the stiff path's Nchem reaches ~100 in the igniting cells. (At the
    shock-bubble's dt of ~1e-7 s the reference's own scheme fails on this
    gas: its Nchem prediction, which ignores species below Y = 1e-6, lets the
    first radicals overshoot into a non-positive Nchem or non-finite state.)"""
    import torch
    import eu3d
    import learned
    grid = (48, 32, 32)
    ext = (0.0, 0.012, 0.0, 0.008, 0.0, 0.008)
    mech = eu3d.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = cases.hot_reacting_block(grid[0] + 4, grid[1] + 4, grid[2] + 4, mech["mw"], mech["ns"])
    ncell = grid[0] * grid[1] * grid[2]
    out, ys = {}, {}
    for name, chem, prec in (("stiff_fp64", "stiff", "fp64"), ("learned_mixed", "learned", "mixed")):
        s = eu3d.Solver(*grid, ext, precision=prec, chemistry=chem, arith="fast", device=local)
        s.set_mechanism(mech)
        s.set_primitive(*prim)
        if chem == "learned":
            learned.attach(s, model, gate)
        s.step(args.warmup, dt)
        torch.cuda.synchronize()
        st = s.step(args.steps, dt)
        torch.cuda.synchronize()
        out[name] = {"value": round(ncell * args.steps / (st["device_ms"] / 1e3) / 1e6, 3),
                     "ms_per_step": round(st["device_ms"] / args.steps, 4), "substeps_last_step": st["sum_nchem"],
                     "max_nchem": st["max_nchem"], "learned_cells": st["learned"], "fallback_cells": st["fallback"]}
        ys[name] = s.get("Yi")
        s.close()
    l1 = np.abs(ys["learned_mixed"] - ys["stiff_fp64"])[:, 2:-2, 2:-2, 2:-2].sum(axis=0)
    shift = cases.front_shift(ys["learned_mixed"], ys["stiff_fp64"])
    return {"grid": list(grid), "cells": ncell, **out,
            "speedup": round(out["learned_mixed"]["value"] / out["stiff_fp64"]["value"], 3),
            "species_l1_mean": float(l1.mean()), "species_l1_max": float(l1.max()),
            "front_shift_cells_max": shift, "dt": dt, "after_steps": args.warmup + args.steps}


def znd_case(args, local, steps=1000, cells=4000, dx=25e-6):
    """The 1-D ZND initiation: 4000 cells of 25 um (4001 x 2 x 2 nodes over
    0.1 m), 2H2+O2+7Ar at 6.67 kPa / 298 K, a 1 MPa / 3000 K driver on the 40
    nodes at the reflecting wall (data/input-1dZND.txt; its edge a 2-cell tanh
    profile, see eu3d_cases.znd), outflow at the far end,
    plain FP64 stiff chemistry, each step's dt from the CFL rule at 0.5 on the
    device, 1000 steps. Reports the device throughput, the time advanced and
    where the leading shock (the largest x with p > 2 x the quiescent
    pressure) is at the end."""
    import eu3d
    ni = cells + 1
    ext = (0.0, cells * dx, 0.0, dx, 0.0, dx)
    x = cases.node_coordinates(ni, ext[0], ext[1])
    y = cases.node_coordinates(2, ext[2], ext[3])
    mech = eu3d.parse_mechanism(cases.MECH_JA919_AR, cases.THERMO_AR)
    prim = cases.znd(x, y, y, mech["mw"], mech["ns"])
    p, cs, T, E = eu3d.initial_state(mech, ni, 2, 2, *prim)
    s = eu3d.Solver(ni, 2, 2, ext, precision="fp64", chemistry="stiff", arith="fast", device=local, boundary="znd")
    s.set_mechanism(mech)
    s.set_state(state_dict((p, cs, T, E)))
    tuned = s.autotune(reps=3)  # a 2 x 2 cross-section: the x-march length matters most
    st, t_adv = s.step_cfl(steps, CFL_THIN)
    pr = s.get("P")[0, 2:-2, 2, 2]
    t_end = s.get("T")[0, 2:-2, 2, 2]
    s.close()
    p0 = eu3d.read_value(cases.INPUT_ZND, "P")
    front = int(np.nonzero(pr > 2 * p0)[0].max()) if (pr > 2 * p0).any() else 0
    return {"grid": [ni, 2, 2], "steps": steps, "time_advanced_s": t_adv,
            "value": round(ni * 4 * steps / (st["device_ms"] / 1e3) / 1e6, 3), "unit": "Mcell-steps/s",
            "ms_per_step": round(st["device_ms"] / steps, 4), "max_nchem_last_step": st["max_nchem"],
            "shock_node": front, "shock_x_m": round(front * dx, 6), "peak_T_K": round(float(t_end.max()), 1),
            "peak_p_Pa": round(float(pr.max()), 1), "autotune": {"flux_ci": tuned["flux_ci"],
                                                                 "recover_block": tuned["recover_block"]}}


def odw_case(args, local, model, gate, grid=(1024, 512, 2), steps=2000, extent=(0.040, 0.020, None),
             phi_seed=None, cfl=CFL_THIN, input_path=None, chem="learned", precision="mixed", keep_y=False):
    """The oblique detonation case (data/input-ODW-M7.txt: Mach 7, 300 K,
    101.325 kPa stoichiometric H2-air, a 25 degree wedge whose tip is 5 mm
    from the inflow face). 2-D (default): 1024 x 512 x 2 nodes over 40 x 20
    mm (the z spacing equals the x spacing). 3-D: 384 x 192 x 96 nodes over 40
    x 20 x 10 mm with the equivalence ratio phi(z) of eu3d_cases.odw_phi on
    the inflow. The grid is wedge-aligned (the y-low face is the wedge surface
    from the tip on, the freestream ahead of it, eu_set_odw_wall), with the
    reference's ODW ghost fill (EU_BC_ODW) and each dt from the CFL rule on
    the device: 2000 steps at CFL 0.5 in 2-D, 1000 steps at CFL 0.25 in 3-D
    (the reference's forward-Euler MUSCL step goes non-finite at CFL 0.5 once
    the gas ignites on grids as coarse as the 3-D one's, in the C restatement
    as well). chem/precision: "learned"/"mixed" or the plain "stiff"/"fp64".
    Reports the device throughput, the time advanced, the peak temperature
    and the shock angle in the middle z plane: where p first exceeds 1.5 x the
    freestream pressure from the top down, fitted over the wedge's middle
    half, plus the wedge angle (the oblique-shock relation gives about 32
    degrees for an ideal gas at gamma 1.4)."""
    import eu3d
    input_path = input_path or cases.INPUT_ODW_M7
    ni, nj, nk = grid
    dx = extent[0] / (ni - 1)
    ext = (0.0, extent[0], 0.0, extent[1], 0.0, dx * (nk - 1) if extent[2] is None else extent[2])
    x = cases.node_coordinates(ni, ext[0], ext[1])
    y = cases.node_coordinates(nj, ext[2], ext[3])
    z = cases.node_coordinates(nk, ext[4], ext[5])
    mech = eu3d.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    phi = cases.odw_phi(z, seed=phi_seed) if phi_seed is not None else None
    prim, inflow = cases.odw(x, y, z, mech, input_path=input_path, phi=phi)
    p, cs, T, E = eu3d.initial_state(mech, ni, nj, nk, *prim)
    if chem == "learned" and model is None:
        chem = "stiff"
    s = eu3d.Solver(ni, nj, nk, ext, precision=precision, chemistry=chem, arith="fast", device=local,
                    boundary="odw")
    s.set_mechanism(mech)
    s.set_state(state_dict((p, cs, T, E)))
    s.set_inflow(*inflow)
    wall = cases.odw_wall_node(x, input_path)
    s.set_odw_wall(wall)
    if chem == "learned":
        import learned
        learned.attach(s, model, gate)
    tuned = s.autotune(reps=3)
    st, t_adv = s.step_cfl(steps, cfl)
    pr = s.get("P")[0, 2:-2, 2:-2, 2 + nk // 2]  # the middle z plane
    t_end = s.get("T")[0, 2:-2, 2:-2, :]
    yi = s.get("Yi") if keep_y else None
    s.close()
    p0 = eu3d.read_value(input_path, "P")
    angle = eu3d.read_value(input_path, "angle")
    xs, hs = [], []
    span = ni - wall
    for i in range(wall + span // 4, wall + 3 * span // 4):
        hit = np.nonzero(pr[i, ::-1] > 1.5 * p0)[0]
        if hit.size:
            xs.append(x[2 + i])
            hs.append(y[2 + nj - 1 - hit[0]])
    beta = (math.degrees(math.atan(np.polyfit(xs, hs, 1)[0])) + angle) if len(xs) > 8 else None
    out = {"grid": list(grid), "extent_m": [ext[1], ext[3], ext[5]], "steps": steps, "cfl": cfl,
           "time_advanced_s": t_adv, "chemistry": chem, "precision": precision,
           "freestream": {k: eu3d.read_value(input_path, k) for k in ("Mach", "P", "T")}, "wall_first_node": wall,
           "value": round(ni * nj * nk * steps / (st["device_ms"] / 1e3) / 1e6, 3), "unit": "Mcell-steps/s",
           "ms_per_step": round(st["device_ms"] / steps, 4), "peak_T_K": round(float(t_end.max()), 1),
           "peak_p_Pa": round(float(pr.max()), 1), "shock_angle_deg": None if beta is None else round(beta, 2),
           "learned_cells_last_step": st["learned"], "fallback_cells_last_step": st["fallback"],
           "max_nchem_last_step": st["max_nchem"],
           "autotune": {"flux_ci": tuned["flux_ci"], "recover_block": tuned["recover_block"]}}
    return (out, yi) if keep_y else out


def odw_2d(args, local, model, gate):
    """Config 2: the 2-D oblique detonation, plain FP64 stiff against learned +
    mixed, each 2000 steps at CFL 0.5 from the same initial state, with the
    species L1 and the reaction-front shift between the two at the end."""
    plain, y_ref = odw_case(args, local, model, gate, chem="stiff", precision="fp64", keep_y=True)
    fast, y_fast = odw_case(args, local, model, gate, keep_y=True)
    l1 = np.abs(y_fast - y_ref)[:, 2:-2, 2:-2, 2:-2].sum(axis=0)
    return {"plain_fp64": plain, "learned_mixed": fast,
            "speedup": round(fast["value"] / plain["value"], 3) if plain["value"] else None,
            "species_l1_mean": float(l1.mean()), "species_l1_max": float(l1.max()),
            "reaction_front_shift_cells": cases.front_shift(y_fast, y_ref)}


BATCH_SIZES = ((64, 64, 64), (128, 64, 64), (192, 96, 96))


def batch_specs(count=32, seed=5):
    """The uneven batch: `count` shock-bubble instances with grids drawn from
    BATCH_SIZES, shock Mach U[1.8, 3.5] and bubble radius U[4, 10] mm
    (numpy.random.default_rng(seed)). Domains: 64 x 32 x 32 mm for the
    elongated grids, 32 mm cubes for 64^3; the radius is scaled by
    min(1, 0.3 L_y / 10 mm) so every bubble fits its domain."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        grid = BATCH_SIZES[int(rng.integers(len(BATCH_SIZES)))]
        mach = float(rng.uniform(1.8, 3.5))
        radius = float(rng.uniform(4e-3, 10e-3))
        ext = (0.0, 0.032, 0.0, 0.032, 0.0, 0.032) if grid[0] == grid[1] else (0.0, 0.064, 0.0, 0.032, 0.0, 0.032)
        out.append((grid, mach, radius * min(1.0, 0.3 * ext[3] / 10e-3), ext))
    return out


def batch_instances(args, model, gate, local, mech, count=32):
    """The batched uneven shock-bubble workload: the instances of batch_specs,
    learned chemistry + mixed precision, advanced together by one graph
    launch per step (eu_batch), against running them one by one on the plain
    FP64 stiff path. Aggregate cell-steps per device second of each, and each
    instance's own step time one by one."""
    import torch
    import eu3d
    import learned
    built = []
    for q, (grid, mach, radius, ext) in enumerate(batch_specs(count)):
        x, y, z = (cases.node_coordinates(n, ext[2 * a], ext[2 * a + 1]) for a, n in enumerate(grid))
        center_x = 0.55 * ext[1]
        prim = cases.shock_bubble(x, y, z, mech["mw"], mech["ns"], mach=mach, radius=radius,
                                  shock_x=center_x - radius - 2e-3, standoff=radius + 2e-3, seed=100 + q, band=0.5)
        p, cs, T, E = eu3d.initial_state(mech, *grid, *prim)
        dt = cases.cfl_dt(x, y, p[0], p[1], p[2], p[3], p[6], CFL)
        built.append((grid, ext, state_dict((p, cs, T, E)), dt))
    cells = [g[0] * g[1] * g[2] for g, _, _, _ in built]
    total = sum(cells)

    def solver(grid, ext, st, chem, prec):
        s = eu3d.Solver(*grid, ext, precision=prec, chemistry=chem, arith="fast", device=local)
        s.set_mechanism(mech)
        s.set_state(st)
        if chem == "learned":
            learned.attach(s, model, gate)
        return s

    # one by one, plain FP64 stiff: each instance's own step time
    single_ms = []
    for (grid, ext, st, dt) in built:
        s = solver(grid, ext, st, "stiff", "fp64")
        s.step(args.warmup, dt)
        r = s.step(args.steps, dt)
        single_ms.append(r["device_ms"] / args.steps)
        s.close()
    torch.cuda.synchronize()
    # together: learned + mixed, one graph launch per step; the fallback and
    # deferred-cell kinetics of all instances as one shared stage, and (for
    # comparison) inside each instance's branch
    dts = [dt for (_, _, _, dt) in built]
    runs = {}
    for shared in (False, True):
        solvers = [solver(grid, ext, st, "learned", "mixed") for (grid, ext, st, _) in built]
        b = eu3d.Batch(solvers)
        b.set_shared_kinetics(shared)
        b.step(args.warmup, dts)
        stats, ms = b.step(args.steps, dts)
        runs[shared] = (stats, ms, b.launches())
        b.close()
        for s in solvers:
            s.close()
    stats, ms, (per_step, stage) = runs[True]
    branch_ms = runs[False][1]
    one_by_one = total * args.steps / (sum(single_ms) * args.steps / 1e3) / 1e6
    together = total * args.steps / (ms / 1e3) / 1e6
    return {"instances": count, "cells": total, "grids": {f"{g[0]}x{g[1]}x{g[2]}": sum(1 for b_ in built if b_[0] == g)
                                                           for g in BATCH_SIZES},
            "learned_mixed_batch": {"value": round(together, 3), "ms_per_step": round(ms / args.steps, 4),
                                    "graph_launches_per_step": 1, "kernels_per_step": per_step,
                                    "shared_kinetics_launches_per_step": stage,
                                    # launches per stage: the ghost fill, flux, recovery and model
                                    # stages run once per instance; the fallback and deferred-cell
                                    # kinetics stages once for the whole batch
                                    "launches_per_stage": {"per_instance_stages": len(built),
                                                           "shared_kinetics_stages": stage // 2 if stage else 0},
                                    "ms_per_step_kinetics_in_branches": round(branch_ms / args.steps, 4),
                                    "kernels_per_step_kinetics_in_branches": runs[False][2][0],
                                    "learned_cells_last_step": int(sum(st_["learned"] for st_ in stats)),
                                    "max_nchem": int(max(st_["max_nchem"] for st_ in stats))},
            "plain_fp64_one_by_one": {"value": round(one_by_one, 3), "ms_per_step": round(sum(single_ms), 4),
                                      "instance_ms_per_step": {"min": round(min(single_ms), 4),
                                                               "median": round(float(np.median(single_ms)), 4),
                                                               "max": round(max(single_ms), 4)}},
            "speedup": round(together / one_by_one, 3), "steps": args.steps, "warmup": args.warmup,
            "seed": 5, "unit": "Mcell-steps/s"}


def flux_roofline(phase, steps, ncell, precision):
    """The flux + update kernel's algorithmic bytes per launch over its CUDA-event
    time, against the measured copy bandwidth; the dominant kernel phase."""
    hbm, _, peak_kind = measured_peaks()
    names = ["ghost_fill", "flux_update", "recover_kinetics"]
    flux_ms = phase[1] / steps
    flux_gbs = FLUX_BYTES[precision] * ncell / (flux_ms / 1e3) / 1e9
    dominant = max(range(3), key=lambda q: phase[q])
    return {"kernel": "flux_update", "bound": "hbm", "achieved": round(flux_gbs, 1), "peak": hbm,
            "unit": "GB/s", "frac": round(flux_gbs / hbm, 4),
            "traffic": (round(FLUX_TRAFFIC_PER_CELL[precision] * ncell / 1e9, 4)
                        if precision in FLUX_TRAFFIC_PER_CELL else None),
            "traffic_unit": "GB per launch (ncu, scaled from 256x128x64)",
            "algorithmic_bytes_per_cell": FLUX_BYTES[precision], "flux_ms": round(flux_ms, 4),
            "peak_source": f"{peak_kind} hbm_gbs", "dominant_kernel": names[dominant],
            "dominant_share": round(phase[dominant] / max(sum(phase[:3]), 1e-9), 3)}


def our_arm_blocks(args, world, rank, local, dist):
    """The workload decomposed along x over the ranks (eu3d-gpu_b200/slab.py),
    one 256 x 128 x 128-node block per GPU, halo planes exchanged over NCCL
    every step, advanced untimed to the same window as the one-GPU run (the
    shock inside the bubble of block 0) before the timed steps. The
    single-GPU side studies (reacting block, batch, ZND, model roofline, CPU
    baseline) are N = 1 measurements and are not repeated."""
    import torch
    import eu3d
    import slab
    device = f"cuda:{local}"
    ni, nj, nk = args.grid
    total_ni = world * (ni - 1) + 1
    ext = (EXTENT[0], EXTENT[0] + (EXTENT[1] - EXTENT[0]) * (total_ni - 1) / (ni - 1), *EXTENT[2:])
    x = cases.node_coordinates(total_ni, ext[0], ext[1], blocks=world, block=rank)
    y = cases.node_coordinates(nj, ext[2], ext[3])
    z = cases.node_coordinates(nk, ext[4], ext[5])
    mech = eu3d.parse_mechanism(cases.MECH_JA919, cases.THERMO)
    prim = cases.shock_bubble(x, y, z, mech["mw"], mech["ns"], seed=3)
    p, cs, T, E = eu3d.initial_state(mech, ni, nj, nk, *prim)
    sd = state_dict((p, cs, T, E))
    ncell = ni * nj * nk
    # dt: the reference's CFL rule, minimum over the blocks
    dt_t = torch.tensor([cases.cfl_dt(x, y, p[0], p[1], p[2], p[3], p[6], CFL)], dtype=torch.float64, device=device)
    dist.all_reduce(dt_t, op=dist.ReduceOp.MIN)
    dt = float(dt_t.item())
    model = gate = None
    if args.chem == "learned":
        import learned
        model, gate = learned.load(device=local)
    start = min(getattr(args, "window_start", WINDOW_START), TOTAL_STEPS)

    def make(chem, precision, arith, profile=False, state=sd):
        s = slab.SlabSolver(dist, total_ni, nj, nk, ext, device=local, precision=precision, chemistry=chem,
                            arith=arith, profile=profile)
        s.set_mechanism(mech)
        s.set_state(state)
        if chem == "learned":
            import learned
            learned.attach(s.solver, model, gate)
        return s

    def timed(s, clocks=False):
        """Device time of args.steps exchanged steps (events on the handle's
        stream), max over ranks, and the last step's statistics."""
        s.step(args.warmup, dt, stats=False)
        s.sync()
        barrier(dist, device)
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        clk = ClockSampler(torch.cuda.current_device()) if clocks else None
        if clk:
            clk.__enter__()
        ev0.record(s.stream)
        st = s.step(args.steps, dt, stats=True)
        ev1.record(s.stream)
        ev1.synchronize()
        if clk:
            clk.__exit__(None, None, None)
        barrier(dist, device)
        return st, reduce_max(dist, ev0.elapsed_time(ev1), device), (clk.summary() if clk else None)

    s = make(args.chem, args.precision, args.arith)
    if start:
        s.step(start, dt, stats=False)
    window_state = snapshot(s.solver)
    tuned = s.autotune(reps=5) if not args.no_autotune else None
    stats, ms, clocks = timed(s, clocks=True)
    value = ncell * args.steps * world / (ms / 1e3) / 1e6
    y_fast = s.get("Yi")
    halo_bytes = s.halo_bytes()
    faces = len(s.halo.faces)
    s.close()

    plain = None
    if (args.chem, args.precision) != ("stiff", "fp64"):
        sp_ = make("stiff", "fp64", "fast")
        if start:
            sp_.step(start, dt, stats=False)
        ptuned = sp_.autotune(reps=5) if not args.no_autotune else None
        _, pms, _ = timed(sp_)
        y_ref = sp_.get("Yi")
        sp_.close()
        err_all, err_reactive = species_error(y_fast, y_ref)
        pvalue = ncell * args.steps * world / (pms / 1e3) / 1e6
        plain = {"value": round(pvalue, 3), "ms_per_step": round(pms / args.steps, 4),
                 "speedup": round(value / pvalue, 3), "autotune": ptuned, "species_l1_vs_plain": err_all,
                 "species_l1_vs_plain_reactive_cells": err_reactive, "after_steps": start + args.warmup + args.steps,
                 "note": "rank 0's block"}

    # per-kernel phases of one exchanged step (CUDA events inside the library)
    sp = make(args.chem, args.precision, args.arith, profile=True, state=window_state)
    sp.step(args.warmup, dt, stats=False)
    phase = sp.step(1, dt, stats=True)["phase_ms"]
    sp.close()
    names = ["ghost_fill", "flux_update", "recover_kinetics" if args.chem != "learned" else "recover_learned_chem"]
    per_kernel = {n: round(phase[q], 4) for q, n in enumerate(names)}
    roofline = flux_roofline(phase, 1, ncell, args.precision)

    # end to end through the public API with host buffers: the configured run
    # (each block's initial state up once, the exchanged steps each synchronous,
    # the conserved state down at the end)
    pinned = {}
    for k in ("CS", "T", "E"):
        src = sd[k] if k == "CS" else sd[k][None]
        t = torch.empty(src.shape, dtype=torch.float64, pin_memory=True)
        t.numpy()[...] = src
        pinned[k] = t.numpy()
    cs_host = torch.empty(sd["CS"].shape, dtype=torch.float64, pin_memory=True).numpy()
    se = make(args.chem, args.precision, args.arith, state=window_state)
    se.step(args.warmup, dt, stats=False)
    se.sync()
    e2e_steps = max(getattr(args, "total_steps", TOTAL_STEPS), start + args.warmup + args.steps)
    barrier(dist, device)
    t0 = time.perf_counter()
    se.set_conserved(pinned["CS"], pinned["T"], pinned["E"])
    for _ in range(e2e_steps):
        se.step(1, dt, stats=True)
    cs_out = se.get("CS", out=cs_host)
    e2e_s = reduce_max(dist, time.perf_counter() - t0, device)
    e2e_value = ncell * e2e_steps * world / e2e_s / 1e6
    h2d = sum(v.nbytes for v in pinned.values()) / e2e_steps + 8
    d2h = cs_out.nbytes / e2e_steps + 96
    se.close()

    if rank == 0:
        line = {"metric": METRIC, "value": round(value, 3), "unit": "Mcell-steps/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4),
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f32+f64" if args.precision == "mixed" else "f64",
                "data": "synthetic",
                "config": {"workload": f"3-D reacting shock-bubble decomposed along x: {world} blocks of "
                                       f"{ni}x{nj}x{nk} nodes ({total_ni}x{nj}x{nk} global over "
                                       f"{ext[1] * 1e3:.0f}x32x32 mm), H2_JA919, Mach 2.83 in N2, seed 3",
                           "grid": [ni, nj, nk], "global_grid": [total_ni, nj, nk], "dt": dt,
                           "window": f"steps {start + args.warmup} .. {start + args.warmup + args.steps}",
                           "precision": args.precision, "chemistry": args.chem, "arith": args.arith,
                           "parallelism": f"x blocks {world}, halo exchange over NCCL every step",
                           "halo_bytes_per_face": halo_bytes, "autotune": tuned,
                           "l2": f"inputs larger than L2: {sd['CS'].nbytes * 3 // 2**20} MiB state per GPU > 126 MiB"},
                "plain_fp64": plain,
                "roofline": roofline, "kernels_ms_per_step": per_kernel,
                "max_nchem": stats["max_nchem"], "reacting_cells": stats["reacting"],
                "learned_cells": stats["learned"], "fallback_cells": stats["fallback"],
                "clocks": clocks,
                "e2e": {"value": round(e2e_value, 3), "unit": "Mcell-steps/s",
                        "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h), "steps": e2e_steps},
                # the step's kernels plus one halo pack and unpack per neighbour face
                "gpu_launches": (stats["launches"] + 2 * faces) * args.steps,
                "cpu_baseline": None}
        print(json.dumps(line), flush=True)
    dist.destroy_process_group()
    return 0


def our_arm(args):
    import torch
    import eu3d
    world, rank, local, dist = dist_setup(args)
    if world > 1:
        return our_arm_blocks(args, world, rank, local, dist)
    device = f"cuda:{local}"
    torch.cuda.set_device(local)
    grid = tuple(args.grid)
    ncell = grid[0] * grid[1] * grid[2]
    mech, prim, st0, dt = build_workload(grid)
    sd = state_dict(st0)
    model = gate = None
    if args.chem == "learned":
        import learned
        model, gate = learned.load(device=local)
    start = min(args.window_start, args.total_steps)
    window_end = start + args.warmup + args.steps
    run_end = max(args.total_steps, window_end)

    def make_solver(chem, precision, arith, profile=False, state=sd):
        s = eu3d.Solver(*grid, EXTENT, precision=precision, chemistry=chem, arith=arith, device=local,
                        profile=profile)
        s.set_mechanism(mech)
        s.set_state(state)
        # every arm the same way; the benchmark reads interior nodes only
        s.set_ghost_mode(args.ghosts)
        if chem == "learned":
            import learned
            learned.attach(s, model, gate)
        return s

    def window_run(s, clocks=False, tune=False):
        """Advance to the window untimed, (autotune,) warm up, time args.steps
        steps, keep the state at the window's end, run on to run_end."""
        if start:
            s.step(start, dt, stats=False)
        ws = snapshot(s) if clocks else None
        tuned = s.autotune(reps=5) if tune else None
        s.step(args.warmup, dt, stats=False)
        torch.cuda.synchronize()
        clk = ClockSampler(torch.cuda.current_device()) if clocks else None
        if clk:
            clk.__enter__()
        st = s.step(args.steps, dt)
        torch.cuda.synchronize()
        if clk:
            clk.__exit__(None, None, None)
        end = {"Yi": s.get("Yi"), "P": s.get("P"), "CS": s.get("CS"), "T": s.get("T"), "Nchem": s.get("Nchem")}
        if run_end > window_end:
            s.step(run_end - window_end, dt, stats=False)
        last = {"Yi": s.get("Yi"), "P": s.get("P"), "CS": s.get("CS")}
        return st, end, last, ws, tuned, (clk.summary() if clk else None)

    # -- the configured path (learned + mixed by default): value -------------------------------
    s = make_solver(args.chem, args.precision, args.arith)
    stats, end_fast, last_fast, window_state, tuned, clocks = window_run(s, clocks=True, tune=not args.no_autotune)
    s.close()
    ms = reduce_max(dist, stats["device_ms"], device)
    value = ncell * args.steps * world / (ms / 1e3) / 1e6
    window = window_composition({"Yi": end_fast["Yi"], "T": end_fast["T"][0]})

    # -- the plain FP64 stiff step, its own trajectory (the comparison the metric names) --------
    plain = None
    if (args.chem, args.precision) != ("stiff", "fp64"):
        sp_ = make_solver("stiff", "fp64", "fast")
        pst, end_ref, last_ref, _, ptuned, _ = window_run(sp_, tune=not args.no_autotune)
        sp_.close()
        pms = pst["device_ms"]
        err_all, err_reactive = species_error(end_fast["Yi"], end_ref["Yi"])
        err_all_500, err_reactive_500 = species_error(last_fast["Yi"], last_ref["Yi"])
        # the kinetics phase of the plain step against the FP64 roofline, on the window state
        spk = make_solver("stiff", "fp64", "fast", profile=True, state=window_state)
        spk.step(args.warmup, dt)
        kst = spk.step(args.steps, dt)
        plain_phase = kst["phase_ms"]
        spk.close()
        kin_ms = plain_phase[2] / args.steps
        kin_tf = F_SUB * kst["sum_nchem"] / (kin_ms / 1e3) / 1e12
        kin = {"kernel": "recover_react", "bound": "fp64", "achieved": round(kin_tf, 3),
               "peak": FP64_PEAK_TFLOPS, "unit": "TFLOP/s", "frac": round(kin_tf / FP64_PEAK_TFLOPS, 4),
               "peak_source": "datasheet", "flop_per_substep": F_SUB, "substeps_per_step": kst["sum_nchem"],
               "ms_per_step": round(kin_ms, 4)}
        pvalue = ncell * args.steps * world / (pms / 1e3) / 1e6
        plain = {"value": round(pvalue, 3), "ms_per_step": round(pms / args.steps, 4),
                 "speedup": round(value / pvalue, 3), "autotune": ptuned,
                 "kernels_ms_per_step": {n: round(plain_phase[q] / args.steps, 4)
                                         for q, n in enumerate(("ghost_fill", "flux_update", "recover_kinetics"))},
                 "flux_roofline": flux_roofline(plain_phase, args.steps, ncell, "fp64"),
                 "kinetics_roofline": kin,
                 "substeps_per_cell": round(pst["sum_nchem"] / ncell, 6), "max_nchem": pst["max_nchem"],
                 "nchem_histogram_window_end": nchem_histogram(end_ref["Nchem"]),
                 "error_vs_plain": {
                     "at_window_end": {"step": window_end, "species_l1": err_all,
                                       "species_l1_fuel_cells": err_reactive,
                                       "interface_shift_cells": cases.front_shift(end_fast["Yi"], end_ref["Yi"],
                                                                                  product=cases.S_H2),
                                       "reaction_front_shift_cells": cases.front_shift(end_fast["Yi"], end_ref["Yi"]),
                                       "shock_shift_cells": shock_shift(end_fast["P"], end_ref["P"]),
                                       "cs_rel_linf_max": max(rel_linf(end_fast["CS"], end_ref["CS"]))},
                     "at_step_500": {"step": run_end, "species_l1": err_all_500,
                                     "species_l1_fuel_cells": err_reactive_500,
                                     "interface_shift_cells": cases.front_shift(last_fast["Yi"], last_ref["Yi"],
                                                                                product=cases.S_H2),
                                     "reaction_front_shift_cells": cases.front_shift(last_fast["Yi"], last_ref["Yi"]),
                                     "shock_shift_cells": shock_shift(last_fast["P"], last_ref["P"]),
                                     "cs_rel_linf": rel_linf(last_fast["CS"], last_ref["CS"])}}}
        del end_ref, last_ref
    del last_fast

    # -- reacting gas: the chemistry phase the learned model replaces ---------------------------
    block = reacting_block(args, model, gate, local) if args.chem == "learned" else None
    mlp = mlp_roofline(model) if args.chem == "learned" else None

    # -- uneven instances advanced together (one graph launch per step) ----------------------
    batch = None
    if args.chem == "learned" and not args.no_batch:
        batch = batch_instances(args, model, gate, local, mech)
    znd = odw = odw3 = None
    if not args.no_batch:
        try:
            znd = znd_case(args, local)
        except eu3d.EU3DError as e:  # reported, not fatal to the headline measurement
            znd = {"error": str(e)}
        try:
            odw = odw_2d(args, local, model, gate)
        except eu3d.EU3DError as e:
            odw = {"error": str(e)}
        try:
            odw3 = odw_case(args, local, model, gate, grid=(384, 192, 96), steps=1000, extent=(0.040, 0.020, 0.010),
                            phi_seed=4, cfl=0.25)
        except eu3d.EU3DError as e:
            odw3 = {"error": str(e)}

    # -- per-kernel times on the window state (same stream, CUDA events around each phase) ----
    sp = make_solver(args.chem, args.precision, args.arith, profile=True, state=window_state)
    sp.step(args.warmup, dt)
    pst = sp.step(args.steps, dt)
    phase = pst["phase_ms"]
    names = ["ghost_fill", "flux_update", "recover_kinetics" if args.chem != "learned" else "recover_learned_chem"]
    per_kernel = {n: round(phase[q] / args.steps, 4) for q, n in enumerate(names)}
    sp.close()
    roofline = flux_roofline(phase, args.steps, ncell, args.precision)

    # -- end to end through the public API with host buffers: the configured run --------------
    # the whole run a user makes: the initial conserved state (CS, T, E) from
    # pinned host memory (eu_set_conserved forms the primitives on the device as
    # the step's recovery does), run_end steps each reading its health counters
    # back to the host, the final conserved state read back
    pinned = {}
    for k in ("CS", "T", "E"):
        src = sd[k] if k == "CS" else sd[k][None]
        t = torch.empty(src.shape, dtype=torch.float64, pin_memory=True)
        t.numpy()[...] = src
        pinned[k] = t.numpy()
    cs_host = torch.empty(sd["CS"].shape, dtype=torch.float64, pin_memory=True).numpy()
    se = make_solver(args.chem, args.precision, args.arith, state=window_state)
    se.step(args.warmup, dt)  # first capture and attribute set-up, then the run from the initial state
    e2e_steps = max(run_end, args.steps)
    barrier(dist, device)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    se.set_conserved(pinned["CS"], pinned["T"], pinned["E"])
    for _ in range(e2e_steps):
        se.step(1, dt)  # synchronous: reads the step's health counters back
    cs = se.get("CS", out=cs_host)
    torch.cuda.synchronize()
    e2e_s = reduce_max(dist, time.perf_counter() - t0, device)
    e2e_value = ncell * e2e_steps * world / e2e_s / 1e6
    state_bytes = sum(v.nbytes for v in pinned.values())
    h2d = state_bytes / e2e_steps + 8
    d2h = cs.nbytes / e2e_steps + 96
    se.close()

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(dt)

    if rank == 0:
        line = {"metric": METRIC, "value": round(value, 3), "unit": "Mcell-steps/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4),
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f32+f64" if args.precision == "mixed" else "f64",
                "data": "synthetic",
                "config": {"workload": "3-D reacting shock-bubble, 256x128x128 nodes over 64x32x32 mm, "
                                       "H2_JA919 (9 species, 19 reactions), Mach 2.83 in N2, seed 3",
                           "grid": list(grid), "dt": dt,
                           "window": {"start_step": start, "timed_steps": [start + args.warmup, window_end],
                                      "run_steps": run_end,
                                      "why": "the shock reaches the bubble after about 160 steps; from then on it "
                                             "runs through the bubble gas"},
                           "precision": args.precision, "chemistry": args.chem,
                           "arith": args.arith, "parallelism": f"replicas x{world}", "autotune": tuned,
                           "ghosts": args.ghosts,
                           "l2": f"inputs larger than L2: {sd['CS'].nbytes * 3 // 2**20} MiB state > 126 MiB"},
                "window_state": {**window,
                                 "note": "the transmitted shock heats the bubble gas to about 600 K and the "
                                         "shocked N2 is at 745 K: below the 800 K activity threshold, no radical "
                                         "pool forms and no cell ignites within the run's 500 steps (24.5 us), so "
                                         "the learned path finds no chemically active cell; reacting_block is "
                                         "the figure on igniting gas"},
                "plain_fp64": plain,
                "reacting_block": block,
                "batch_instances": batch,
                "mlp_roofline": mlp,
                "znd_1d": znd,
                "odw_2d": odw,
                "odw_3d": odw3,
                "roofline": roofline, "kernels_ms_per_step": per_kernel,
                "max_nchem": stats["max_nchem"], "reacting_cells": stats["reacting"],
                "learned_cells": stats["learned"], "fallback_cells": stats["fallback"],
                "nchem_histogram_window_end": nchem_histogram(end_fast["Nchem"]),
                "clocks": clocks,
                "e2e": {"value": round(e2e_value, 3), "unit": "Mcell-steps/s",
                        "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
                        "steps": e2e_steps,
                        "what": "the configured run through the C-ABI from host buffers: the initial conserved "
                                "state uploaded from pinned memory, every step synchronous with its health "
                                "counters read back, the final conserved state downloaded; bytes per step "
                                "are the run's copies over its steps"},
                "gpu_launches": stats["launches"],
                "cpu_baseline": cpu}
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()
    return 0


def side_study(args):
    """One side study on cuda:0, its result printed as JSON (for profiling a
    kernel that the full run launches among many others)."""
    import torch
    import learned
    torch.cuda.set_device(0)
    model, gate = learned.load(device=0)
    out = reacting_block(args, model, gate, 0) if args.only == "reacting_block" else mlp_roofline(model)
    print(json.dumps({args.only: out}), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--precision", choices=["fp64", "mixed"], default="mixed")
    ap.add_argument("--chem", choices=["stiff", "frozen", "learned"], default="learned")
    ap.add_argument("--arith", choices=["strict", "fast"], default="fast")
    ap.add_argument("--grid", type=int, nargs=3, default=list(GRID))
    ap.add_argument("--window-start", type=int, default=WINDOW_START,
                    help="steps advanced untimed before the timed window")
    ap.add_argument("--total-steps", type=int, default=TOTAL_STEPS,
                    help="steps each arm runs in all (the window included); the errors are stated at the end")
    ap.add_argument("--only", choices=["reacting_block", "mlp_roofline"],
                    help="run one side study alone and print its result (profiling runs)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-batch", action="store_true", help="skip the batched uneven-instance workload")
    ap.add_argument("--no-autotune", action="store_true", help="keep the default launch shapes")
    ap.add_argument("--ghosts", choices=["reference", "stored"], default="stored",
                    help="z-face ghosts formed by the ghost fill (the reference's placement) or stored with the "
                         "interior (eu_set_ghost_mode; the same interior state)")
    args = ap.parse_args()
    if args.impl == "reference":
        return reference_arm(args)
    if args.chem == "learned":
        import learned
        if not os.path.exists(learned.CHECKPOINT):
            print("no trained learned-chemistry checkpoint; measuring the stiff kinetics", file=sys.stderr)
            args.chem = "stiff"
    if args.warmup < 3:
        args.warmup = 3
    if args.only:
        return side_study(args)
    return our_arm(args)


if __name__ == "__main__":
    sys.exit(main())
