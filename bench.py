#!/usr/bin/env python3
"""Benchmark of the GB300 ADER-DG element path.

Workload (default): Kelvin-Helmholtz, 2D compressible Euler, modal Legendre
p=3 (Np_s=10), 3 AMR levels 64^2 -> 128^2 -> 256^2 (ratio 2, max grid 32,
blocking factor 8, normalised density gradient > 0.1, regrid every 4 steps)
on periodic [0,1]^2, seeded noise, FP64 corrector -- the configuration the
headline metric is quoted on.  A step is the whole evolve-loop body: regrid
when due, ADER predictor-corrector of every element of every level in one
launch per stage, reflux, average down, ghost fill, device time step.
Metric: DOF-updates/s = sum over steps of valid elements of all levels times
Q * Np_s.  The plain path (named plain_fp64: FP64 state and fluxes, the
predictor's operators in 60-bit fixed point) and the learned-seed path run on
the same workload; the headline value is the fastest seed variant whose L2 density
error against a converged-Picard FP64 run stays within 1.01x of the plain
path's.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

--impl reference times the reference algorithm's CPU restatement (the
oracle, C++/OpenMP on all host cores) on the same workload.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
# the library's autotuner records its choices next to the build
os.environ.setdefault("ADG_TUNE_CACHE", os.path.join(ROOT, "ader-dg-amr_gb300", "_build", "tune_cache.txt"))
sys.path.insert(0, os.path.join(ROOT, "ader-dg-amr_gb300"))
sys.path.insert(0, os.path.join(ROOT, "tests"))

WORKLOADS = {
    # configs 3 + 4: batched 3-level KH, plain FP64 vs learned-seed path
    "kh_p3_amr3": dict(D=2, P=3, n=(64, 64, 1), lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0), periodic=(1, 1, 1),
                       ic="kh_noise", seed=12345, noise_amp=1e-3, c_dt=0.5,
                       amr=dict(max_level=2, max_grid=32, blocking_factor=8, dtn_regrid=4, tag_kind=0,
                                tag_threshold=0.1)),
    # config 5: 3D blast, 2 levels
    # (the unlimited scheme does not survive this blast: TVB limiter as the
    # reference's shock presets use it, every step, M = 10)
    "blast3d_p2_amr2": dict(D=3, P=2, n=(64, 64, 64), lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0), periodic=(0, 0, 0),
                            ic="blast3d", c_dt=0.5, limiter=dict(TVB_M=10.0, t_limit=1),
                            amr=dict(max_level=1, max_grid=32, blocking_factor=8, dtn_regrid=4, tag_kind=1,
                                     tag_threshold=0.1)),
    "kh_p3_256": dict(D=2, P=3, n=(256, 256, 1), lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0), periodic=(1, 1, 1),
                      ic="kh_noise", seed=12345, noise_amp=1e-3, c_dt=0.5),
    "vortex_p1_32": dict(D=2, P=1, n=(32, 32, 1), lo=(0.0, 0.0, 0.0), hi=(10.0, 10.0, 1.0), periodic=(1, 1, 1),
                         ic="vortex", u_inf=1.0, v_inf=1.0, c_dt=0.5),
    "blast3d_p2_64": dict(D=3, P=2, n=(64, 64, 64), lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0), periodic=(0, 0, 0),
                          ic="blast3d", c_dt=0.5),
}
GPU_IC = {"kh_noise": "kh_noise", "vortex": "isentropic_vortex", "blast3d": "blast3d"}
METRIC = "DOF-updates/s at 1 GB300: learned-seed+batched vs plain GPU FP64 vs CPU, at equal L2"


def _jsonable(o):
    """numpy scalars in the JSON line as plain numbers / booleans."""
    if hasattr(o, "item"):
        return o.item()
    raise TypeError(f"{type(o).__name__} is not JSON serializable")


def dist_env():
    return int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")), int(os.environ.get("LOCAL_RANK", "0"))


def max_over_ranks(x, dist=None, device="cpu"):
    """The largest x over the ranks of the process group (x itself alone)."""
    if dist is None:
        return x
    import torch

    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(units_per_rank, world, ms_max):
    """Replicas: every rank processes the same work; the job's rate is all
    ranks' units over the slowest rank's time."""
    return units_per_rank * world / (ms_max * 1e-3)


class ClockSampler:
    """nvidia-smi clock / throttle samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
            time.sleep(0.3)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        try:
            rows = [l.strip().split(",") for l in open(self.path) if l.strip()]
        except Exception:
            return out
        finally:
            try:
                os.unlink(self.path)
            except Exception:
                pass
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            r = [x.strip() for x in r]
            if len(r) < 9:
                continue
            try:
                sm.append(float(r[1]))
                mx.append(float(r[2]))
            except ValueError:
                continue
            for nm, v in zip(names, r[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if sm:
            out = {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                   "samples": len(sm)}
        return out


def make_sim(G, w, E=0, sweeps=0, seed=None, noise_amp=None):
    s = G.AmrDG(P=w["P"], D=w["D"])
    amr = w.get("amr", {})
    s.setGeometrySettings(prob_lo=w["lo"], prob_hi=w["hi"], n_cell=w["n"], periodic=w["periodic"],
                          max_level=amr.get("max_level", 0), max_grid=amr.get("max_grid", 1 << 20),
                          blocking_factor=amr.get("blocking_factor", 8), dtn_regrid=amr.get("dtn_regrid", 4))
    if amr:
        s.setAmrSettings(tag_kind=amr["tag_kind"], tag_threshold=amr["tag_threshold"])
    lim = w.get("limiter")
    s.settings(c_dt=w["c_dt"], elems_per_block=E, picard_sweeps=sweeps,
               **(dict(limiter_type="TVB", TVB_M=lim["TVB_M"], t_limit=lim["t_limit"]) if lim else {}))
    w = dict(w)
    if seed is not None:
        w["seed"] = seed
    if noise_amp is not None:
        w["noise_amp"] = noise_amp
    extra = {k: w[k] for k in ("seed", "noise_amp", "u_inf", "v_inf") if k in w}
    s.init(G.Compressible_Euler().settings(GPU_IC[w["ic"]], **extra))
    return s


def autotune(G, w, steps=3):
    """The library's autotuner (adg_autotune) on this workload: every
    elements-per-block choice of the plain predictor timed on the workload's
    own layout after two steps (state restored); the choice is recorded in
    the tune cache (ADG_TUNE_CACHE) and taken by the contexts created
    afterwards with elems_per_block = 0, which is what the timed runs use."""
    s = make_sim(G, w, 0)
    s.advance(2, use_graph=False)
    r = s.autotune(steps)
    s.close()
    return 0, {"E": r["E"], "predictor_ms": {str(k): v for k, v in r["ms"].items()}}


def autotune_seeded(G, w, seed, steps=3):
    """The same for the seeded FP32 predictor (two sweeps from the seed)."""
    s = make_sim(G, w, 0)
    seed.attach(s, mode=2, sweeps=2, tol=1e-3)
    s.advance(2, use_graph=False)
    r = s.autotune(steps)
    s.close()
    return {"E": r["E"], "predictor_ms": {str(k): v for k, v in r["ms"].items()}}


def oracle_sim(w):
    """The CPU oracle configured as the workload (same boxes as the GPU run)."""
    import oracle_ffi as O

    amr = w.get("amr", {})
    cfg = O.make_cfg(D=w["D"], P=w["P"], n=w["n"], lo=w["lo"], hi=w["hi"], periodic=w["periodic"],
                     ic=w["ic"], c_dt=w["c_dt"], max_grid=amr.get("max_grid", 1 << 20),
                     max_level=amr.get("max_level", 0), blocking_factor=amr.get("blocking_factor", 8),
                     dtn_regrid=amr.get("dtn_regrid", 4), tag_kind=amr.get("tag_kind", 0),
                     tag_threshold=amr.get("tag_threshold", 0.1),
                     **({"t_limit": w["limiter"]["t_limit"], "tvb_M": w["limiter"]["TVB_M"]} if "limiter" in w else {}),
                     **{k: w[k] for k in ("seed", "noise_amp", "u_inf", "v_inf") if k in w})
    return O.OracleSim(cfg)


def run_accuracy(args, w):
    """Plain FP64 GPU path against the CPU oracle on the workload from the
    same initial state for --steps steps: box layouts, the largest modal
    difference per level (relative to each variable's largest cell mean) and
    the exact L2 norm of the density difference over the level-0 field."""
    import numpy as np

    import adg_gb300 as G
    import oracle_ffi as O

    O.set_threads(os.cpu_count())
    o = oracle_sim(w)
    o.init()
    g = make_sim(G, w)
    for l in range(o.num_levels()):
        g.set_U_w(o.get_uw(l), l)
    g.Dt = o.dt
    t_cpu = t_gpu = 0.0
    same_layout = True
    for _ in range(args.steps):
        t0 = time.perf_counter()
        o.step()
        t1 = time.perf_counter()
        g.time_integration()
        g.Dt  # sync
        t2 = time.perf_counter()
        t_cpu += t1 - t0
        t_gpu += t2 - t1
        same_layout = same_layout and g.num_levels() == o.num_levels() and all(
            np.array_equal(g.boxes(l), o.boxes(l)) for l in range(o.num_levels()))

    def rel(a, b):
        scale = np.maximum(np.max(np.abs(b[:, :, 0]), axis=0), 1e-300)
        return float(np.max(np.max(np.abs(a - b), axis=(0, 2)) / scale))

    levels = [{"level": l, "cells": int(o.ncells_level(l)), "max_rel_modal": rel(g.get_U_w(l), o.get_uw(l))}
              for l in range(min(o.num_levels(), g.num_levels()))]
    line = {"accuracy": {"workload": args.workload, "steps": args.steps, "same_layout_every_step": same_layout,
                         "levels": levels,
                         "l2_density_level0": l2_density_level0(g.get_U_w(0), o.get_uw(0), w),
                         "dt_rel": abs(g.Dt - o.dt) / o.dt, "gpu_status": g.status(),
                         "limited": [g.limited_count(), o.limited_count()] if "limiter" in w else None,
                         "wall_s": {"oracle": t_cpu, "gpu_stream_steps": t_gpu}}}
    print(json.dumps(line, default=_jsonable))
    return 0


def cpu_baseline(w, max_seconds=20.0, threads=None, max_steps=50):
    """The oracle (C++/OpenMP restatement of the reference) on the host cores:
    a bounded sample of the same workload (whole grid, the steps after the
    first, which allocates and, with AMR, builds the first hierarchy from the
    initial full-domain levels; later regrids are inside the sample): up to
    max_steps steps or max_seconds."""
    import oracle_ffi as O
    from math import comb

    threads = threads or os.cpu_count()
    O.set_threads(threads)
    amr = w.get("amr", {})
    s = oracle_sim(w)
    s.init()
    per_cell = (w["D"] + 2) * comb(w["P"] + w["D"], w["D"])
    s.step()  # untimed, as the GPU arm's warm-up
    steps, dof, t0 = 0, 0, time.perf_counter()
    while True:
        s.step()
        steps += 1
        dof += sum(s.ncells_level(l) for l in range(s.num_levels())) * per_cell
        el = time.perf_counter() - t0
        if el > max_seconds or steps >= max_steps:
            break
    grid = "x".join(map(str, w["n"][:w["D"]]))
    what = f"{steps} steps of the full {grid}" + (f" base grid with {s.num_levels()} levels" if amr else " grid")
    return {"value": dof / el, "unit": "DOF-updates/s", "cores": threads, "kind": "port", "steps": steps,
            "ms_per_step": el * 1e3 / steps,
            "sample": f"{what} ({el:.1f} s), CPU oracle (reference algorithm restated in C++/OpenMP)"}


def base_config(args, w, world):
    """The workload keys both arms report (identical in both; how each arm ran
    goes under "run")."""
    return {"workload": args.workload, "D": w["D"], "P": w["P"], "base_cells": list(w["n"][:w["D"]]),
            "amr": w.get("amr"), "ic": w["ic"], "c_dt": w["c_dt"], "limiter": w.get("limiter")}


def run_reference(args, w):
    """The reference's algorithm on the host cores (the oracle: the reference
    itself cannot be built here) for --steps steps after one untimed step,
    unless that exceeds a few minutes; "steps" reports the steps timed."""
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    base = cpu_baseline(w, max_seconds=180.0, max_steps=max(1, args.steps))
    val = base["value"]
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": "DOF-updates/s", "n_gpus": args.gpus,
            "steps": base["steps"], "warmup": args.warmup, "ms_per_step": base["ms_per_step"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": base_config(args, w, 1),
            "run": {"parallelism": f"host cores of rank 0 ({base['cores']} threads)", "warmup_steps_run": 1},
            "cpu_baseline": base,
            "e2e": {"value": val, "unit": "DOF-updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line, default=_jsonable))
    return 0


# ---------------------------------------------------------------------------
# accuracy: exact L2 of the density difference over level 0 (coarse cells
# covered by finer levels hold the averaged-down fine solution, so level 0
# carries the whole field on a layout shared by every run)
# ---------------------------------------------------------------------------
def mass_diag(w):
    """Diagonal of the Legendre mass matrix, prod_d 2/(2k_d+1), in the
    reference's total-degree mode order (first index slowest)."""
    D, P = w["D"], w["P"]
    m = []

    def rec(prefix, left, depth):
        if depth == D:
            yield tuple(prefix)
            return
        for v in range(left + 1):
            yield from rec(prefix + [v], left - v, depth + 1)
    for n in rec([], P, 0):
        v = 1.0
        for k in n:
            v *= 2.0 / (2 * k + 1)
        m.append(v)
    return m


def l2_density_level0(Ua, Ub, w):
    import numpy as np
    M = np.array(mass_diag(w))
    d = Ua[:, 0, :] - Ub[:, 0, :]
    vol = 1.0
    for k in range(w["D"]):
        vol *= (w["hi"][k] - w["lo"][k])
    # cell integral of the squared difference = (cell volume / 2^D) sum_n M_n d_n^2
    ncell = Ua.shape[0]
    integral = (vol / ncell) / 2 ** w["D"] * float(np.sum(M[None, :] * d * d))
    return (integral / vol) ** 0.5


L2_FLUSH_BYTES = 256 << 20  # twice the 129 MB L2: written before every timed step

# Per launch of the dominant kernels on the headline workload (ncu, same
# code and layout; profiles/fp64_issue_k_predictor_kh_p3_amr3.md): warp
# instructions issued, FP64-pipe thread instruction slots
# (smsp__inst_executed_pipe_fp64 x 32), the DFMA+DADD+DMUL part of them, DRAM
# bytes read + written, issue and FP64 pipe activity, elements predicted.
PROFILED_LAUNCH = {
    "kh_p3_amr3": {
        "plain_predictor": dict(kernel="k_predictor_fx<D2P3, E=8> (3 Picard sweeps in fixed point, corrector volume "
                                       "term, face traces)",
                                inst=171.249e6, fp64_pipe_slots=41.351e6, fp64_arith=38.353e6, dram_bytes=31.01e6,
                                issue_active=0.502, fp64_active=0.242, elements=15616,
                                source="profiles/fp64_issue_k_predictor_kh_p3_amr3.md"),
        "seeded_predictor": dict(kernel="k_split_base<D2P3, E=8> (time-independent part in fixed point) and "
                                        "k_predictor<D2P3, E=8, MODE 2> (2 FP32 sweeps from the seed, FP32 changes)",
                                 inst=38.176e6, fp64_pipe_slots=5.309e6, fp64_arith=3.670e6, dram_bytes=29.57e6,
                                 issue_active=0.443, fp64_active=0.121, elements=15616,
                                 source="profiles/fp64_issue_k_predictor_kh_p3_amr3.md"),
    },
}


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}

SEED_VARIANTS = {"seed_1sweep_fp64": dict(mode=1, sweeps=1),
                 "seed_2sweeps_fp32": dict(mode=2, sweeps=2),
                 "seed_3sweeps_fp32": dict(mode=2, sweeps=3)}


def seed_cache_path(name):
    return os.path.join(ROOT, "ader-dg-amr_gb300", "_build", f"seed_{name}.npy")


# Adam schedules of the seed, (epochs, batch, learning rate) stages: the
# headline's (2 M pairs, 8 s on a GB300) and config 4's recipe for a single
# sweep from the seed (8 M pairs and a three-stage decay, about 70 s)
SEED_SCHEDULE = ((40, 8192, 1e-3), (20, 8192, 2e-4))
SEED_SCHEDULE_1SWEEP = ((80, 16384, 2e-3), (60, 16384, 5e-4), (40, 16384, 1e-4))


def train_seed(G, w, n_pairs=2_000_000, schedule=SEED_SCHEDULE, cache=None):
    """Learned seed trained on pairs from the Picard predictor (8 sweeps) of
    perturbed single-level and AMR runs of the workload's configuration (2D),
    or of the workload's own AMR run (3D).
    With `cache` (a file path), reuse the parameters stored there by an
    earlier run of the same workload, or store them after training."""
    import numpy as np

    seed = G.PredictorSeed(w["D"], w["P"], hidden=128, rng_seed=2024)
    if cache and os.path.exists(cache):
        seed.set_params(np.load(cache))
        return seed, {"cached": cache}
    t0 = time.perf_counter()
    runs = []
    base = dict(w)
    single = dict(w)
    single.pop("amr", None)
    single["n"] = tuple((w["n"][d] << w["amr"]["max_level"]) if d < w["D"] else 1 for d in range(3)) if "amr" in w else w["n"]
    k = 0
    if w["D"] == 3:
        # the 3D blast has no seeded perturbation and a 128^3 single level is
        # heavy: pairs from the workload's own AMR run, spread over its course
        s = make_sim(G, base)
        for st in range(100):
            if st % 12 == 11:
                seed.collect(s, target_sweeps=8)
                if seed.num_samples() >= n_pairs:
                    break
            s.time_integration()
        s.close()
    while seed.num_samples() < n_pairs and k < 16:
        cfgw = single if k % 2 == 0 else base
        s = make_sim(G, cfgw, seed=1000 + k, noise_amp=1e-3 * (1 + k % 4))
        for st in range(40):
            if st % 2 == 1:
                seed.collect(s, target_sweeps=8)
                if seed.num_samples() >= n_pairs:
                    break
            s.time_integration()
        s.close()
        k += 1
    t1 = time.perf_counter()
    loss = None
    for ep, batch, lr in schedule:
        loss = seed.train(ep, batch=batch, lr=lr)
    t2 = time.perf_counter()
    if cache:
        os.makedirs(os.path.dirname(cache), exist_ok=True)
        np.save(cache, seed.get_params())
    return seed, {"pairs": seed.num_samples(), "collect_s": t1 - t0, "train_s": t2 - t1, "final_loss": loss,
                  "epochs": sum(st[0] for st in schedule), "schedule": [list(st) for st in schedule]}


def timed_run(G, w, E, steps, warmup, seed=None, mode=0, sweeps=0, tol=1e-3, plain_sweeps=0, clocks=True):
    s = make_sim(G, w, E, sweeps=plain_sweeps)
    if seed is not None and mode:
        seed.attach(s, mode=mode, sweeps=sweeps, tol=tol)
    s.advance(warmup, use_graph=True)
    s.Dt  # sync
    d0, _ = s.dof_updates()
    lf0 = s.leaf_dof_updates()
    n0 = s.launch_count()
    r0 = s.regrid_count()
    ph0 = s.regrid_profile()
    local = dist_env()[2]
    with ClockSampler(local) as clk:  # nvidia-smi samples during the timed steps themselves
        ms = s.advance_timed_flushed(steps, flush_bytes=L2_FLUSH_BYTES, use_graph=True)
    d1, rms = s.dof_updates()
    ph1 = s.regrid_profile()
    out = {"ms": ms, "dof": d1 - d0, "launches": s.launch_count() - n0, "regrids": s.regrid_count() - r0,
           "regrid_host_ms": {k: ph1[k] - ph0[k] for k in ph1}, "sim": s, "dof_per_s": (d1 - d0) / (ms * 1e-3),
           "leaf_dof_per_s": (s.leaf_dof_updates() - lf0) / (ms * 1e-3), "clocks": clk.summary()}
    if seed is not None and mode:
        fb, n = G.seed_stats(s)
        out["fallback_rate"] = fb / max(1, n)
    return out


def leaf_masks(sim, w):
    """Per level, which valid cells (in the level's state order: x fastest
    over the level's index space) are not covered by the next finer level."""
    import numpy as np

    D, nl = w["D"], sim.num_levels()
    out = []
    for l in range(nl):
        n = [w["n"][d] << l for d in range(D)]
        mask = np.zeros(n[::-1], bool)
        for bx in sim.boxes(l):
            mask[tuple(slice(bx[d], bx[3 + d] + 1) for d in range(D))[::-1]] = True
        idx = np.argwhere(mask)
        leaf = np.ones(len(idx), bool)
        if l + 1 < nl:
            fm = np.zeros(n[::-1], bool)
            for bx in sim.boxes(l + 1):
                fm[tuple(slice(bx[d] // 2, bx[3 + d] // 2 + 1) for d in range(D))[::-1]] = True
            leaf = ~fm[tuple(idx.T)]
        out.append(leaf)
    return out


def same_layout(a, b):
    import numpy as np

    return a.num_levels() == b.num_levels() and all(
        np.array_equal(a.boxes(l), b.boxes(l)) for l in range(a.num_levels()))


def l2_density_leaf(sa, sb, w):
    """Exact modal L2 norm of the density difference of two runs with the same
    layout over the leaf cells of every level (the fine data where a level is
    refined, as the reference's LpNorm_DG_AMR counts it)."""
    import numpy as np

    M = np.array(mass_diag(w))
    vol_dom = 1.0
    for k in range(w["D"]):
        vol_dom *= w["hi"][k] - w["lo"][k]
    total = 0.0
    for l, leaf in enumerate(leaf_masks(sa, w)):
        d = sa.get_U_w(l)[leaf, 0, :] - sb.get_U_w(l)[leaf, 0, :]
        cell = vol_dom / np.prod([w["n"][k] << l for k in range(w["D"])])
        total += cell / 2 ** w["D"] * float(np.sum(M[None, :] * d * d))
    return (total / vol_dom) ** 0.5


def e2e_device_patches(G, s, w, steps):
    """The same metric through the zero-copy boundary: the state of every box
    of every level in its own per-variable device arrays laid out as AMReX
    FArrayBoxes (one ghost cell, modes as components); every step gathers the
    valid cells into the library (adg_read_patches), runs the step and
    scatters them back (adg_write_patches).  No host copies."""
    import torch

    D, Q = w["D"], w["D"] + 2
    Nps = s.Np_s
    keep = []

    def register():
        keep.clear()
        patches = []
        for l in range(s.num_levels()):
            for b in s.boxes(l):
                ext = [int(b[3 + d] - b[d] + 1 + 2) if d < D else 1 for d in range(3)]
                p = G.AdgPatch()
                p.level, p.nghost = l, 1
                for d in range(3):
                    p.lo[d], p.hi[d] = int(b[d]), int(b[3 + d])
                for q in range(Q):
                    a = torch.full((Nps, ext[2], ext[1], ext[0]), float("nan"), dtype=torch.float64, device="cuda")
                    keep.append(a)
                    p.U_w[q] = a.data_ptr()
                p.jstride, p.kstride, p.nstride = ext[0], ext[0] * ext[1], ext[0] * ext[1] * ext[2]
                patches.append(p)
        s.set_patches(patches)
        s.write_patches()
        return len(patches)

    torch.cuda.synchronize()
    npatch = register()
    L, ctx = s._L, s.ctx
    # one untimed step: a graph made stale by the caller's earlier settings
    # is captured again here, not in the timed steps
    if L.adg_read_patches(ctx) != 0 or L.adg_advance(ctx, 1, 1) != 0 or L.adg_write_patches(ctx) != 0:
        npatch = register()
    d0, _ = s.dof_updates()
    s.synchronize()
    t0 = time.perf_counter()
    reregistered = 0
    for _ in range(steps):
        if L.adg_read_patches(ctx) != 0:  # a regrid changed the layout: the caller re-binds its arrays
            npatch = register()
            reregistered += 1
            s.read_patches()
        if L.adg_advance(ctx, 1, 1) != 0:
            raise G.AdgError("adg_advance failed")
        if L.adg_write_patches(ctx) != 0:
            npatch = register()
            reregistered += 1
        s.synchronize()
    el = time.perf_counter() - t0
    d1, _ = s.dof_updates()
    return {"value": (d1 - d0) / el, "unit": "DOF-updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0,
            "patches": npatch, "rebinds_after_regrid": reregistered, "steps": steps,
            "path": "adg_read_patches + adg_advance(1 step, graph) + adg_write_patches per step on per-(box, q) "
                    "device arrays with one ghost cell (AMReX FArrayBox layout)"}


def sm_count():
    try:
        import torch

        return torch.cuda.get_device_properties(0).multi_processor_count, "this device's SMs"
    except Exception:
        return 152, "152 SMs (torch absent)"


def roofline_line(G, w, workload, head_name, km_head, km_plain, el_per_step, clocks):
    """roofline of the headline path's dominant kernels: instruction issue (the
    ncu-counted warp instructions of one launch over the live CUDA-event
    duration, against four a clock and SM at the SM clock sampled in this run),
    and beside it the FP64 pipe's (its instruction slots, 2 flops each, against
    the DFMA rate measured in this run)."""
    from math import comb

    D, P = w["D"], w["P"]
    Q, Nps = D + 2, comb(P + D, D)
    peak = G.fp64_peak_gflops() / 1e3
    alg, issued = G.flops_per_element(D, P)
    qbd = (P + 1) ** D
    alg_pred = alg - 2 * Q * 2 * D * Nps * qbd
    seeded = head_name.startswith("seed") and km_head.get("seed_inference", 0.0) > 0.0
    key = "seeded_predictor" if seeded else "plain_predictor"
    t = km_head["seeded_predictor"] if seeded else km_plain["predictor"]
    prof = PROFILED_LAUNCH.get(workload, {}).get(key)
    sms, sms_source = sm_count()
    mhz = (clocks or {}).get("sm_mhz") or 2070.0
    issue_peak = 4 * sms * mhz * 1e-3  # G warp instructions/s
    line = {"bound": "issue", "unit": "G warp instructions/s", "peak": issue_peak,
            "peak_source": f"four schedulers on each of {sms} SMs ({sms_source}) at {mhz:.0f} MHz "
                           + ("(sampled in the timed region)" if (clocks or {}).get("sm_mhz") else "(no clock sample)"),
            "fp64_peak_tflops": peak,
            "fp64_peak_source": "FP64 DFMA-chain probe on this GPU in this run (adg_fp64_peak_probe; "
                                "MEASURED_PEAKS.json has no FP64 figure)",
            "kernel_ms": t}
    if prof:
        achieved = prof["inst"] / (t * 1e-3) / 1e9
        line.update({
            "kernel": prof["kernel"], "achieved": achieved, "frac": achieved / issue_peak,
            "issue_active_ncu": prof["issue_active"],
            "fp64_issue_frac": 2.0 * prof["fp64_pipe_slots"] / (t * 1e-3) / 1e12 / peak,
            "traffic": prof["dram_bytes"], "traffic_source": prof["source"],
            "fp64_pipe_slots_per_launch": prof["fp64_pipe_slots"],
            "fp64_arith_frac": 2.0 * prof["fp64_arith"] / (t * 1e-3) / 1e12 / peak,
            "fp64_pipe_active_ncu": prof["fp64_active"],
            "elements_per_launch": prof["elements"],
            "effective_dense_tflops": alg_pred * prof["elements"] / (t * 1e-3) / 1e12,
            "note": ("achieved = the kernels' warp instructions per launch (ncu) / their event-timed duration, "
                     "cross-checked by issue_active_ncu; "
                     "effective_dense_tflops counts the method's dense matrix-form flops per element (" +
                     f"{alg_pred:.0f}) instead, which the generated sum-factorised operators do not issue"),
        })
    else:
        line.update({"kernel": key, "achieved": None, "frac": None, "traffic": None,
                     "effective_dense_tflops": alg_pred * el_per_step / (t * 1e-3) / 1e12,
                     "note": "no instruction count profiled for this workload"})
    return line


def seed_roofline(w, km_head, el_per_step, peak):
    """The TF32 tensor-core seed network and the seeded predictor's FP64 part."""
    from math import comb

    D, P = w["D"], w["P"]
    Q, Nps = D + 2, comb(P + D, D)
    Nst = comb(P + D + 1, D + 1)
    n_in, n_out, hid = Q * Nps + 1, Q * Nst, 128
    tf32 = 2 * (n_in * hid + 2 * hid * hid + hid * n_out)
    t_inf = km_head["seed_inference"]
    tf32_peak = measured_peaks().get("bf16_tflops", 1900.0) / 2.0
    a32 = tf32 * el_per_step / (t_inf * 1e-3) / 1e12
    return {"tf32_tensor": {"kernel": "k_seed_infer_tc (4 layers, tcgen05 kind::tf32)",
                            "algorithmic_flops_per_element": tf32, "elements_per_launch": el_per_step,
                            "ms": t_inf, "ms_source": "stage timing (adg_time_kernels: CUDA events around "
                                                      "the launch in a stream-launched step, 3 steps)",
                            "achieved": a32,
                            "peak": tf32_peak, "unit": "TFLOP/s", "frac": a32 / tf32_peak,
                            "peak_source": "half the measured dense bf16 burst (MEASURED_PEAKS.json)"},
            "fallback_ms": km_head.get("fallback")}


OTHER_CONFIGS = ("vortex_p1_32", "kh_p3_256", "blast3d_p2_amr2")


def run_other_configs(G, args):
    """The other benchmark configurations at their stated sizes, plain FP64
    (and the 3D blast with its learned seed), timed the same way."""
    out = {}
    for name in OTHER_CONFIGS:
        w = WORKLOADS[name]
        steps = min(args.steps, 20)
        r = timed_run(G, w, 0, steps, 3)
        entry = {"plain_fp64": {"value": r["dof_per_s"], "ms_per_step": r["ms"] / steps, "steps": steps,
                                "leaf_value": r["leaf_dof_per_s"], "clocks": r["clocks"]}}
        r["sim"].close()
        if "amr" in w and not args.no_seed:
            seed, info = train_seed(G, w, n_pairs=1_000_000, schedule=((30, 8192, 1e-3), (15, 8192, 2e-4)))
            rs = timed_run(G, w, 0, steps, 3, seed=seed, mode=2, sweeps=2, tol=1e-3)
            entry["seed_2sweeps_fp32"] = {"value": rs["dof_per_s"], "ms_per_step": rs["ms"] / steps,
                                          "fallback_rate": rs.get("fallback_rate"), "seed_training": info,
                                          "clocks": rs["clocks"]}
            rs["sim"].close()
            seed.close()
        out[name] = entry
    return out


def run_ours(args, w):
    rank, world, local = dist_env()
    import adg_gb300 as G
    import numpy as np

    G.set_device(local)
    dist = None
    if world > 1:
        import torch
        import torch.distributed as tdist

        torch.cuda.set_device(local)
        tdist.init_process_group("nccl")
        dist = tdist

    def barrier_max(x):
        return max_over_ranks(x, dist, f"cuda:{local}")

    from math import comb
    Q = w["D"] + 2
    Nps = comb(w["P"] + w["D"], w["D"])
    E, tune = autotune(G, w)
    variants = {}
    seed = None
    seed_info = None
    is_amr = "amr" in w
    only = args.only
    tune_seeded = None
    if is_amr and not args.no_seed and only != "plain_fp64":
        seed, seed_info = train_seed(G, w, cache=seed_cache_path(args.workload) if args.seed_cache else None)
        tune_seeded = autotune_seeded(G, w, seed)
    if only:  # one variant, for profiling: no accuracy reference, no JSON contract line
        kw = SEED_VARIANTS.get(only, {})
        r = timed_run(G, w, E, args.steps, args.warmup, seed=seed if kw else None, **kw,
                      plain_sweeps=1 if only == "noseed_1sweep_fp64" else 0)
        if rank == 0:
            print(json.dumps({"variant": only, **{k: v for k, v in r.items() if k != "sim"},
                              "kernel_ms": r["sim"].time_kernels(3)}))
        return 0
    # plain FP64 path (P sweeps)
    plain = timed_run(G, w, E, args.steps, args.warmup)
    variants["plain_fp64"] = plain
    accuracy = None
    if seed is not None:
        ref = make_sim(G, w, E, sweeps=8)  # converged Picard, accuracy reference
        ref.advance(args.warmup + args.steps, use_graph=True)
        U_ref = ref.get_U_w(0)
        for name, kw in SEED_VARIANTS.items():
            variants[name] = timed_run(G, w, E, args.steps, args.warmup, seed=seed, tol=1e-3, **kw)
        variants["noseed_1sweep_fp64"] = timed_run(G, w, E, args.steps, args.warmup, plain_sweeps=1)
        c4_info = None
        if not args.no_config4_recipe:  # config 4 as stated: one sweep from a seed trained longer
            seed4, c4_info = train_seed(G, w, n_pairs=8_000_000, schedule=SEED_SCHEDULE_1SWEEP)
            for name, kw in (("c4_seed_1sweep_fp64", dict(mode=1, sweeps=1)),
                             ("c4_seed_1sweep_fp32", dict(mode=2, sweeps=1))):
                variants[name] = timed_run(G, w, E, args.steps, args.warmup, seed=seed4, tol=1e-3, **kw)
        orc = None
        if not args.no_oracle_accuracy:
            import oracle_ffi as O

            O.set_threads(os.cpu_count())
            orc = oracle_sim(w)
            orc.init()
            for _ in range(args.warmup + args.steps):
                orc.step()
        for v in variants.values():
            sv = v["sim"]
            v["l2_density_vs_converged"] = l2_density_level0(sv.get_U_w(0), U_ref, w)
            v["l2_density_leaf_vs_converged"] = l2_density_leaf(sv, ref, w) if same_layout(sv, ref) else None
            if orc is not None and same_layout(sv, orc):
                v["l2_density_leaf_vs_oracle"] = orc.norm_diff([sv.get_U_w(l) for l in range(sv.num_levels())], 2, 0)
        plain_err = variants["plain_fp64"]["l2_density_vs_converged"]
        plain_leaf = variants["plain_fp64"].get("l2_density_leaf_vs_converged")

        def passes(v):  # within 1.01x of the plain path on the level-0 field and on the leaf cells
            leaf = v.get("l2_density_leaf_vs_converged")
            return (v["l2_density_vs_converged"] <= 1.01 * plain_err and
                    (leaf is None or plain_leaf is None or leaf <= 1.01 * plain_leaf))
        ok = {k: v for k, v in variants.items() if (k.startswith("seed") or k.startswith("c4_")) and passes(v)}
        head_name = max(ok, key=lambda k: ok[k]["dof_per_s"]) if ok else "plain_fp64"
        accuracy = {
            "criterion": "L2 density against a converged-Picard (8 FP64 sweeps) run of the same workload after the "
                         "same steps within 1.01x of the plain FP64 path's, on the level-0 field (exact modal norm) "
                         "and on the leaf cells of every level: the headline variant passes both",
            "plain": plain_err, "headline": variants[head_name].get("l2_density_vs_converged"),
            "leaf_cells": {"plain": plain_leaf, "headline": variants[head_name].get("l2_density_leaf_vs_converged"),
                           "headline_passes": (None if plain_leaf is None or
                                               variants[head_name].get("l2_density_leaf_vs_converged") is None else
                                               variants[head_name]["l2_density_leaf_vs_converged"] <= 1.01 * plain_leaf)},
            "vs_fp64_oracle": {k: v.get("l2_density_leaf_vs_oracle") for k, v in variants.items()},
            "vs_fp64_oracle_note": ("the oracle runs the reference's algorithm (P = 3 FP64 sweeps): the plain path "
                                    "differs from it by rounding only, so against the oracle every seeded variant's "
                                    "figure is its deviation from the reference's predictor, not an error that the "
                                    "1.01x criterion can compare"),
            "config4_as_stated": {v: {"l2_level0": variants[v]["l2_density_vs_converged"],
                                      "l2_leaf": variants[v].get("l2_density_leaf_vs_converged"),
                                      "passes_level0": bool(variants[v]["l2_density_vs_converged"] <= 1.01 * plain_err),
                                      "passes_leaf": (None if variants[v].get("l2_density_leaf_vs_converged") is None
                                                      or plain_leaf is None else
                                                      bool(variants[v]["l2_density_leaf_vs_converged"]
                                                           <= 1.01 * plain_leaf)),
                                      "dof_per_s": variants[v]["dof_per_s"]}
                                  for v in ("seed_1sweep_fp64", "c4_seed_1sweep_fp64", "c4_seed_1sweep_fp32")
                                  if v in variants},
            "config4_seed_training": c4_info,
        }
    else:
        head_name = "plain_fp64"
    head = variants[head_name]
    ms = barrier_max(head["ms"])
    value = whole_job_rate(head["dof"], world, ms)

    # end to end through the C ABI with host buffers: every step copies the
    # state of every level in from page-locked host memory (one packed copy),
    # runs the step (graph replay) and reads every level back out (the step
    # readback: each level's copy starts once the step has finished writing
    # it, beside the step's tail); the host waits once per step for the result
    s = head["sim"]
    L, ctx = s._L, s.ctx
    e2e_steps = max(50, args.steps)  # host-timed: enough steps (and regrids) to average the host's jitter

    def check(rc, what):
        if rc != 0:
            raise G.AdgError(f"{what} failed (status {rc})")

    def level_cells():
        return [s.level_cells(l) for l in range(s.num_levels())]

    # one page-locked host copy of every level packed in level order, sized
    # for the largest layout (every level fully refined) and registered for
    # the step readback (adg_set_readback): the state goes in with one copy
    # and each level's result comes back beside the step's tail
    amr_levels = w.get("amr", {}).get("max_level", 0) + 1
    full = 0
    for lev in range(amr_levels):
        c = 1
        for d in range(w["D"]):
            c *= w["n"][d] << lev
        full += c
    host = G.PinnedArray((full, Q, Nps))
    ptr = host.array.ctypes.data
    check(L.adg_get_state(ctx, G.ADG_ALL_LEVELS, ptr, G.ADG_MEM_HOST), "adg_get_state")
    check(L.adg_set_readback(ctx, G.ADG_ALL_LEVELS, ptr, full), "adg_set_readback")
    s.advance(1, use_graph=True)  # capture the step with its readback copies before timing
    s.synchronize()
    h2d = d2h = 0
    t0 = time.perf_counter()
    d_before, _ = s.dof_updates()
    for _ in range(e2e_steps):
        n0 = sum(level_cells())
        check(L.adg_set_state(ctx, G.ADG_ALL_LEVELS, ptr, G.ADG_MEM_HOST_ASYNC), "adg_set_state")
        h2d += n0 * Q * Nps * 8
        check(L.adg_advance(ctx, 1, 1), "adg_advance")
        n1 = sum(level_cells())
        if not s.readback_active(G.ADG_ALL_LEVELS):  # cannot happen with the full-size buffer
            check(L.adg_get_state(ctx, G.ADG_ALL_LEVELS, ptr, G.ADG_MEM_HOST_ASYNC), "adg_get_state")
        d2h += n1 * Q * Nps * 8
        check(L.adg_synchronize(ctx), "adg_synchronize")
    e2e_s = barrier_max(time.perf_counter() - t0)
    d_after, _ = s.dof_updates()
    e2e_val = (d_after - d_before) * world / e2e_s
    check(L.adg_set_readback(ctx, G.ADG_ALL_LEVELS, None, 0), "adg_set_readback")
    s.synchronize()
    host.free()
    try:
        e2e_dev = e2e_device_patches(G, s, w, e2e_steps)
    except Exception as ex:  # torch absent or no device memory: report, do not fail the line
        e2e_dev = {"unavailable": f"{type(ex).__name__}: {ex}"}

    km_plain = plain["sim"].time_kernels(3)
    seeded = head_name.startswith("seed")
    n_seed0 = G.seed_stats(head["sim"])[1] if seeded else 0
    km_head = head["sim"].time_kernels(3)
    el_per_step = plain["dof"] / args.steps / (Q * Nps)
    roof = roofline_line(G, w, args.workload, head_name, km_head, km_plain, el_per_step, head["clocks"])
    if seeded and km_head.get("seed_inference", 0.0) > 0.0:
        # the seed network runs over every element of the layout, the
        # coarse-fine ghosts included: its count over the same three steps
        seed_el = (G.seed_stats(head["sim"])[1] - n_seed0) / 3.0
        roof["seed_path"] = seed_roofline(w, km_head, seed_el, roof["fp64_peak_tflops"])
    line = {
        "metric": METRIC, "value": value, "unit": "DOF-updates/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64" if head_name == "plain_fp64" else "f64+f32",
        "dtype_detail": ("FP64 state, corrector, numerical flux, final-stage fluxes and face physics; predictor "
                         "operators and the sweeps' fluxes in 60-bit fixed point with one exponent per column"
                         if head_name == "plain_fp64" else
                         "FP64 state, corrector and numerical-flux moments; the time-independent part of the "
                         "predictor in 60-bit fixed point; FP32 Picard sweeps and flux changes; TF32 tensor-core "
                         "seed network"),
        "data": "synthetic",
        "config": base_config(args, w, world),
        "run": {"path": head_name, "autotune": {"plain": tune, "seeded": tune_seeded}, "cuda_graph": True,
                "parallelism": "replicas" if world > 1 else "1 GPU",
                "l2": f"flushed before every timed step ({L2_FLUSH_BYTES >> 20} MiB device memset, outside "
                      "the per-step CUDA-event intervals that are summed)"},
        "leaf_value": head["leaf_dof_per_s"] * world,
        "e2e": {"value": e2e_val, "unit": "DOF-updates/s", "h2d_bytes_per_step": h2d // e2e_steps,
                "d2h_bytes_per_step": d2h // e2e_steps, "steps": e2e_steps,
                "path": "per step: adg_set_state(ADG_ALL_LEVELS) from page-locked host memory (one copy), "
                        "adg_advance(1 step, graph) with the packed step readback (adg_set_readback: each "
                        "level copied to the host buffer once the step has written it), adg_synchronize; "
                        "host-timed"},
        "e2e_device_patches": e2e_dev,
        "roofline": roof,
        "kernel_ms": {"plain": km_plain, "headline": km_head},
        "variants": {k: {kk: vv for kk, vv in v.items() if kk != "sim"} for k, v in variants.items()},
        "gpu_launches": head["launches"],
        "clocks": head["clocks"],
        "status": head["sim"].status(),
    }
    if seed_info:
        line["seed_training"] = dict(seed_info)
        cost = seed_info.get("collect_s", 0.0) + seed_info.get("train_s", 0.0)
        gain_ms = (variants["plain_fp64"]["ms"] - head["ms"]) / args.steps
        line["seed_training"]["collect_plus_train_s"] = cost
        line["seed_training"]["break_even_steps"] = (cost * 1e3 / gain_ms) if gain_ms > 0 else None
        line["seed_training"]["note"] = ("collection (Picard predictor on perturbed runs) and training are outside "
                                         "the timed steps; break_even_steps = their time / the per-step saving of "
                                         "the headline path over the plain FP64 path")
    if accuracy:
        line["equal_l2"] = accuracy
    if not args.no_other_configs and rank == 0:
        line["other_configs"] = run_other_configs(G, args)
    if rank == 0:
        if world == 1 and not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(w, max_seconds=args.cpu_seconds)
        print(json.dumps(line, default=_jsonable))
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="kh_p3_amr3", choices=list(WORKLOADS))
    ap.add_argument("--no-seed", action="store_true")
    ap.add_argument("--cpu-seconds", type=float, default=20.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-oracle-accuracy", action="store_true",
                    help="skip the equal-L2 comparison of every variant with the FP64 oracle")
    ap.add_argument("--no-config4-recipe", action="store_true",
                    help="skip config 4's single-sweep recipe (a longer-trained seed, about a minute)")
    ap.add_argument("--no-other-configs", action="store_true",
                    help="skip the timing of the other benchmark configurations")
    ap.add_argument("--only", default=None,
                    choices=["plain_fp64", "noseed_1sweep_fp64"] + list(SEED_VARIANTS),
                    help="time one variant only and print its record (profiling runs)")
    ap.add_argument("--accuracy", action="store_true",
                    help="compare the plain GPU path with the CPU oracle over --steps steps and print the errors")
    ap.add_argument("--seed-cache", action="store_true",
                    help="reuse (or store) the trained seed parameters under the package build folder")
    args = ap.parse_args()
    args.warmup = max(3, args.warmup)
    w = WORKLOADS[args.workload]
    if args.impl == "reference":
        return run_reference(args, w)
    if args.accuracy:
        return run_accuracy(args, w)
    return run_ours(args, w)


if __name__ == "__main__":
    sys.exit(main())
