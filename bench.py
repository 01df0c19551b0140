#!/usr/bin/env python
"""Headline benchmark: Barnes-Hut KDK particle-steps/s on one GB300.

Workload (default): the two-component galaxy, N = 4,194,304 (Hernquist halo
3,774,874 + exponential disk 419,430), G = 1, eps = 0.002, dt = 2e-4,
monopole+quadrupole, split precision, plain theta-MAC.  A step is one KDK
leapfrog step (kick-drift, 63-bit keys, radix sort, octree, moments, grouped
walk with P2P/P2C, closing kick) over the whole system.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Headline: the learned opening test against the plain theta test at equal
rms relative force error (1e-3, FP64-summed direct sum on 4,096 targets).
Setup, untimed: for each leaf capacity of --leaf-grid (the target-group
size), the network is trained on the run itself (16 snapshots, 2^22
labelled pairs, 8 epochs), and theta and the learned budget are each set to the
largest grid value whose error stays within the target; each arm then runs
at the leaf capacity whose calibrated evaluation is fastest, with the
faster of the two walk-stack sizes.  Both arms
step the same input state K times.

value   = N * K / (device time of the learned arm's K timed steps, CUDA
          events on the engine's stream), inputs resident in HBM; the theta
          arm's figure and the ratio are in config.
e2e     = the same metric through the C-ABI with host buffers: per step
          ngrav_gpu_set_state_f32 from pinned host memory, ngrav_gpu_step(1),
          ngrav_gpu_get_state into pinned FP64 arrays, wall clock (20 steps;
          the three calls' shares are on the line).
drift   = energy, momentum and angular-momentum drift of each arm over its
          timed steps (FP64 diagnostics; the potential is the exact pair sum
          with FP32 pair terms and FP64 sums).
roofline: the evaluation kernel (P2P + P2C, FP32 pipe): algorithmic
          flops (20 per P2P pair + 60 per P2C term, device-counted) / its
          event-timed duration, against the measured FP32 FMA peak.
roofline_p2p: the evaluation kernel's P2P phase alone (a 262,144-particle
          Plummer sphere at theta 0: every pair near, no P2C), 20 flops per
          pair over its event time, against the same FP32 peak.
roofline_sort: the HBM-bound part of the tree build (radix sort + the
          permutation into key order), algorithmic bytes / event time of
          that phase, against the measured copy bandwidth.
cpu_baseline: the oracle (C restatement of the reference's CPU path) on the
          host cores, bounded sample: full tree build + walk over every
          k-th leaf group, extrapolated to a full step; its own rms error
          against the FP64 direct sum is stated.
configs: compact records of the task's other configurations: C2 (Plummer
          1M, plain vs split precision, 100 steps, error and drift), C3 (512-
          system ensemble, autotuned, graph steps) and C5 (16.8M cold
          collapse, 200 steps, error and key-depth limit every 20 steps);
          --workload plummer1m / ensemble512 / collapse16m runs each alone.
With --gpus N > 1 (torchrun), each rank runs an independent replica (the
path has no data-parallel split on one system); value sums the replicas.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import __graft_entry__ as ge  # noqa: E402

WORKLOADS = {
    # name: (generator, kwargs, eps, dt, theta, leaf capacity)
    "galaxy4m": ("galaxy", {}, 0.002, 2e-4, 0.6, 16),
    "galaxy1m": ("galaxy", {"n_halo": 943718, "n_disk": 104858}, 0.002, 2e-4, 0.6, 16),
    "plummer1m": ("plummer", {"n": 1048576, "seed": 1}, 0.005, 5e-4, 0.5, 16),
    "plummer16k": ("plummer", {"n": 16384, "seed": 0}, 0.01, 1e-3, 0.5, 16),
    # cold collapse of a uniform ball, 16.8M, learned test (its own line: collapse_run)
    "collapse16m": ("uniform_ball", {"n": 16777216, "seed": 4}, 0.001, 1e-4, 0.6, 32),
    # 512 Plummer spheres, N_i log-uniform in [1024, 65536] (~7.9M), one launch per phase
    "ensemble512": ("ensemble", {"nsys": 512}, 0.01, 1e-3, 0.6, 16),
}
# DRAM bytes (read + write) per interaction-list entry of one eval_kernel launch,
# from dram__bytes_read.sum + dram__bytes_write.sum of one ncu capture at
# N = 1,048,576, leaf capacity 48, learned test (211.8 + 14.9 MB for 7.57e7
# entries; profiles/eval_kernel_galaxy1m.txt).  The lists, the first touch of
# the particles and the closing kick are the kernel's DRAM stream, so traffic
# scales with entries.
EVAL_DRAM_BYTES_PER_LIST_ENTRY = 3.00
METRIC = "particle-steps/s at N=4M, learned-MAC vs plain θ-MAC at equal 1e-3 rms force err"


def dist_env():
    return int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")), \
        int(os.environ.get("LOCAL_RANK", "0"))


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.rows = []
        self._stop = threading.Event()
        self._proc = None
        self._t = None

    def start(self):
        try:
            self._proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except (FileNotFoundError, OSError):
            self._proc = None
            return
        self._t = threading.Thread(target=self._read, daemon=True)
        self._t.start()

    def _read(self):
        for line in self._proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) == 7:
                self.rows.append(parts)

    def stop(self):
        if self._proc:
            self._proc.terminate()
            try:
                self._proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self._proc.kill()
        if self._t:
            self._t.join(timeout=5)
        sm = [float(r[0]) for r in self.rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({names[k] for r in self.rows for k in range(4) if r[3 + k].lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def make_inputs(pkg_ic, workload):
    gen, kw, eps, dt, theta, ncrit = WORKLOADS[workload]
    arrs = getattr(pkg_ic, gen)(**kw)
    if gen == "ensemble":
        arrs = arrs[0]  # offsets: see run_ensemble
    return arrs, eps, dt, theta, ncrit


def ensemble_run(pkg, ic, dev, steps, warmup, tune_reps=2, clocks=None):
    """C3: 512 independent Plummer spheres (log-uniform N in [1024, 65536],
    system i seed i, ~7.9M particles), eps 0.01, theta 0.6, dt 1e-3: the
    leaf capacity autotuned, one launch per phase for all systems, CUDA-graph
    steps; per-system force error on 256 targets each (FP32 pairs, FP64
    sums) and per-system energy drift over the timed steps (exact FP64 pair
    potential of each system)."""
    gen, kw, eps, dt, theta, ncrit = WORKLOADS["ensemble512"]
    arrs, off = ic.ensemble(**kw)
    n, nsys = len(arrs[0]), len(off) - 1
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=theta, dt=dt), leaf_capacity=ncrit, device=dev,
                         timing=True) as sim:
        sim.set_particles_f32(*arrs)
        sim.set_ensemble(off)
        sim.prime()
        tune = sim.autotune(reps=tune_reps, check_targets=4096)
        sim.prime()
        st, ms_step, clk, (d0, d1) = timed(sim, steps, warmup, dt, clocks,
                                           diag=lambda: sim.ensemble_diagnostics(exact_potential=True))
        rms, mx = sim.ensemble_force_error(256, seed=1)
    dE = np.array([(b["energy"] - a["energy"]) / abs(a["energy"]) for a, b in zip(d0, d1)])
    flops = 20.0 * st["cum_p2p_pairs"] + 60.0 * st["cum_p2c_terms"]
    achieved = flops / (st["cum_ms_force"] * 1e-3) / 1e12 if st["cum_ms_force"] > 0 else None
    return {"n": n, "systems": nsys, "n_min": int(np.diff(off).min()), "n_max": int(np.diff(off).max()),
            "eps": eps, "theta": theta, "dt": dt, "steps": steps, "warmup": warmup,
            "value": n / (ms_step * 1e-3), "ms_per_step": ms_step, "leaf_capacity": tune["leaf_capacity"],
            "autotune": tune, "graph_replays": st["graph_replays"], "gpu_launches": st["cum_launches"],
            "p2p_pairs_per_step": st["cum_p2p_pairs"] / max(1, st["cum_evals"]),
            "p2c_terms_per_step": st["cum_p2c_terms"] / max(1, st["cum_evals"]),
            "eval_tflops": achieved, "ms_phases_last_eval": phases(st),
            "per_system_force_err_rms": {"median": float(np.median(rms)), "max": float(rms.max()),
                                         "targets_per_system": 256},
            "per_system_force_err_max": float(mx.max()),
            "per_system_energy_drift": {"median_abs": float(np.median(np.abs(dE))), "max_abs": float(np.abs(dE).max())},
            "clocks": clk}


def run_ensemble(args, pkg, ic, rank, world, dev):
    """The C3 ensemble as its own bench line."""
    r = ensemble_run(pkg, ic, dev, args.steps, args.warmup, clocks=ClockSampler(dev))
    peak = pkg.probe_fp32_peak(dev)
    if rank == 0:
        line = {
            "metric": "particle-steps/s, ensemble of 512 Plummer spheres (log-uniform N in [1024, 65536])",
            "value": world * r["value"], "unit": "particle-steps/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": r["ms_per_step"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded Plummer generator, system i seed i)",
            "config": {"workload": "ensemble512", **{k: v for k, v in r.items() if k not in ("clocks", "value")}},
            "roofline": {"bound": "fp32", "achieved": r["eval_tflops"], "peak": peak, "unit": "TFLOP/s",
                         "frac": (r["eval_tflops"] / peak) if r["eval_tflops"] and peak else None, "traffic": None,
                         "kernel": "eval_kernel (P2P 20 flops/pair + P2C 60 flops/term)"},
            "cpu_baseline": None, "e2e": None, "gpu_launches": r["gpu_launches"], "clocks": r["clocks"],
        }
        print(json.dumps(line), flush=True)
    return 0


def precision_run(pkg, ic, dev, steps=100):
    """C2: Plummer N = 1,048,576 (seed 1), eps 0.005, theta 0.5, leaf
    capacity 16, monopole + quadrupole, KDK dt 5e-4 for `steps` steps, in
    PLAIN (FP32 absolute positions, plain sums) and SPLIT precision
    (double-float state, leaf-frame FP32 offsets, Kahan sums; FP64 only in
    the top moments and the diagnostics).  Each: rms / max / median relative
    force error against the FP64 direct sum (FP64 pair terms) on 4,096
    uniformly sampled targets, at the start and after the steps, and the
    energy, momentum and angular-momentum drift (exact pair potential)."""
    arrs = ic.plummer(1048576, seed=1)
    eps, dt, theta = 0.005, 5e-4, 0.5
    mtot = float(np.sum(arrs[6], dtype=np.float64))
    out = {"n": 1048576, "eps": eps, "theta": theta, "dt": dt, "leaf_capacity": 16, "steps": steps}
    for name, prec in (("plain", pkg.PRECISION_PLAIN), ("split", pkg.PRECISION_SPLIT)):
        with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=theta, dt=dt), leaf_capacity=16, precision=prec,
                             device=dev, timing=True) as sim:
            sim.set_particles_f32(*arrs)
            sim.prime()
            fe0 = sim.force_error(4096, seed=2024, fp64_pairs=True)
            d0 = sim.diagnostics(exact_potential=2)
            sim.reset_cumulative()
            sim.step(steps, dt)
            st = sim.stats()
            d1 = sim.diagnostics(exact_potential=2)
            fe1 = sim.force_error(4096, seed=2024, fp64_pairs=True)
        out[name] = {"force_err_start": {k: fe0[k] for k in ("rms", "max", "median")},
                     "force_err_end": {k: fe1[k] for k in ("rms", "max", "median")},
                     **drift(d0, d1, mtot), "ms_per_step": st["cum_ms_step"] / steps,
                     "value": 1048576 / (st["cum_ms_step"] / steps * 1e-3)}
    return out


def collapse_run(pkg, ic, dev, steps=200, every=20, model=None, budget=None, energy=False, n=16777216):
    """C5: cold collapse of a uniform ball, N = 16,777,216 (cube rejection,
    seed 4), at rest, G = 1, eps 0.001, KDK dt 1e-4 for `steps` steps with the
    learned opening test (trained on this run unless a model is given; its
    budget, unless given, calibrated on the initial state to the largest
    grid value whose rms error stays within 0.95 x 1e-3, the margin for the
    error's growth during the run), split precision, CUDA-graph steps.  Every `every`
    steps: the rms / max force error against the direct sum (FP32 pairs,
    FP64 sums) on 4,096 targets, the leaves at the 21-level key limit, and
    |L|; energy (exact pair potential, FP32 pair terms, about a minute at
    this N) at the start and the end when `energy`."""
    arrs = ic.uniform_ball(n, seed=4)
    eps, dt = 0.001, 1e-4
    mtot = float(np.sum(arrs[6], dtype=np.float64))
    rec = {"n": n, "eps": eps, "dt": dt, "steps": steps, "mac": "learned", "budget": budget, "timeline": []}
    with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=0.6, dt=dt), leaf_capacity=32, device=dev,
                         timing=True) as sim:
        sim.set_particles_f32(*arrs)
        sim.prime()
        t0 = time.perf_counter()
        if model is None:
            rec["train"] = sim.lmac_train(snapshots=4, steps_between=1, dt=dt, pairs=1 << 21, epochs=4, batch=8192,
                                          seed=1)
            model = sim.lmac_get_model()
            sim.set_particles_f32(*arrs)
            sim.prime()
        rec["train_wall_s"] = time.perf_counter() - t0
        sim.lmac_set_model(*model)
        sim.set_opts(mac=pkg.MAC_LEARNED)
        screen = None
        if budget is None:
            # the screen factor too: the relative error near the ball's centre,
            # where |a| -> 0, is more sensitive to the error bound's slack
            best = None
            for scr in (1000.0, 300.0):
                def set_budget(v, scr=scr):
                    sim.lmac_set_opts(budget=v, check_every=0, screen=scr)
                b, tab = calibrate(sim, COLLAPSE_BUDGET_GRID, set_budget, target=0.95 * TARGET_RMS, stop=1.3)
                set_budget(b)
                ms = []
                for _ in range(3):
                    sim.compute_accel()
                    ms.append(sum(phases(sim.stats()).values()))
                ms = min(ms)
                if best is None or ms < best[0]:
                    best = (ms, scr, b, tab)
            _, screen, budget, rec["calibration"] = best
            rec["budget"], rec["screen"] = budget, screen
        kw = {} if screen is None else {"screen": screen}
        sim.lmac_set_opts(budget=budget, check_every=10, check_targets=CHECK_TARGETS, revert_rms=1.5e-3, **kw)
        sim.prime()
        d0 = sim.diagnostics(exact_potential=2 if energy else 0)
        ms = 0.0
        for k in range(steps // every):
            sim.reset_cumulative()
            sim.step(every, dt)
            st = sim.stats()
            ms += st["cum_ms_step"]
            fe = sim.force_error(4096, seed=100 + k, fp64_pairs=False)
            d = sim.diagnostics(exact_potential=0)
            rec["timeline"].append({"step": (k + 1) * every, "ms_per_step": st["cum_ms_step"] / every,
                                    "force_err_rms": fe["rms"], "force_err_max": fe["max"],
                                    "depth_limited_leaves": st["depth_limited_leaves"], "levels": st["levels"],
                                    "L_mag": float(np.linalg.norm(d["L"])), "lmac_active": st["lmac_active"]})
        st = sim.stats()
        d1 = sim.diagnostics(exact_potential=2 if energy else 0)
    rec["ms_per_step"] = ms / steps
    rec["value"] = n / (rec["ms_per_step"] * 1e-3)
    rec["lmac_reverted"] = bool(st["lmac_reverted"])
    rec["lmac_checks"] = st["lmac_checks"]
    rec["L_scale"] = float(np.sqrt(2.0 * mtot * max(d1["kinetic"], 1e-300)))  # |L| per unit length at the end
    if energy:
        rec.update(drift(d0, d1, mtot))
    else:
        rec["energy_drift"] = None
        rec["energy_drift_note"] = "exact potential at 16.8M takes about a minute; run --workload collapse16m"
    return rec


def cpu_error(O, x, y, z, m, eps, acc, ntargets=4096, seed=7):
    """rms / max relative error of the oracle's sampled Barnes-Hut
    accelerations against its FP64 direct sum, on ntargets of the walked
    targets (the accuracy the CPU arm runs at)."""
    ax, ay, az = acc
    walked = np.flatnonzero(np.isfinite(ax))
    rng = np.random.default_rng(seed)
    t = np.sort(rng.choice(walked, size=min(ntargets, walked.size), replace=False))
    dx, dy, dz = O.direct_targets(x, y, z, m, 1.0, eps, t)
    ref = np.sqrt(dx ** 2 + dy ** 2 + dz ** 2)
    e = np.sqrt((ax[t] - dx) ** 2 + (ay[t] - dy) ** 2 + (az[t] - dz) ** 2) / ref
    return {"rms": float(np.sqrt(np.mean(e ** 2))), "max": float(e.max()), "targets": int(t.size)}


def cpu_baseline(orc, arrs, eps, theta, ncrit, target_s=15.0):
    """Oracle on the host cores: full tree + a strided sample of leaf groups,
    and the rms error of that sample against the FP64 direct sum."""
    O = orc.Oracle()
    x, y, z, _, _, _, m = (a.astype(np.float64) for a in arrs)
    n = len(x)
    stride = max(1, int(n // 65536))
    build_ms, walk_ms, frac, _ = O.time_sampled(x, y, z, m, 1.0, eps, theta, ncrit, stride)
    # grow the sample while it is short of the target
    while build_ms + walk_ms < 1e3 * target_s * 0.3 and stride > 1:
        stride = max(1, stride // 4)
        build_ms, walk_ms, frac, _ = O.time_sampled(x, y, z, m, 1.0, eps, theta, ncrit, stride)
    step_ms = build_ms + walk_ms / max(frac, 1e-12)
    _, _, _, _, acc = O.time_sampled(x, y, z, m, 1.0, eps, theta, ncrit, max(stride, 16), with_acc=True)
    return {"value": n / (step_ms * 1e-3), "unit": "particle-steps/s", "cores": O.num_threads(),
            "kind": "port", "step_ms_extrapolated": step_ms, "theta": theta, "leaf_capacity": ncrit,
            "force_err": cpu_error(O, x, y, z, m, eps, acc),
            "sample": f"N={n}: full FP64 tree build ({build_ms:.0f} ms) + grouped walk over every "
                      f"{stride}-th leaf group ({100 * frac:.1f}% of particles, {walk_ms:.0f} ms), "
                      f"extrapolated to one full force evaluation"}


# The theta test's setting at the 1e-3 rms target on the galaxy (the GPU
# theta arm calibrates to it: theta 0.63 at leaf capacity 40); the CPU arm
# runs the reference's algorithm at that setting and states its own error.
REF_THETA, REF_LEAF = 0.63, 40


def run_reference(args, rank, world):
    """The reference's CPU path (the oracle port of Tree.cpp / Solvers.cpp,
    OpenMP on every host core) on this config.  Each timed step is a bounded
    sample of one KDK force evaluation: the full FP64 tree build plus the
    grouped walk over every k-th leaf group; the line's value extrapolates it
    to the whole walk ("extrapolated": true), ms_per_step is the sample's own
    wall time."""
    if rank != 0:
        return 0
    orc = ge.load_oracle()
    orc.build_oracle()
    ic = __import__(ge.PKG_NAME + ".ic", fromlist=["ic"]) if ge.load_package() else None
    arrs, eps, dt, _, _ = make_inputs(ic, args.workload)
    theta, ncrit = REF_THETA, REF_LEAF
    O = orc.Oracle()
    x, y, z, _, _, _, m = (a.astype(np.float64) for a in arrs)
    n = len(x)
    stride = max(1, int(n // 16384))
    sample_ms, full_ms, parts = [], [], []
    for k in range(args.warmup + args.steps):
        t0 = time.perf_counter()
        build_ms, walk_ms, frac, _ = O.time_sampled(x, y, z, m, 1.0, eps, theta, ncrit, stride)
        wall = 1e3 * (time.perf_counter() - t0)
        if k >= args.warmup:
            sample_ms.append(wall)
            full_ms.append(build_ms + walk_ms / max(frac, 1e-12))
            parts.append((build_ms, walk_ms, frac))
    step_ms = float(np.mean(full_ms))
    value = n / (step_ms * 1e-3)
    _, _, _, _, acc = O.time_sampled(x, y, z, m, 1.0, eps, theta, ncrit, stride, with_acc=True)
    err = cpu_error(O, x, y, z, m, eps, acc)
    b, w, f = (float(np.mean([p[i] for p in parts])) for i in range(3))
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "particle-steps/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": float(np.mean(sample_ms)),
            "higher_is_better": True, "scaling": "replicas", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "extrapolated": True,
            "config": {"workload": args.workload, "n": n, "theta": theta, "eps": eps, "leaf_capacity": ncrit,
                       "force_err_rms": err["rms"], "force_err_max": err["max"], "force_err_targets": err["targets"],
                       "sampled_fraction": f, "ms_build": b, "ms_walk_sampled": w,
                       "ms_per_step_extrapolated": step_ms,
                       "implementation": "oracle/ngrav_oracle.c, the C restatement of Tree.cpp + Solvers.cpp "
                                         "(the reference's own sources are not on this machine)"},
            "cpu_baseline": {"value": value, "unit": "particle-steps/s", "cores": O.num_threads(), "kind": "port",
                             "sample": f"each step: full FP64 tree build + grouped walk over every {stride}-th "
                                       f"leaf group ({100 * f:.2f}% of particles), extrapolated to one full KDK "
                                       f"force evaluation"},
            "e2e": {"value": value, "unit": "particle-steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


THETA_GRID = (0.5, 0.55, 0.575, 0.6, 0.605, 0.61, 0.615, 0.62, 0.625, 0.63, 0.635, 0.64, 0.645, 0.65, 0.6625,
              0.675, 0.7, 0.75, 0.8)
# budgets ~12 % apart from 2e-5 to 1e-3 (the cold collapse's calibration)
COLLAPSE_BUDGET_GRID = tuple(float("%.3g" % (2e-5 * 1.12 ** k)) for k in range(35))
BUDGET_GRID = (5e-5, 1e-4, 1.5e-4, 2e-4, 2.5e-4, 2.75e-4, 3e-4, 3.1e-4, 3.2e-4, 3.3e-4, 3.4e-4, 3.5e-4, 3.6e-4,
               3.7e-4, 3.8e-4, 3.9e-4, 4e-4, 4.5e-4, 5e-4, 7e-4, 1e-3)
TARGET_RMS = 1e-3
# The learned test's in-run safety check: every 10 steps an FP64-summed
# direct sum on this many sampled targets estimates the rms error (about +-3 %
# on the rms at 1,024 targets), reverting to the theta test above 1.5x the
# target.  The error reported on the line is measured separately, on 4,096.
CHECK_TARGETS = 1024


def error_at(sim, seed=2024):
    """One force evaluation of the current state and its rms / max relative
    error against the direct sum (FP32 pairs, FP64 sums) on 4,096 targets."""
    sim.compute_accel()
    return sim.force_error(nsample=4096, seed=seed, fp64_pairs=False)


def calibrate(sim, grid, setter, target=TARGET_RMS, stop=None):
    """Largest grid value whose rms error stays within the target (the grid
    ascends in error; with `stop`, the scan ends once the rms passes stop x
    the target)."""
    table, best = [], None
    for v in grid:
        setter(v)
        fe = error_at(sim)
        table.append([v, fe["rms"], fe["max"]])
        if fe["rms"] <= target:
            best = v
        elif stop and fe["rms"] > stop * target:
            break
    return (best if best is not None else grid[0]), table


def replica_max(v, dist, device):
    """The largest of a per-rank figure over the replicas (the slowest one sets
    the pace of the job); v itself with one process."""
    if dist is None:
        return v
    import torch
    t = torch.tensor([float(v)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_value(n, world, ms_max):
    """Whole-job particle-steps/s: every replica advances n particles per step."""
    return world * n / (ms_max * 1e-3)


def timed(sim, steps, warmup, dt, clocks=None, dist=None, diag=None):
    """W untimed steps, then exactly K steps between barriers (each
    ngrav_gpu_step call returns with its stream synchronised); the time is the
    device time of the K steps on the engine's stream.  diag: a callable run
    just before and just after the K steps (outside the timed region); its
    two results are returned too."""
    sim.step(warmup, dt)
    d0 = diag() if diag else None
    if dist is not None:
        dist.barrier()
    if clocks:
        clocks.start()
    sim.reset_cumulative()
    sim.step(steps, dt)
    st = sim.stats()
    clk = clocks.stop() if clocks else None
    if dist is not None:
        dist.barrier()
    d1 = diag() if diag else None
    if diag:
        return st, st["cum_ms_step"] / steps, clk, (d0, d1)
    return st, st["cum_ms_step"] / steps, clk


def drift(d0, d1, mtot):
    """Relative conservation errors between two FP64 diagnostics: energy
    (E1 - E0) / |E0|; momentum |P1 - P0| over the momentum scale
    sqrt(2 M K) (the net momentum is ~0 in the COM frame; K the larger of the
    two kinetic energies, so a cold start is measured against the motion it
    develops); angular momentum |L1 - L0| / |L0|, or, when the system starts
    without angular momentum (a cold collapse), over sqrt(2 M K) x one length
    unit (the ball's radius).  The absolute changes are given too."""
    dP = float(np.linalg.norm(np.subtract(d1["P"], d0["P"])))
    dL = float(np.linalg.norm(np.subtract(d1["L"], d0["L"])))
    L0 = float(np.linalg.norm(d0["L"]))
    pscale = float(np.sqrt(2.0 * mtot * max(d0["kinetic"], d1["kinetic"])))
    return {"energy_drift": (d1["energy"] - d0["energy"]) / abs(d0["energy"]),
            "momentum_drift": dP / pscale if pscale > 0 else None, "momentum_change": dP,
            "angular_momentum_drift": dL / L0 if L0 > 0 else (dL / pscale if pscale > 0 else None),
            "angular_momentum_change": dL,
            "angular_momentum_scale": "|L0|" if L0 > 0 else "sqrt(2 M K) x 1 length unit (L0 = 0)",
            "potential": "exact pair sum, FP32 pair terms, FP64 sums" if d0["potential_exact"] == 2 else
                         ("exact pair sum, FP64" if d0["potential_exact"] == 1 else "none")}


def hbm_peak():
    """Measured copy bandwidth of the GB300s (driver-written), else the fallback."""
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    except (OSError, KeyError, ValueError):
        return 6800.0, "fallback"


def fp32_peak_detail(dev, probe, clk):
    """The FP32 denominator beside the figures it should be near: the SM
    count, the SM clock (median under load in the timed region, and the
    maximum), and the theoretical FMA peak SMs x 128 lanes x 2 flops x
    clock."""
    import torch
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    mhz = (clk or {}).get("sm_mhz")
    mx = (clk or {}).get("sm_max_mhz")
    th = lambda f: sms * 128 * 2 * f * 1e6 / 1e12 if f else None  # noqa: E731
    return {"probe_tflops": probe, "sms": sms, "sm_mhz_under_load": mhz, "sm_max_mhz": mx,
            "theoretical_at_load_clock": th(mhz), "theoretical_at_max_clock": th(mx),
            "probe_frac_of_theoretical_max": probe / th(mx) if probe and mx else None}


# DRAM bytes per particle of one radix-sort scatter pass at N = 4,194,304:
# dram__bytes_read.sum + dram__bytes_write.sum of the six rs_scatter_kernel
# launches of one sort (329.9 MB), a cold-cache ncu capture
# (profiles/sort_scatter_galaxy4m.txt).  The keys and slots are L2-resident
# between passes, so the traffic is below the algorithmic bytes.
SORT_SCATTER_DRAM_BYTES_PER_PARTICLE_PASS = 13.1


def sort_roofline(st, n, split):
    """The HBM-bound part of the tree build: the LSD radix sort (the
    evaluation's passes of 9-bit digits, up to 7; each reads and writes 8 B
    keys + 4 B slots) and the permutation of the state into key order
    (split: pos, plo, vel, vlo, acc read and written, id moved, the
    permutation read), algorithmic bytes over the phase's event time."""
    passes = st.get("sort_passes", 7)
    per = passes * 24 + ((5 * 16 + 4 + 4) + (5 * 16 + 4) if split else (3 * 16 + 4 + 4) + (3 * 16 + 4))
    ms = st["ms_sort"]
    peak, src = hbm_peak()
    ach = per * n / (ms * 1e-3) / 1e9 if ms > 0 else None
    return {"bound": "hbm", "achieved": ach, "peak": peak, "unit": "GB/s", "frac": ach / peak if ach else None,
            "traffic": SORT_SCATTER_DRAM_BYTES_PER_PARTICLE_PASS * passes * n,
            "traffic_unit": "DRAM bytes of the phase's scatter passes (ncu bytes per particle-pass x passes x N)",
            "bytes_per_particle": per, "sort_passes": passes,
            "kernel": "radix sort (rs_hist, rs_scan, rs_scatter) + permute",
            "peak_source": src}


def p2p_phase_roofline(pkg, ic, dev, peak, prec, leaf_capacities=(32, 64, 128)):
    """The evaluation kernel's P2P phase on its own: a Plummer sphere of
    262,144 particles at theta = 0, where the walk opens every node, so every
    interaction is a near-field pair (no P2C term); 20 algorithmic flops per
    pair over the kernel's event time (best of three evaluations), against
    the measured FP32 peak.  The headline figure is at leaf capacity 32 (a
    mean of 9.6 targets per group); the same at larger groups shows how the
    staging cost per source spreads over more targets."""
    arrs = ic.plummer(262144, seed=5)
    rows = {}
    for L in leaf_capacities:
        best = None
        with pkg.NBodySystem(pkg.StepParams(G=1.0, eps=0.01, theta=0.0), leaf_capacity=L, precision=prec,
                             device=dev, timing=True) as s:
            s.set_particles_f32(*arrs)
            for _ in range(3):
                s.compute_accel()
                st = s.stats()
                if best is None or st["ms_force"] < best[0]:
                    best = (st["ms_force"], st["p2p_pairs"], st["p2c_terms"], st["leaves"])
        ms, pairs, terms, leaves = best
        ach = 20.0 * pairs / (ms * 1e-3) / 1e12 if ms > 0 else None
        rows[L] = {"achieved": ach, "frac": ach / peak if ach and peak else None, "ms": ms, "p2p_pairs": pairs,
                   "p2c_terms": terms, "mean_group": 262144 / max(1, leaves)}
    r = rows[leaf_capacities[0]]
    return {"bound": "fp32", "achieved": r["achieved"], "peak": peak, "unit": "TFLOP/s", "frac": r["frac"],
            "kernel": "eval_kernel, P2P only (20 flops/pair)",
            "workload": f"Plummer N=262144, theta 0 (all pairs near), leaf capacity {leaf_capacities[0]}",
            "p2p_pairs": r["p2p_pairs"], "p2c_terms": r["p2c_terms"], "ms": r["ms"],
            "by_leaf_capacity": {str(L): v for L, v in rows.items()}}


def phases(st):
    return {k: st[k] for k in ("ms_bbox_keys", "ms_sort", "ms_build", "ms_moments", "ms_walk", "ms_force")}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=30)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="galaxy4m", choices=sorted(WORKLOADS))
    ap.add_argument("--mac", default="learned", choices=["learned", "geometric"],
                    help="learned: train, calibrate both tests to the target rms, time both arms")
    ap.add_argument("--theta", type=float, default=None, help="geometric arm theta (default: calibrated)")
    ap.add_argument("--budget", type=float, default=None, help="learned arm budget (default: calibrated)")
    ap.add_argument("--lmac-pairs", type=int, default=1 << 22)
    ap.add_argument("--lmac-snapshots", type=int, default=16)
    ap.add_argument("--precision", default="split", choices=["split", "plain"])
    ap.add_argument("--leaf-grid", default="16,24,32,40,48,64",
                    help="leaf capacities tried per arm (comma list; one value fixes it)")
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-configs", action="store_true",
                    help="skip the compact records of the other BASELINE configs (C2, C3, C5)")
    args = ap.parse_args()
    rank, world, local = dist_env()
    if args.impl == "reference":
        return run_reference(args, rank, world)

    pkg = ge.load_package()
    ic = __import__(ge.PKG_NAME + ".ic", fromlist=["ic"])
    dev = local
    if WORKLOADS[args.workload][0] == "ensemble":
        return run_ensemble(args, pkg, ic, rank, world, dev)
    if args.workload == "plummer1m":
        if rank == 0:
            print(json.dumps({"metric": "C2 Plummer 1M: plain FP32 vs split precision + Kahan, 100 KDK steps",
                              "config": {"workload": "plummer1m", **precision_run(pkg, ic, dev, steps=100)}}),
                  flush=True)
        return 0
    if args.workload == "collapse16m":
        r = collapse_run(pkg, ic, dev, energy=True)
        if rank == 0:
            print(json.dumps({"metric": "C5 cold collapse 16.8M, learned test, 200 KDK steps", "value": r["value"],
                              "unit": "particle-steps/s", "ms_per_step": r["ms_per_step"],
                              "config": {"workload": "collapse16m", **r}}), flush=True)
        return 0
    arrs, eps, dt, theta0, ncrit = make_inputs(ic, args.workload)
    n = len(arrs[0])
    prec = pkg.PRECISION_SPLIT if args.precision == "split" else pkg.PRECISION_PLAIN
    sim = pkg.NBodySystem(pkg.StepParams(G=1.0, eps=eps, theta=theta0, dt=dt), leaf_capacity=ncrit, precision=prec,
                          device=dev, timing=True)
    sim.set_particles_f32(*arrs)
    sim.prime()
    learned = args.mac == "learned"

    # ---- setup (untimed): per leaf capacity (the target-group size), train
    # on the run itself and calibrate both tests to the error target; each arm
    # then runs at its own fastest leaf capacity ----
    leaf_grid = [int(v) for v in args.leaf_grid.split(",")] if args.leaf_grid else [ncrit]

    def restart(L):
        sim.set_opts(leaf_capacity=L, mac=pkg.MAC_GEOMETRIC)
        sim.set_particles_f32(*arrs)
        sim.prime()

    def eval_ms(reps=3):
        ms = 0.0
        for _ in range(reps):
            sim.compute_accel()
            ms += sum(phases(sim.stats()).values())
        return ms / reps

    def set_budget(v):
        sim.set_opts(mac=pkg.MAC_LEARNED)
        sim.lmac_set_opts(budget=v, check_every=0)

    tuning = []
    for L in leaf_grid:
        row = {"leaf_capacity": L}
        restart(L)
        if args.theta is None:
            row["theta"], row["cal_theta"] = calibrate(sim, THETA_GRID,
                                                       lambda v: sim.set_opts(theta=v, mac=pkg.MAC_GEOMETRIC))
        else:
            row["theta"] = args.theta
        sim.set_opts(theta=row["theta"], mac=pkg.MAC_GEOMETRIC)
        row["ms_eval_theta"] = eval_ms()
        if learned:
            t0 = time.perf_counter()
            row["train"] = sim.lmac_train(snapshots=args.lmac_snapshots, steps_between=1, dt=dt,
                                          pairs=args.lmac_pairs, epochs=8, batch=8192, seed=1)
            row["train"]["wall_s"] = time.perf_counter() - t0
            row["model"] = sim.lmac_get_model()
            restart(L)  # training stepped the system: start again from the inputs
            sim.set_opts(theta=row["theta"])
            if args.budget is None:
                row["budget"], row["cal_budget"] = calibrate(sim, BUDGET_GRID, set_budget)
            else:
                row["budget"] = args.budget
            set_budget(row["budget"])
            row["ms_eval_learned"] = eval_ms()
        tuning.append(row)
    best_t = min(tuning, key=lambda r: r["ms_eval_theta"])
    theta, cal_theta, ncrit_t = best_t["theta"], best_t.get("cal_theta"), best_t["leaf_capacity"]
    budget, cal_budget, train, ncrit_l = None, None, None, ncrit_t
    if learned:
        best_l = min(tuning, key=lambda r: r["ms_eval_learned"])
        budget, cal_budget, train = best_l["budget"], best_l.get("cal_budget"), best_l["train"]
        ncrit_l = best_l["leaf_capacity"]
    tuning_table = [{k: v for k, v in r.items() if k in ("leaf_capacity", "theta", "budget", "ms_eval_theta",
                                                         "ms_eval_learned")} for r in tuning]

    dist = None
    if world > 1:
        import torch
        import torch.distributed as tdist
        torch.cuda.set_device(dev)
        tdist.init_process_group("nccl")
        dist = tdist
        dist.barrier()
    clocks = ClockSampler(dev)

    def pick_walk_stack():
        """The arm's per-warp walk stack (2,048 entries at 6 CTAs per SM, or
        1,024 at 8): the faster evaluation of this state (under replicas, by
        the slowest rank's time for each size, so every rank runs the same
        size), installed."""
        ms = {}
        for ws in (2048, 1024):
            sim.set_tuning(0, ws)
            ms[ws] = replica_max(eval_ms(reps=5), dist, f"cuda:{dev}")
        best = min(ms, key=ms.get)
        sim.set_tuning(0, best)
        return best

    # ---- geometric (plain theta) arm ----
    restart(ncrit_t)
    sim.set_opts(theta=theta, mac=pkg.MAC_GEOMETRIC)
    ws_t = pick_walk_stack()
    mtot = float(np.sum(arrs[6], dtype=np.float64))
    diag2 = lambda: sim.diagnostics(exact_potential=2)  # noqa: E731
    st_g, ms_g, clk_g, dg = timed(sim, args.steps, args.warmup, dt, None if learned else clocks, dist, diag=diag2)
    ms_g = replica_max(ms_g, dist, f"cuda:{dev}")
    fe_g = error_at(sim)
    arm_theta = {"theta": theta, "leaf_capacity": ncrit_t, "walk_stack": ws_t, "value": job_value(n, world, ms_g),
                 "ms_per_step": ms_g,
                 "force_err_rms": fe_g["rms"], "force_err_max": fe_g["max"],
                 "p2p_pairs_per_step": st_g["cum_p2p_pairs"] / max(1, st_g["cum_evals"]),
                 "p2c_terms_per_step": st_g["cum_p2c_terms"] / max(1, st_g["cum_evals"]),
                 "ms_walk_per_step": st_g["cum_ms_walk"] / max(1, st_g["cum_evals"]),
                 "ms_force_per_step": st_g["cum_ms_force"] / max(1, st_g["cum_evals"]),
                 "ms_phases_last_eval": phases(st_g), "calibration": cal_theta, **drift(dg[0], dg[1], mtot)}

    # ---- learned arm (the method) ----
    ws_l = ws_t
    if learned:
        restart(ncrit_l)
        sim.lmac_set_model(*best_l["model"])
        sim.set_opts(theta=best_l["theta"], mac=pkg.MAC_LEARNED)
        sim.lmac_set_opts(budget=budget, check_every=10, check_targets=CHECK_TARGETS, revert_rms=TARGET_RMS * 1.5)
        ws_l = pick_walk_stack()
        sim.lmac_reset()
        st, ms_step, clk, dl = timed(sim, args.steps, args.warmup, dt, clocks, dist, diag=diag2)
        fe = error_at(sim)
    else:
        st, ms_step, clk, fe, dl = st_g, ms_g, clk_g, fe_g, dg
    ms_max = replica_max(ms_step, dist, f"cuda:{dev}")
    value = job_value(n, world, ms_max)

    # roofline of the evaluation kernel (P2P + P2C on the FP32 pipe)
    flops = 20.0 * st["cum_p2p_pairs"] + 60.0 * st["cum_p2c_terms"]
    force_s = st["cum_ms_force"] * 1e-3
    achieved = flops / force_s / 1e12 if force_s > 0 else None
    peak = pkg.probe_fp32_peak(dev)

    # e2e through the C-ABI with host buffers: each step writes the state from
    # pinned host memory (ngrav_gpu_set_state_f32), runs one KDK step and reads
    # positions and velocities back (ngrav_gpu_get_state), wall clock.
    import ctypes
    try:
        import torch
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()  # noqa: E731
        hin = [pin(a.astype(np.float32)) for a in sim.state()]
        hout = [torch.empty(n, dtype=torch.float64).pin_memory().numpy() for _ in range(6)]
    except Exception:
        hin = [np.ascontiguousarray(a, dtype=np.float32) for a in sim.state()]
        hout = [np.empty(n) for _ in range(6)]
    fin = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for a in hin]
    dout = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in hout]
    L = sim.L
    t_e2e, t_parts = [], []
    for k in range(1 + args.e2e_steps):
        t0 = time.perf_counter()
        rc = L.ngrav_gpu_set_state_f32(sim.h, *fin)
        t1 = time.perf_counter()
        rc |= L.ngrav_gpu_step(sim.h, 1, ctypes.c_double(dt))
        t2 = time.perf_counter()
        rc |= L.ngrav_gpu_get_state(sim.h, *dout)
        t3 = time.perf_counter()
        if rc:
            raise RuntimeError("e2e call failed: " + L.ngrav_gpu_last_error(sim.h).decode())
        if k > 0:
            t_e2e.append(t3 - t0)
            t_parts.append((t1 - t0, t2 - t1, t3 - t2))
        for a, b in zip(hin, hout):
            a[:] = b  # the next step starts from this step's result
    e2e_ms = 1e3 * float(np.mean(t_e2e))
    e2e_ms = replica_max(e2e_ms, dist, f"cuda:{dev}")
    parts = [1e3 * float(np.mean([p[i] for p in t_parts])) for i in range(3)]
    e2e = {"value": job_value(n, world, e2e_ms), "unit": "particle-steps/s", "h2d_bytes_per_step": 6 * 4 * n,
           "d2h_bytes_per_step": 6 * 8 * n, "ms_per_step": e2e_ms, "steps": args.e2e_steps,
           "ms_per_step_median": 1e3 * float(np.median(t_e2e)), "ms_per_step_max": 1e3 * float(np.max(t_e2e)),
           "ms_set_state": parts[0], "ms_step": parts[1], "ms_get_state": parts[2],
           "h2d_gbs": 6 * 4 * n / (parts[0] * 1e-3) / 1e9, "d2h_gbs": 6 * 8 * n / (parts[2] * 1e-3) / 1e9,
           "call": "ngrav_gpu_set_state_f32 + ngrav_gpu_step(1) + ngrav_gpu_get_state (pinned host buffers)"}

    cpu = None
    if rank == 0 and not args.no_cpu_baseline:
        try:
            cpu = cpu_baseline(ge.load_oracle(), arrs, eps, theta, ncrit_t)
        except Exception as exc:  # the baseline must not sink the GPU line
            cpu = {"error": str(exc)}

    if rank == 0:
        cfg = {"workload": args.workload, "n": n, "mac": args.mac, "eps": eps, "dt": dt,
               "leaf_capacity": ncrit_l if learned else ncrit_t, "leaf_capacity_tuning": tuning_table,
               "walk_stack": ws_l if learned else ws_t,
               "precision": args.precision, "quadrupole": True, "target_rms": TARGET_RMS,
               "parallelism": "replicas" if world > 1 else "single-gpu",
               "l2": "per-step working set > 0.5 GB, larger than the 129 MB L2",
               "force_err_rms": fe["rms"], "force_err_max": fe["max"], "force_err_median": fe["median"],
               "force_err_targets": fe["nsample"],
               "interactions_per_s": (st["cum_p2p_pairs"] + st["cum_p2c_terms"]) / (st["cum_ms_step"] * 1e-3),
               "p2p_pairs_per_step": st["cum_p2p_pairs"] / max(1, st["cum_evals"]),
               "p2c_terms_per_step": st["cum_p2c_terms"] / max(1, st["cum_evals"]),
               "ms_walk_per_step": st["cum_ms_walk"] / max(1, st["cum_evals"]),
               "ms_force_per_step": st["cum_ms_force"] / max(1, st["cum_evals"]),
               "ms_eval_per_step": st["cum_ms_eval"] / max(1, st["cum_evals"]),
               "list_entries_per_step": st["far_entries"] + st["near_entries"],
               "mac_tests_per_step": st["mac_tests"], "walk_stack_max": st["walk_stack_max"],
               "leaves": st["leaves"], "nodes": st["nodes"], "ms_phases_last_eval": phases(st),
               "graph_replays": st["graph_replays"], "theta_arm": arm_theta, **drift(dl[0], dl[1], mtot),
               "drift_over": f"the {args.steps} timed steps"}
        if learned:
            cfg["learned"] = {"budget": budget, "calibration": cal_budget, "train": train,
                              "queries_last_eval": st["lmac_queries"], "accepts_last_eval": st["lmac_accepts"],
                              "fallbacks_last_eval": st["lmac_fallbacks"], "screened_last_eval": st["lmac_screened"],
                              "tensor_flushes_last_eval": st["lmac_flushes"],
                              "mlp_flops_last_eval": 2624.0 * st["lmac_queries"],
                              "checks": st["lmac_checks"], "last_check_rms": st["lmac_last_check_rms"],
                              "check_every": 10, "check_targets": CHECK_TARGETS,
                              "reverted": bool(st["lmac_reverted"])}
            cfg["speedup_vs_theta_arm"] = value / arm_theta["value"]
        line = {
            "metric": METRIC, "value": value, "unit": "particle-steps/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_max, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded galaxy generator)" if args.workload.startswith("galaxy") else "synthetic",
            "config": cfg,
            "roofline": {"bound": "fp32", "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                         "frac": (achieved / peak) if achieved and peak else None,
                         "traffic": EVAL_DRAM_BYTES_PER_LIST_ENTRY * (st["far_entries"] + st["near_entries"]),
                         "traffic_unit": "DRAM bytes per eval_kernel launch (ncu bytes/entry x entries)",
                         "kernel": "eval_kernel (P2P 20 flops/pair + P2C 60 flops/term)",
                         "peak_source": "measured FP32 FMA probe (ngrav_gpu_probe_fp32_peak)",
                         "peak_detail": fp32_peak_detail(dev, peak, clk)},
            "roofline_sort": sort_roofline(st, n, args.precision == "split"),
            "roofline_p2p": p2p_phase_roofline(pkg, ic, dev, peak, prec),
            "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": st["cum_launches"], "clocks": clk,
        }
    sim.close()
    if rank == 0 and world == 1 and not args.no_configs:
        # compact records of the other configs of the task (untimed by the
        # headline): C2 plain vs split precision, C3 ensemble, C5 cold collapse
        extra = {}
        for name, fn in (("C2_plummer1m_precision", lambda: precision_run(pkg, ic, dev, steps=100)),
                         ("C3_ensemble512", lambda: ensemble_run(pkg, ic, dev, steps=10, warmup=3, tune_reps=1)),
                         ("C5_collapse16m", lambda: collapse_run(pkg, ic, dev))):
            t0 = time.perf_counter()
            try:
                extra[name] = fn()
            except Exception as exc:  # a side record must not sink the headline line
                extra[name] = {"error": str(exc)}
            extra[name]["wall_s"] = time.perf_counter() - t0
        line["configs"] = extra
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
