#!/usr/bin/env python
"""Benchmark of the ePlace global-placement iteration on one GB300.

Workload: the 2M-cell synthetic netlist (2M movable cells with log-normal
widths, 20k fixed macros, 2.1M nets / 9.4M pins with 80% index locality,
1024x1024 bins, target density 0.8, seed 1).  One step is one trial step of
the Nesterov loop (density scatter + position update, density/overflow, WA
gradient, field solve, field gather + step control); `value` is accepted
Nesterov iterations per second of device time with everything resident in
HBM.  `e2e` is the same metric through the host-buffer C ABI call
(ap_step_host: positions in from pinned host memory, positions + readout out
every step).  The time to 10% overflow of the mixed-precision and plain
forms is measured on fresh instances after the timed region, and of the
mixed+surrogate form: a learned density-to-field surrogate trained here on the
GPU (pairs from other seeded netlists of the same shape) stands in for the
exact solve while the overflow exceeds 0.3, judged by the exact solve every 8
trials (reported with the net and, as the ablation, with its coarse spectral
layer alone).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

--impl reference times the CPU restatement of the reference path (oracle/,
FP64, OpenMP, field solve by fast transforms) on this host's cores: the
reference ships no GPU code and its own CPU loop (host C++ behind XRT) does
not build outside the VCK5000 flow.  That process loads only oracle/
libraries (the netlist comes from oracle/libsynth.so).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)
sys.path.insert(0, os.path.join(HERE, "oracle"))

METRIC = "Nesterov iters/s & time-to-10% overflow, 2M cells: mixed+surrogate vs plain"
UNIT = "iters/s"
# resident blocks of one launch over all nets (k_wirelength.cu): up to so many, the
# wirelength gradient is one launch, beyond four
WA_ONE_LAUNCH_BLOCKS = 456


def tensor_cores(solver: str) -> bool:
    """Whether the field solve runs on the tensor cores (AP_TC_VARIANT pins a
    candidate of the mixed-precision solver) and not as FP32 fast transforms."""
    return solver == "bf16x3" and bool(os.environ.get("AP_TC_VARIANT"))


def wa_launches(nl) -> int:
    d = np.diff(nl["net_ptr"])
    d = d[d >= 2]
    blocks = 0
    for lo, hi, lanes, most in ((2, 2, 1, 2432), (3, 4, 1, 2432), (5, 8, 1, 2432), (9, 16, 8, 608), (17, 32, 16, 608),
                                (33, 64, 16, 608), (65, 1 << 30, 32, 608)):
        items = int(((d >= lo) & (d <= hi)).sum()) * lanes
        blocks += min(max(1, (items + 255) // 256), most)
    return 1 if blocks <= WA_ONE_LAUNCH_BLOCKS else 4


def trial_launches(nl, info: dict, solver: str) -> int:
    """Kernels of one loop trial: position update, bin adds, wirelength gradient,
    field solve, gather.  The solve is three FP32 passes, the first with the density
    (32 bins: one launch); where AP_TC_VARIANT pins a tensor-core candidate it is
    the density and four stage launches, or one of the persistent candidates (3, 4)."""
    if tensor_cores(solver):
        field = 1 + (1 if info.get("tc_variant", -1) in (3, 4) else 4)
    else:
        field = 1 if int(nl["bins"]) == 32 else 3
    return 1 + 1 + wa_launches(nl) + field + 1


STAGES = ["scatter+update", "density+overflow", "wirelength", "field", "gather+control"]


def workload_desc(nl, preset):
    n_nodes = len(nl["node_w"])
    n_mov = int((nl["node_fixed"] == 0).sum())
    return {
        "workload": f"{preset}: {n_mov} movable cells, {n_nodes - n_mov} fixed macros, "
                    f"{len(nl['net_ptr']) - 1} nets / {len(nl['pin_node'])} pins (80% pins within a "
                    f"64-node window), {nl['bins']}x{nl['bins']} bins, target density {nl['target_density']}, "
                    f"seed {nl['seed']}",
        "bins": int(nl["bins"]),
        "cells": n_mov,
        "nets": len(nl["net_ptr"]) - 1,
        "pins": len(nl["pin_node"]),
        "l2": "inputs larger than L2 (per-step working set > 0.5 GB)",
    }


def stage_model(nl, solver):
    """Algorithmic bytes (HBM) or FLOPs per launch of each stage that the loop has."""
    n_nodes = len(nl["node_w"])
    n_mov = int((nl["node_fixed"] == 0).sum())
    e = len(nl["net_ptr"]) - 1
    p = len(nl["pin_node"])
    m2 = int(nl["bins"]) ** 2
    m3 = int(nl["bins"]) ** 3
    model = {
        # update: read v, g, u, w, h, write u', v' and the 20-byte bin record;
        # bin adds: read the record; int64 map written once
        "scatter+update": ("hbm", 88 * n_mov + 8 * m2),
        # read mov, fixed, fixed-scaled maps; clear mov; write solver input
        "density+overflow": ("hbm", 36 * m2),
        # net_ptr, pin_node, node positions, int64 gradient per movable node
        "wirelength": ("hbm", 4 * (e + 1) + 4 * p + 8 * n_nodes + 16 * n_mov),
        # mov, fixed, fixed-scaled maps in, mov cleared, both fields out; pinned to the
        # tensor cores: 6 dense m x m x m contractions (useful FLOPs)
        "field": ("tensor", 12 * m3) if tensor_cores(solver) else ("hbm", 40 * m2),
        # bin record, int64 WA gradient read+clear, pins, charge, g_prev, g out; field maps
        "gather+control": ("hbm", 60 * n_mov + 8 * m2),
    }
    if not tensor_cores(solver):  # the density is part of the field solve's first pass
        del model["density+overflow"]
    return model


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the measured region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = os.path.join("/tmp", f"ap_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=self.out, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.close()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [t.strip() for t in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "samples": len(sm),
                "reasons": sorted(reasons)}


def read_traffic(stage: str, preset: str):
    """Per-launch DRAM bytes of a stage from the committed ncu summary, if any."""
    path = os.path.join(HERE, "profiles", "traffic.md")
    if not os.path.exists(path):
        return None
    key = f"{preset} {stage}:"
    for line in open(path):
        if line.strip().startswith(key):
            try:
                return float(line.split(":", 1)[1].split()[0])
            except (ValueError, IndexError):
                return None
    return None


def cpu_baseline(nl, budget_s: float = 20.0):
    import numpy as np  # noqa: F401

    import oracle

    oracle.build(with_ref=False)
    cores = oracle.set_threads(os.cpu_count() or 1)
    pl = oracle.Placer(nl, int(nl["bins"]), float(nl["target_density"]))
    pl.init(nl["node_x"], nl["node_y"])
    t0 = time.perf_counter()
    n = 0
    while True:
        pl.step(1)
        n += 1
        el = time.perf_counter() - t0
        if el > budget_s or el / n * (n + 1) > budget_s * 1.5:
            break
    return {"value": n / el, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"FP64 oracle loop on the full workload: init (2 evaluations, untimed) + {n} "
                      f"iteration(s) in {el:.1f} s on {cores} threads; field solve by fast transforms "
                      f"(O(M^2 log M))"}


def load_presets():
    """The workload presets (aieplace_gb300/presets.py, data only), read
    without importing the product package."""
    import importlib.util

    spec = importlib.util.spec_from_file_location("ap_presets", os.path.join(HERE, "aieplace_gb300", "presets.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod.PRESETS


def reference_arm(args):
    """The reference path's CPU implementation on this host's cores: the FP64
    oracle loop (oracle/, OpenMP; its field solve by fast transforms like the
    reference's Ooura/RePlAce solver).  The netlist comes from the standalone
    generator library (oracle/libsynth.so): this process loads no library of
    the GPU product."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import oracle

    oracle.build(with_ref=False)
    nl = oracle.synth_generate(load_presets()[args.preset], seed=1)
    cores = oracle.set_threads(os.cpu_count() or 1)
    pl = oracle.Placer(nl, int(nl["bins"]), float(nl["target_density"]))
    pl.init(nl["node_x"], nl["node_y"])
    budget = float(os.environ.get("AP_REFERENCE_BUDGET_S", "150"))
    t0 = time.perf_counter()
    done = 0
    for _ in range(args.warmup):
        pl.step(1)
        if time.perf_counter() - t0 > budget / 4:
            break
    t0 = time.perf_counter()
    for k in range(args.steps):
        pl.step(1)
        done += 1
        el = time.perf_counter() - t0
        if el / done * (done + 1) > budget:
            break
    el = time.perf_counter() - t0
    v = done / el
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
        "steps": done, "warmup": args.warmup, "ms_per_step": 1000 * el / done, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": workload_desc(nl, args.preset),
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{done} of {args.steps} requested FP64 iterations of the full workload "
                                   f"(bounded to ~{budget:.0f} s); field solve by fast transforms "
                                   f"(O(M^2 log M))"},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def profile_mode(args):
    """A capture target for ncu: the workload after `profile_after` iterations."""
    import torch

    import aieplace_gb300 as ap
    from aieplace_gb300 import build as b

    b.build()
    nl = ap.synth.generate(args.preset, seed=1)
    solver = "fp32" if args.solver == "fp32" else "bf16x3"
    with ap.Placer(nl, field_solver=solver) as pl:
        pl.initialize_placement(seed=11, sigma=1.0)
        if args.profile_after:
            pl.perform_iteration(args.profile_after)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_push("ap_profile")
        ms = pl.profile_stages(1)
        torch.cuda.nvtx.range_pop()
        torch.cuda.synchronize()
        s = pl.stats()
    print(json.dumps({"profile_after": args.profile_after, "stage_ms": dict(zip(STAGES, ms)),
                      "overflow": s["overflow"], "iteration": s["iteration"]}))


def batch_mode(args):
    """Batched form: n instances (cell counts LogUniform[5k, 150k], bins 128..512)
    stepped together.  Reports instance-iterations per second over K graph
    launches for the persistent form (six persistent launches per trial step
    over all instances, FP32 field, the default), for the graph of
    per-instance branches with the FP32 field and, where AP_TC_VARIANT pins a
    candidate, with the BF16x3 tensor-core field, the wall time until every instance is below 10% overflow, and the
    instances stepped one after another on their own graphs."""
    import torch

    import aieplace_gb300 as ap
    from aieplace_gb300 import build as b

    b.build()
    specs = ap.synth.batch_specs(args.batch, seed=1)
    nls = [ap.synth.generate(s, seed=100 + i) for i, s in enumerate(specs)]
    cells = sum(int((nl["node_fixed"] == 0).sum()) for nl in nls)
    forms = {}
    for form in ("persistent", "graph") + (("graph_bf16x3",) if tensor_cores("bf16x3") else ()):
        solver = "bf16x3" if form == "graph_bf16x3" else "fp32"
        with ap.BatchPlacer(nls, field_solver=solver, max_iterations=4000, check_interval=32) as bp:
            bp.set_form("graph" if form == "graph_bf16x3" else form)
            bp.initialize_placement(seed=5, sigma=1.0)
            bp.step(args.warmup)
            it0 = sum(bp.stats(i)["iteration"] for i in range(bp.n))
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            bp.step(args.steps)
            el = time.perf_counter() - t0
            it1 = sum(bp.stats(i)["iteration"] for i in range(bp.n))
            info = bp.info()
            stage_ms = bp.profile(10) if form == "persistent" else None
            one_block = None
            if form == "persistent":
                # the same launches with one block per work item
                bp.set_item_blocks(1)
                bp.step(args.warmup)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                bp.step(args.steps)
                one_block = {"graph_launch_ms": 1000 * (time.perf_counter() - t0) / args.steps,
                             "stage_ms": bp.profile(10), "info": bp.info()}
        with ap.BatchPlacer(nls, field_solver=solver, max_iterations=4000, check_interval=32) as bp:
            bp.set_form("graph" if form == "graph_bf16x3" else form)
            bp.initialize_placement(seed=5, sigma=1.0)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            its = bp.run()
            ttt = time.perf_counter() - t0
            st = [bp.stats(i) for i in range(bp.n)]
        over = [s["overflow"] for s in st]
        missed = [{"instance": i, "cells": specs[i]["num_cells"], "bins": specs[i]["bins"],
                   "iteration": s["iteration"], "overflow": s["overflow"], "lambda": s["lambda"],
                   "status": s["status"]} for i, s in enumerate(st) if not s["overflow"] < 0.10]
        forms[form] = {"instance_iters_per_s": (it1 - it0) / el, "graph_launch_ms": 1000 * el / args.steps,
                       "time_to_10pct_all_s": ttt, "iterations": its, "reached": sum(o < 0.10 for o in over),
                       "not_reached": missed, "info": info}
        if stage_ms:
            forms[form]["stage_ms"] = stage_ms
            forms[form]["one_block_per_item"] = one_block
    # the same instances one after another, each on its own graph
    t0 = time.perf_counter()
    seq_its = 0
    for i, nl in enumerate(nls[: min(8, len(nls))]):
        with ap.Placer(nl) as pl:
            pl.initialize_placement(seed=5 + i, sigma=1.0)
            pl.step_async(args.steps)
            torch.cuda.synchronize()
            seq_its += pl.stats()["iteration"]
    seq_el = time.perf_counter() - t0
    print(json.dumps({
        "metric": "batched instance-iterations/s", "value": max(f["instance_iters_per_s"] for f in forms.values()),
        "best_form": max(forms, key=lambda k: forms[k]["instance_iters_per_s"]),
        "unit": "instance-iters/s", "instances": len(nls), "cells_total": cells, "steps": args.steps,
        "warmup": args.warmup, "forms": forms,
        "sequential_instance_iters_per_s_first8": seq_its / seq_el,
        "bins": [s["bins"] for s in specs], "dtype": "f32", "data": "synthetic"}))


TTT_SEEDS = (11, 12, 13)


def time_to_target(ap, nl, solver, target=0.10, max_iter=4000, surrogate=None, use_net=True):
    """Time to overflow < target from three seeded initial placements (the
    loop is chaotic: its iteration count varies by a few percent with the
    start); the run of median time, with every run's seconds and iterations."""
    runs = [time_to_target_once(ap, nl, solver, target, max_iter, surrogate, use_net, seed) for seed in TTT_SEEDS]
    med = sorted(runs, key=lambda r: r["seconds"])[len(runs) // 2]
    return {**med, "seconds_all": [r["seconds"] for r in runs], "iterations_all": [r["iterations"] for r in runs],
            "init_seeds": list(TTT_SEEDS)}


def time_to_target_once(ap, nl, solver, target, max_iter, surrogate, use_net, seed):
    import torch

    with ap.Placer(nl, field_solver=solver, target_overflow=target, max_iterations=max_iter,
                   check_interval=32) as pl:
        pl.initialize_placement(seed=seed, sigma=1.0)
        if surrogate is not None:
            pl.attach_surrogate(surrogate, overflow_min=0.3, judge_every=8, max_error=0.02, use_net=use_net)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        it = pl.run()
        torch.cuda.synchronize()
        el = time.perf_counter() - t0
        s = pl.stats()
        out = {"solver": solver, "init_seed": seed, "seconds": el, "iterations": it, "evals": s["evals"],
               "overflow": s["overflow"], "hpwl": s["hpwl"], "reached": s["overflow"] < target}
        if surrogate is not None:
            out["surrogate"] = {**pl.surrogate_stats(), "use_net": bool(use_net)}
    return out


def c4_block(ap):
    """The learned surrogate's own workload: 200k cells, 512^2 bins, the
    surrogate on the 256^2-pooled density (factor 2), trained here to the
    full budget (20k pairs from 10 seeded runs, SURROGATE_BUDGET); time to 10%
    overflow of the plain, mixed and mixed + surrogate forms."""
    nl = ap.synth.generate("c1", seed=1)
    out = {"workload": "c1: 200000 movable cells, 4000 fixed macros, 210000 nets, 512x512 bins, target "
                       "density 0.7, seed 1; surrogate factor 2 (256x256 coarse grid)",
           "plain": time_to_target(ap, nl, "fp32"), "mixed": time_to_target(ap, nl, "bf16x3")}
    surr, info = train_surrogate(ap, "c1", "bf16x3")
    out["surrogate_training"] = info
    out["mixed_surrogate"] = time_to_target(ap, nl, "bf16x3", surrogate=surr, use_net=True)
    out["mixed_surrogate_coarse_only"] = time_to_target(ap, nl, "bf16x3", surrogate=surr, use_net=False)
    surr.close()
    for k in ("mixed", "mixed_surrogate", "mixed_surrogate_coarse_only"):
        out[k]["speedup_vs_plain"] = out["plain"]["seconds"] / out[k]["seconds"]
    return out


# Training budgets of the learned surrogate: pairs from `runs` seeded exact
# loops (every `every`-th of their first `runs_trials` trials), Adam steps, and
# held-out pairs from another netlist.  The 200k-cell workload (coarse factor
# 2, 3.7 MB a pair) takes the full 20k-pair budget; the 2M-cell workload
# (factor 4, 13 MB a pair) 4000 pairs, which fit beside it in HBM.
SURROGATE_BUDGET = {"c1": dict(runs=10, runs_trials=2000, every=1, steps=20000, held=400, held_every=5),
                    "c2": dict(runs=8, runs_trials=1000, every=2, steps=10000, held=100, held_every=20)}


def train_surrogate(ap, preset: str, solver: str):
    """The learned surrogate of the mixed+surrogate form, trained here on the GPU
    by the library's own kernels on (density, field) pairs the exact solve
    produces in seeded loops on other netlists of the same shape
    (SURROGATE_BUDGET), Adam on 8 random 64 x 64 crops a step; then held-out
    pairs from another netlist, their errors also split by the overflow at
    which they were taken (the surrogate stands in above 0.3).  The coarse
    grid is 256^2 (factor bins / 256)."""
    import numpy as np
    import torch

    bud = SURROGATE_BUDGET[preset]
    f = max(1, int(ap.synth.PRESETS[preset]["bins"]) // 256)
    per_run = bud["runs_trials"] // bud["every"]
    n_train = bud["runs"] * per_run
    t0 = time.perf_counter()
    s = ap.Surrogate(factor=f, kernels=(3, 1, 1, 1))
    s.reserve(n_train + bud["held"], 256)
    for k in range(bud["runs"]):
        nl = ap.synth.generate(preset, seed=100 + k)
        with ap.Placer(nl, field_solver=solver) as pl:
            pl.initialize_placement(seed=200 + k, sigma=1.0)
            s.collect(pl, bud["runs_trials"], bud["every"])
    held_tau = []
    nl = ap.synth.generate(preset, seed=150)
    with ap.Placer(nl, field_solver=solver) as pl:
        pl.initialize_placement(seed=250, sigma=1.0)
        for _ in range(bud["held"] // 10):
            tau0 = pl.stats()["overflow"]
            s.collect(pl, 10 * bud["held_every"], bud["held_every"])
            held_tau += [0.5 * (tau0 + pl.stats()["overflow"])] * 10
    torch.cuda.synchronize()
    t1 = time.perf_counter()
    losses = s.train(steps=bud["steps"], batch=8, crop=64, lr=2e-3, seed=1, first=0, count=n_train)
    torch.cuda.synchronize()
    t2 = time.perf_counter()
    en, ec = s.validate(n_train, bud["held"])
    hi = np.array(held_tau) > 0.3

    def stat(v):
        return {"mean": float(v.mean()), "p50": float(np.median(v))} if v.size else None

    info = {"factor": f, "kernels": [3, 1, 1, 1], "width": 32, "params": s.num_params, "train_pairs": n_train,
            "runs": bud["runs"], "train_steps": bud["steps"], "heldout_pairs": bud["held"],
            "collect_s": t1 - t0, "train_s": t2 - t1, "loss_first100": float(losses[:100].mean()),
            "loss_last500": float(losses[-500:].mean()),
            "heldout_field_err_net": stat(en), "heldout_field_err_coarse": stat(ec),
            "heldout_pairs_overflow_above_0.3": int(hi.sum()),
            "heldout_field_err_net_overflow_above_0.3": stat(en[hi]),
            "heldout_field_err_coarse_overflow_above_0.3": stat(ec[hi])}
    return s, info


def surrogate_study(args):
    """The learned surrogate at its own workload (200k cells, 512^2 bins,
    256^2 coarse grid) trained to the full budget (20k pairs from 10 seeded
    runs): held-out errors and the time to 10% overflow of the mixed form with
    the trained net, with its coarse spectral layer alone and without a
    surrogate (three seeded starts each)."""
    import aieplace_gb300 as ap
    from aieplace_gb300 import build as b

    b.build()
    print(json.dumps({"study": "learned surrogate, 200k cells / 512^2 bins / 256^2 coarse grid",
                      **c4_block(ap)}), flush=True)


def main():
    ap_ = argparse.ArgumentParser()
    ap_.add_argument("--gpus", type=int, default=1)
    ap_.add_argument("--steps", type=int, default=200)
    ap_.add_argument("--warmup", type=int, default=20)
    ap_.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap_.add_argument("--preset", default="c2")
    ap_.add_argument("--solver", default="auto", choices=["auto", "fp32", "bf16x3"])
    ap_.add_argument("--no-cpu-baseline", action="store_true")
    ap_.add_argument("--no-ttt", action="store_true", help="skip the time-to-10%% runs")
    ap_.add_argument("--no-c4", action="store_true",
                     help="skip the surrogate's own workload (200k cells, 512^2 bins, 256^2 coarse grid)")
    ap_.add_argument("--surrogate-study", action="store_true",
                     help="train the surrogate on 20k pairs from 10 runs of the 200k-cell workload and report "
                          "held-out errors and time to 10%% overflow")
    ap_.add_argument("--batch", type=int, default=0,
                     help="batched form instead: this many instances (5k-150k cells) in one graph")
    ap_.add_argument("--profile-after", type=int, default=-1,
                     help="profiling mode: run this many iterations, then one eager trial step inside the "
                          "NVTX range 'ap_profile' (for ncu --nvtx-include ap_profile/), print nothing else")
    args = ap_.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.impl == "reference":
        return reference_arm(args)
    if args.profile_after >= 0:
        return profile_mode(args)
    if args.surrogate_study:
        return surrogate_study(args)
    if args.batch:
        return batch_mode(args)

    import numpy as np
    import torch

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    import aieplace_gb300 as ap
    from aieplace_gb300 import build as b

    if rank == 0:
        b.build()
    if world > 1:
        dist.barrier()
    solver = args.solver
    if solver == "auto":
        solver = "bf16x3" if os.environ.get("AP_BENCH_SOLVER", "bf16x3") == "bf16x3" else "fp32"
    # replicas: every rank places its own seeded instance (no data-path exchange)
    nl = ap.synth.generate(args.preset, seed=1 + rank)
    stream = torch.cuda.Stream()
    pl = ap.Placer(nl, field_solver=solver)
    try:
        pl.set_stream(stream.cuda_stream)
        pl.initialize_placement(seed=11 + rank, sigma=1.0)
    except ap.APError:
        if args.solver != "auto" or solver == "fp32":
            raise
        pl.close()
        solver = "fp32"
        pl = ap.Placer(nl, field_solver=solver)
        pl.set_stream(stream.cuda_stream)
        pl.initialize_placement(seed=11 + rank, sigma=1.0)
    clocks = ClockSampler(local)
    clocks.start()
    pl.step_async(args.warmup)
    torch.cuda.synchronize()
    s0 = pl.stats()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    ev0.record(stream)
    torch.cuda.nvtx.range_push("ap_timed")  # launch lists: ncu --nvtx --nvtx-include ap_timed/
    pl.step_async(args.steps)
    torch.cuda.nvtx.range_pop()
    ev1.record(stream)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    ms = ev0.elapsed_time(ev1)
    s1 = pl.stats()
    clk = clocks.stop()
    iters = s1["iteration"] - s0["iteration"]
    evals = s1["evals"] - s0["evals"]
    # roofline of the dominant stage (eager launches, events between stages)
    stage_ms = pl.profile_stages(10)
    # e2e through the host-buffer call: pinned in/out every step
    n = pl.num_nodes
    hx = torch.empty(n, dtype=torch.float32, pin_memory=True)
    hy = torch.empty(n, dtype=torch.float32, pin_memory=True)
    ox = torch.empty(n, dtype=torch.float32, pin_memory=True)
    oy = torch.empty(n, dtype=torch.float32, pin_memory=True)
    x, y = pl.positions()
    hx.copy_(torch.from_numpy(x))
    hy.copy_(torch.from_numpy(y))
    e2e_steps = max(10, min(args.steps, 100))
    torch.cuda.synchronize()
    se0 = pl.stats()
    t0 = time.perf_counter()
    from aieplace_gb300._lib import Stats, check, lib
    import ctypes as C

    st = Stats()
    for _ in range(e2e_steps):
        check("ap_step_host", lib().ap_step_host(pl._h, C.c_void_p(hx.data_ptr()), C.c_void_p(hy.data_ptr()),
                                                 C.c_void_p(ox.data_ptr()), C.c_void_p(oy.data_ptr()),
                                                 C.byref(st)))
        hx, ox = ox, hx
        hy, oy = oy, hy
    e2e_s = time.perf_counter() - t0
    se1 = pl.stats()
    e2e_iters = se1["iteration"] - se0["iteration"]
    n_mov = int((nl["node_fixed"] == 0).sum())
    launches_per_trial = trial_launches(nl, pl.solver_info() if tensor_cores(solver) else {}, solver)
    pl.close()

    t_max = ms / 1000.0
    total_iters = iters
    if world > 1:
        t = torch.tensor([t_max, float(iters), e2e_s, float(e2e_iters)], device="cuda")
        tmax = t.clone()
        dist.all_reduce(tmax, op=dist.ReduceOp.MAX)
        dist.all_reduce(t, op=dist.ReduceOp.SUM)
        t_max, total_iters = float(tmax[0]), int(t[1])
        e2e_s, e2e_iters = float(tmax[2]), int(t[3])

    ttt = None
    cpu = None
    if rank == 0:
        model = stage_model(nl, solver)
        dom = max(range(len(stage_ms)), key=lambda i: stage_ms[i])
        bound, amount = model[STAGES[dom]]
        peaks = {}
        pk_path = os.path.join(HERE, "MEASURED_PEAKS.json")
        if os.path.exists(pk_path):
            peaks = json.load(open(pk_path))
        if bound == "hbm":
            achieved = amount / (stage_ms[dom] / 1000.0) / 1e9
            peak = float(peaks.get("hbm_gbs", 6800.0))
            unit = "GB/s"
        else:
            achieved = amount / (stage_ms[dom] / 1000.0) / 1e12
            peak = float(peaks.get("bf16_tflops", 1900.0))
            unit = "TFLOP/s"
        # every stage against its own roof (HBM copy or dense BF16 burst)
        per_stage = []
        for i, name in enumerate(STAGES):
            if name not in model:
                continue
            b_i, amt_i = model[name]
            sec = stage_ms[i] / 1000.0
            if b_i == "hbm":
                ach_i, pk_i, u_i = amt_i / sec / 1e9, float(peaks.get("hbm_gbs", 6800.0)), "GB/s"
            else:
                ach_i, pk_i, u_i = amt_i / sec / 1e12, float(peaks.get("bf16_tflops", 1900.0)), "TFLOP/s"
            per_stage.append({"stage": name, "bound": b_i, "algorithmic": amt_i, "us": stage_ms[i] * 1000.0,
                              "achieved": ach_i, "unit": u_i, "frac": ach_i / pk_i,
                              "traffic": read_traffic(name, args.preset)})
        roof = {"kernel": STAGES[dom], "bound": bound, "achieved": achieved, "peak": peak, "unit": unit,
                "frac": achieved / peak, "traffic": read_traffic(STAGES[dom], args.preset),
                "peak_source": "measured" if peaks else "fallback",
                "stage_ms": dict(zip(STAGES, stage_ms)), "stages": per_stage}
        if not args.no_ttt:
            ttt = {"mixed": time_to_target(ap, nl, "bf16x3") if solver == "bf16x3" else None,
                   "plain": time_to_target(ap, nl, "fp32")}
            if solver == "bf16x3" and int(nl["bins"]) % 256 == 0:
                surr, sinfo = train_surrogate(ap, args.preset, solver)
                ttt["surrogate_training"] = sinfo
                ttt["mixed_surrogate"] = time_to_target(ap, nl, "bf16x3", surrogate=surr, use_net=True)
                ttt["mixed_surrogate_coarse_only"] = time_to_target(ap, nl, "bf16x3", surrogate=surr,
                                                                    use_net=False)
                surr.close()
                plain_s = ttt["plain"]["seconds"]
                for k in ("mixed", "mixed_surrogate", "mixed_surrogate_coarse_only"):
                    ttt[k]["speedup_vs_plain"] = plain_s / ttt[k]["seconds"]
            if solver == "bf16x3" and not args.no_c4:
                ttt["c4"] = c4_block(ap)
        if not args.no_cpu_baseline:
            cpu = cpu_baseline(nl)
        line = {
            "metric": METRIC, "value": total_iters / t_max, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32+bf16x3" if tensor_cores(solver) else "f32", "data": "synthetic",
            "config": {**workload_desc(nl, args.preset), "field_solver": solver,
                       "step": "one trial step (one gradient evaluation); value counts accepted iterations",
                       "parallelism": "replicas" if world > 1 else "single"},
            "iterations": total_iters, "evals": evals, "evals_per_s": evals / t_max,
            "gpu_launches": launches_per_trial * args.steps,
            "e2e": {"value": e2e_iters / e2e_s, "unit": UNIT, "h2d_bytes_per_step": 8 * n_mov,
                    "d2h_bytes_per_step": 8 * n + 160, "steps": e2e_steps},
            "roofline": roof, "clocks": clk, "time_to_10pct_overflow": ttt, "cpu_baseline": cpu,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
