#!/usr/bin/env python
"""Benchmark of the DMM integrator hot path: clause-updates/s.

Workload (one GPU): planted random 3-SAT, n = 100,000 variables, m = 800,000 clauses
(r = 8; the number of literals agreeing with the planted assignment is 3 with probability
0.08 and 1 or 2 with probability 0.46 each), FP32 production state, initial state
V ~ U[-1,1], Xs ~ U[0,1], Xl = 1.  Synthetic data: the reference's own n = 100,000
instances are not available, so the project generator with these parameters stands in.

A "step" is one accepted integration step (right-hand side of every clause, deterministic
per-variable reduction, adaptive h, Euler update) of that instance.  `value` is
m x steps / device time of the timed steps, with an L2 flush (256 MiB write) before every
timed step so each step starts from HBM; `e2e` is the same metric through the C ABI from
host buffers (create + state upload + steps + assignment readback).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

N > 1 runs under torchrun, one independent instance per GPU (replicas; no collective on
the data path), timed on the device, max over ranks.
"""
from __future__ import annotations

import argparse
import json
import multiprocessing as mp
import os
import re
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "dynex-neuromorphic-chip_b200")
for _p in (ROOT, PKG):
    if _p not in sys.path:
        sys.path.insert(0, _p)

N_VARS, N_CLAUSES, P0, P1 = 100_000, 800_000, 0.08, 0.46
INSTANCE_SEED, INIT_SEED = 1, 1001
FLUSH_BYTES = 256 << 20
METRIC = "clause-updates/s"
WORKLOAD = "planted 3-SAT n=100000 m=800000 r=8 p0=0.08 p1=0.46, one formula per GPU"
E2E_STEPS = 64
CPU_SAMPLE_STEPS = 60
LARGE_N, LARGE_SEED = 1_000_000, 3


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=40)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--procs", type=int, default=0,
                    help="reference arm: host processes (default: one per core)")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the batched and served workloads (rank 0, one GPU)")
    ap.add_argument("--precision-study", action="store_true",
                    help="only run the FP32-vs-FP64 study (n=1,000,000) and print its line")
    ap.add_argument("--study-n", type=int, default=1_000_000)
    ap.add_argument("--study-seeds", type=int, default=64)
    ap.add_argument("--study-ratio", type=float, default=8.0,
                    help="clause-to-variable ratio of the study's formula")
    ap.add_argument("--study-max-steps", type=int, default=5000)
    ap.add_argument("--prior-art-gpu", action="store_true",
                    help="only time the reference's GPU prior art (dynex.cu) on the bench formula "
                         "and print its line (run by the default run in a child process)")
    ap.add_argument("--no-study", action="store_true",
                    help="leave the precision study out of the default run")
    return ap.parse_args()


def run_extras(device: int) -> dict:
    """The batched and served configurations (see dmm_b200/workloads.py), each against the
    plain path that takes the same formulas one at a time.  Per-formula results are
    identical on every path, so the solve rates are equal by construction."""
    import numpy as np

    from dmm_b200 import workloads as w

    from dmm_b200.tuner import autotune_batch

    items = w.make_items(4096, 100, 5000, ratios=(8.0,), seed=1)
    tuned = autotune_batch(items, max_steps=2000, device=device)
    b = w.run_batched(items, max_steps=2000, tuning=tuned["best"], device=device)
    sample = items[:64]
    p = w.run_plain(sample, max_steps=2000, device=device)
    pb = w.run_batched(sample, max_steps=2000, device=device)
    assert p["steps"] == pb["steps"], "per-formula results differ between paths"
    batched = {
        "workload": "4096 planted 3-SAT formulas, n log-uniform [100, 5000], r=8, p0=0.08, "
                    "FP32, step cap 2000, one pack",
        "clause_updates_per_s": b["clause_updates_per_s"], "device_ms": b["device_ms"],
        "solved": b["solved"], "instances": b["instances"],
        "solves_per_s": b["solves_per_s_run"], "solves_per_s_incl_setup": b["solves_per_s"],
        "setup_s": b["setup_s"],
        "steps_p50_p99_max": [float(x) for x in np.percentile(b["steps"], [50, 99, 100])],
        "plain_sample": {"instances": p["instances"], "solved": p["solved"],
                         "solves_per_s": p["solves_per_s"],
                         "clause_updates_per_s": p["clause_updates_per_s"],
                         "path": "dmm_instance create + solve, one formula at a time"},
        "batched_same_sample_solves_per_s": pb["solves_per_s_run"],
        "batched_same_sample_solves_per_s_incl_setup": pb["solves_per_s"],
        "autotune": {"best": tuned["best"],
                     "sample_device_ms": {f"var_group={g},steps_per_graph={sp}": round(ms, 3)
                                          for (g, sp), ms in tuned["table"]},
                     "note": "first 512 formulas, each shape; results identical for every shape"},
        # set-up (formula upload, device CSR build, initial state) is inside both rates
        "solves_ratio_vs_plain": b["solves_per_s"] / max(p["solves_per_s"], 1e-9),
        "solves_ratio_vs_plain_run_only": b["solves_per_s_run"] / max(p["solves_per_s"], 1e-9),
        "roofline": dict(roofline(
            sum((28 * it.formula.m + 8 * it.formula.n) * st for it, st in zip(items, b["steps"])),
            b["device_ms"], "k_inst (one block per formula, many steps per launch)",
            traffic=None,
            note="algorithmic bytes (28m + 8n per accepted step) of every formula's steps over "
                 "the run's device time; traffic_over_algo: ncu DRAM bytes over algorithmic "
                 "bytes of one captured launch (the 512 largest formulas' first 256 steps), "
                 "read from the committed profile summary"),
            traffic_over_algo=profiled_ratio("k_inst_c3.md")),
    }
    sv = w.make_items(300, 100, 100000, ratios=(4.3, 6.0, 8.0), seed=2)
    arr = w.poisson_times(len(sv), 200.0, seed=2)
    s = w.run_served(sv, arr, budget_bytes=150 << 30, max_steps=3000, device=device)
    sp = w.run_served_plain(sv, arr, max_steps=3000, device=device)
    served = {
        "workload": "300 requests, Poisson 200/s, planted 3-SAT n log-uniform [100, 100000], "
                    "r in {4.3, 6, 8}, p0=0.08, FP32, step cap 3000, budget 150 GB",
        "solved": s["solved"], "requests": s["requests"], "solves_per_s": s["solves_per_s"],
        "p50_tts_s": s["p50_tts_s"], "p99_tts_s": s["p99_tts_s"], "wall_s": s["wall_s"],
        "plain": {"solved": sp["solved"], "solves_per_s": sp["solves_per_s"],
                  "p50_tts_s": sp["p50_tts_s"], "p99_tts_s": sp["p99_tts_s"],
                  "path": "same arrivals, one request at a time"},
    }
    # formulas of the bench's size batched: 64 planted 3-SAT formulas at n = 100,000 in one
    # pack (the tile kernels, all formulas stepping together) against the same formulas one
    # at a time on the plain path (the staged kernel, create + solve each)
    big = w.make_items(64, 100_000, 100_000, ratios=(8.0,), seed=4)
    bl = w.run_batched(big, max_steps=1000, device=device)
    pl = w.run_plain(big, max_steps=1000, device=device)
    assert bl["steps"] == pl["steps"], "per-formula results differ between paths"
    batched_large = {
        "workload": "64 planted 3-SAT formulas, n=100000, r=8, p0=0.08, FP32, step cap 1000",
        "solved": bl["solved"], "solves_per_s_incl_setup": bl["solves_per_s"],
        "solves_per_s_run": bl["solves_per_s_run"], "setup_s": bl["setup_s"],
        "clause_updates_per_s": bl["clause_updates_per_s"], "device_ms": bl["device_ms"],
        "plain": {"solved": pl["solved"], "solves_per_s": pl["solves_per_s"],
                  "clause_updates_per_s": pl["clause_updates_per_s"]},
        "solves_ratio_vs_plain": bl["solves_per_s"] / max(pl["solves_per_s"], 1e-9),
    }
    # the literal-agreement split of the bench (0.08 / 0.46 / 0.46, as the benchmark states it)
    # against the split of the reference's own fixtures (0.08 / 0.58 / 0.34, Barthel's
    # balanced ensemble): same size, same seeds, each ensemble solved as one batch
    ens = {}
    for label, p1 in (("bench split p0=0.08 p1=0.46 p2=0.46", 0.46),
                      ("fixture split p0=0.08 p1=0.58 p2=0.34", 0.58)):
        its = w.make_items(64, 10_000, 10_000, ratios=(8.0,), seed=3, p1=p1)
        r = w.run_batched(its, max_steps=5000, device=device)
        solved = [st for st, ok in zip(r["steps"], r["solved_flags"]) if ok]
        ens[label] = {"formulas": len(its), "solve_rate": len(solved) / len(its),
                      "steps_p50": float(np.median(solved)) if solved else None,
                      "steps_p90": float(np.percentile(solved, 90)) if solved else None,
                      "device_ms": r["device_ms"]}
    ensembles = {"workload": "64 planted 3-SAT formulas per ensemble, n=10000, r=8, FP32, "
                             "initial state V~U[-1,1], Xs~U[0,1], Xl=1, step cap 5000",
                 "ensembles": ens}
    return {"batched": batched, "batched_large": batched_large, "served": served,
            "ensembles": ensembles}


# ---- helpers ------------------------------------------------------------------------------

class Clocks:
    """nvidia-smi samples (every 200 ms) during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        time.sleep(0.25)
        if self.p:
            self.p.terminate()
            try:
                self.p.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.p.kill()

    def summary(self) -> dict:
        self.f.flush()
        rows = []
        with open(self.f.name) as fh:
            for line in fh:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        os.unlink(self.f.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"], "samples": 0}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i] == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons, "samples": len(rows)}


def peaks() -> tuple[float, str]:
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback"


KERNELS = {"staged": "k_staged (fused step, staged form)",
           "staged-multi": "k_staged (fused step, staged form, several tiles per block)",
           "cooperative-single": "k_persist (fused step, single formula)",
           "cooperative": "k_persist (fused step)",
           "two-kernel": "k_clause + k_var", "one-block-per-formula": "k_inst",
           "cluster": "k_cluster (fused step, one thread-block cluster)",
           "resident-grid": "k_grid (fused step, voltages resident in shared memory)",
           "streaming": "k_stream (fused step, tables and voltage lists streamed through shared "
                        "memory)"}
# committed ncu summary of each kernel on the formula of 10^6 variables
LARGE_PROFILES = {"streaming": "k_stream_n1m.md", "staged-multi": "k_staged_n1m.md"}


def profiled_ratio(summary: str) -> float | None:
    """DRAM bytes over algorithmic bytes of a captured launch, from a committed ncu summary
    under profiles/ (its line `traffic_over_algo: X`); None when there is none."""
    p = os.path.join(ROOT, "profiles", summary)
    try:
        with open(p) as f:
            m = re.search(r"traffic_over_algo:\s*([0-9.eE+]+)", f.read())
        return float(m.group(1)) if m else None
    except OSError:
        return None


def profiled_traffic(summary: str) -> float | None:
    """DRAM bytes per launch of a step kernel, from a committed ncu summary under profiles/
    (its line `traffic_bytes_per_launch: X`); None when there is none."""
    p = os.path.join(ROOT, "profiles", summary)
    try:
        with open(p) as f:
            m = re.search(r"traffic_bytes_per_launch:\s*([0-9.eE+]+)", f.read())
        return float(m.group(1)) if m else None
    except OSError:
        return None


def make_instance(rank: int):
    import dmm_b200 as dmm

    form, planted = dmm.generate_planted(N_VARS, N_CLAUSES, P0, P1, seed=INSTANCE_SEED + rank)
    x0 = dmm.initial_state_uniform(form, INIT_SEED + rank)
    return form, x0


def bench_config(world: int) -> dict:
    """The workload description both arms print (the reference arm's line must carry the
    same config as this one's)."""
    return {"workload": WORKLOAD, "n": N_VARS, "m": N_CLAUSES, "instance_seed": INSTANCE_SEED,
            "init_seed": INIT_SEED, "per_gpu_instances": 1,
            "l2": "GPU arm: flushed (256 MiB write) before every timed step; CPU reference "
                  "arm: no flush (its working set exceeds the host caches)",
            "parallelism": f"replicas x{world}"}


# ---- reference arm (CPU) ------------------------------------------------------------------

def _ref_worker(args):
    """One host process: the instance and initial state built by the reference harness
    library (no other native library is loaded), then `warmup` untimed and `steps` timed
    accepted steps of the reference's own right-hand side and Euler step."""
    steps, warmup = args
    from oracle.oracle import Reference, planted_instance

    lits, off, _, x0 = planted_instance(N_VARS, N_CLAUSES, P0, P1, INSTANCE_SEED, INIT_SEED)
    ref = Reference(N_VARS, N_CLAUSES, lits, off)
    if warmup:
        ref.run(x0, warmup)
    t0 = time.perf_counter()
    r = ref.run(x0, steps)
    dt = time.perf_counter() - t0
    return r["steps"], dt, repo_libraries()


def repo_libraries() -> list[str]:
    """Shared libraries of this repository mapped into the calling process (Linux)."""
    found = set()
    try:
        with open("/proc/self/maps") as f:
            for line in f:
                path = line.split()[-1] if len(line.split()) >= 6 else ""
                if path.endswith(".so") and path.startswith(ROOT + os.sep):
                    found.add(os.path.relpath(path, ROOT))
    except OSError:
        pass
    return sorted(found)


def reference_missing() -> str | None:
    """Why the reference arm and the CPU baseline cannot run here, or None when they can."""
    from oracle.oracle import REF_SO, reference_available

    if reference_available():
        return None
    return f"{os.path.relpath(REF_SO, ROOT)} was not built: the reference's sources are not here"


def cpu_reference(steps: int, warmup: int, procs: int):
    """The unmodified reference integrator (oracle/_ref, dynex.cc's own right-hand side and
    Euler step) on `procs` host processes at once, all on the bench instance and initial
    state; returns (clause-updates/s over the slowest process, details)."""
    ctx = mp.get_context("spawn")
    with ctx.Pool(procs) as pool:
        t0 = time.perf_counter()
        res = pool.map(_ref_worker, [(steps, warmup)] * procs)
        wall = time.perf_counter() - t0
    done = sum(r[0] for r in res)
    t = max(r[1] for r in res)
    libs = sorted({x for r in res for x in r[2]})
    return N_CLAUSES * done / t, {"procs": procs, "steps_each": [r[0] for r in res],
                                  "timed_s": t, "wall_s": wall, "libraries": libs}


def prior_art_gpu(steps: int, warmup: int) -> dict:
    """The reference's own GPU code (dynex.cu, unmodified, built for sm_100a by
    oracle/Makefile) on the bench formula and initial state: its FP64 kernels with one thread
    per clause and CAS-loop atomics, and its host loop that reads loc, energy and each
    adaptive trial's changed-variable count back every step.  Wall time of `steps` steps
    (the loop synchronizes at every copy) after `warmup` untimed ones."""
    from oracle.oracle import GpuPriorArt, planted_instance

    lits, off, _, x0 = planted_instance(N_VARS, N_CLAUSES, P0, P1, INSTANCE_SEED, INIT_SEED)
    g = GpuPriorArt(N_VARS, N_CLAUSES, lits, off)
    g.run(x0, warmup)
    ms, done, loc = g.run(x0, steps)
    g.close()
    return {"impl": "dynex.cu (the reference's GPU prior art), FP64", "value": N_CLAUSES * done / (ms / 1e3),
            "unit": "clause-updates/s", "ms_per_step": ms / max(1, done), "steps": done,
            "workload": WORKLOAD, "timing": "host wall clock around its synchronous loop"}


def prior_art_child(steps: int, warmup: int) -> dict | None:
    """prior_art_gpu in a child process (its statically linked CUDA runtime stays out of this
    process); None when the prebuilt library is absent or the run fails."""
    from oracle.oracle import REF_GPU_SO

    if not os.path.exists(REF_GPU_SO):
        return None
    r = subprocess.run([sys.executable, os.path.abspath(__file__), "--prior-art-gpu", "--steps",
                        str(steps), "--warmup", str(warmup)], capture_output=True, text=True,
                       timeout=600)
    if r.returncode != 0:
        return {"unavailable": (r.stderr.strip().splitlines() or ["failed"])[-1][:200]}
    return json.loads(r.stdout.strip().splitlines()[-1])


def run_reference_arm(a):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    why = reference_missing()
    if why:
        print(json.dumps({"impl": "reference", "unavailable": why}), flush=True)
        return
    procs = a.procs or max(1, os.cpu_count() or 1)
    steps, warmup = a.steps, max(3, a.warmup)
    value, info = cpu_reference(steps, warmup, procs)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "clause-updates/s",
        "n_gpus": a.gpus, "steps": steps, "warmup": warmup,
        "ms_per_step": 1000.0 * info["timed_s"] / steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": bench_config(a.gpus),
        "cpu_baseline": {"value": value, "unit": "clause-updates/s", "cores": procs,
                         "kind": "reference",
                         "sample": f"{procs} processes, each {warmup} untimed + {steps} timed "
                                   "steps of the bench instance and initial state (the "
                                   "unmodified dynex.cc right-hand side and Euler step with "
                                   "its adaptive loop, one thread each)"},
        "e2e": {"value": value, "unit": "clause-updates/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
        "steps_done_per_process": info["steps_each"],
        "repo_libraries_loaded": info["libraries"],
    }
    print(json.dumps(line), flush=True)


# ---- our arm ------------------------------------------------------------------------------

class Ranks:
    """One process per GPU (torchrun): barrier, max / sum / any over ranks.  The run shards
    nothing (each rank integrates its own replica), so these are the only collectives, and
    every rank takes them in the same order.  backend "nccl" with device "cuda:<local>" on
    GPUs; "gloo" with device "cpu" in the multi-process CPU tests."""

    def __init__(self, world: int, backend: str = "nccl", device: str = "cpu"):
        import torch

        self.torch = torch
        self.world = world
        self.device = device
        self.dist = None
        if world > 1:
            import datetime

            import torch.distributed as dist

            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=120))
            self.dist = dist

    def barrier(self) -> None:
        if self.dist is not None:
            self.dist.barrier()
        if self.device.startswith("cuda"):
            self.torch.cuda.synchronize()

    def _reduce(self, x: float, op) -> float:
        if self.dist is None:
            return float(x)
        t = self.torch.tensor([float(x)], dtype=self.torch.float64, device=self.device)
        self.dist.all_reduce(t, op=op)
        return float(t.item())

    def max(self, x: float) -> float:
        return self._reduce(x, self.dist.ReduceOp.MAX if self.dist else None)

    def sum(self, x: float) -> float:
        return self._reduce(x, self.dist.ReduceOp.SUM if self.dist else None)

    def any(self, flag: bool) -> bool:
        """True on every rank when the flag is set on any rank (collective decisions)."""
        return self.max(1.0 if flag else 0.0) > 0.0

    def close(self) -> None:
        if self.dist is not None:
            self.dist.barrier()
            self.dist.destroy_process_group()
            self.dist = None


def time_plain(inst, x0, K, W, ranks, barrier, clocks_gpu=None):
    """Device time of K steps of `inst` from x0, each launched alone after an L2 flush (W
    untimed steps first), restarting from a later initial state when a replica solved
    inside the timed region (every rank takes the same collective decision).  Returns
    (ms, steps done, clocks summary or None, x0 used)."""
    import dmm_b200 as dmm

    f = inst.formula
    init_seed = INIT_SEED
    clocks = None
    for attempt in range(4):
        inst.set_state(x0)
        inst.time_steps_flushed(W, FLUSH_BYTES)  # warm-up: the same launches as timed
        barrier()
        s0 = inst.report().steps
        if clocks_gpu is not None:
            with Clocks(clocks_gpu) as clk:
                step_ms = inst.time_steps_flushed(K, FLUSH_BYTES)
            clocks = clk.summary()
        else:
            step_ms = inst.time_steps_flushed(K, FLUSH_BYTES)
        barrier()
        steps_done = inst.report().steps - s0
        if not ranks.any(steps_done != K):
            break
        init_seed += 1000
        x0 = dmm.initial_state_uniform(f, init_seed)
    return step_ms, steps_done, clocks, x0


def time_resident(inst, x0, K, W):
    """K steps on the solver's own launch path (cooperative launches of several steps each,
    no flush); returns (ms, steps)."""
    inst.set_state(x0)
    inst.time_steps(W)
    s0 = inst.report().steps
    ms = inst.time_steps(K)
    return ms, inst.report().steps - s0


def time_e2e(form, x0, precision, device, barrier, reps=7):
    """Create + state upload + E2E_STEPS steps + assignment readback through the C ABI from
    pinned host buffers; median wall time of `reps` calls after 2 untimed ones."""
    import torch

    import dmm_b200 as dmm

    lits_p = torch.from_numpy(form.lits).pin_memory()
    off_p = torch.from_numpy(form.clause_off).pin_memory()
    x0_p = torch.from_numpy(x0).pin_memory()
    pform = dmm.Formula(form.n, form.m, lits_p.numpy(), off_p.numpy(), form.max_occurrence)
    times, steps = [], []
    for it in range(2 + reps):
        barrier()
        t0 = time.perf_counter()
        with dmm.Instance(pform, precision=precision, device=device) as e:
            e.set_state(x0_p.numpy())
            r = e.step(E2E_STEPS)
            _, post = e.assignment(pre=False)
        dt = time.perf_counter() - t0
        if it >= 2:
            times.append(dt)
            steps.append(r.steps)
    h2d = form.lits.nbytes + form.clause_off.nbytes + x0.nbytes
    d2h = form.n + 56
    return statistics.median(times), statistics.median(steps), h2d, d2h


def roofline(algo_bytes_per_launch, launch_ms, kernel, traffic=None, note=None):
    peak, peak_kind = peaks()
    achieved = algo_bytes_per_launch / (launch_ms / 1000.0) / 1e9
    r = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
         "frac": achieved / peak, "traffic": traffic, "kernel": kernel, "peak_kind": peak_kind,
         "algo_bytes_per_launch": algo_bytes_per_launch}
    if traffic:
        r["traffic_over_algo"] = traffic / algo_bytes_per_launch
    if note:
        r["note"] = note
    return r


def fp64_line(form, x0, K, W, device, ranks, barrier) -> dict:
    """The same formula and state in FP64, the reference's arithmetic (bit-exact): the
    like-for-like comparison with the reference's precision."""
    import dmm_b200 as dmm

    n, m = form.n, form.m
    with dmm.Instance(form, precision="fp64", device=device) as inst:
        kern = KERNELS[inst.step_kernel]
        ms, done, _, xs = time_plain(inst, x0, K, W, ranks, barrier)
        rms, rsteps = time_resident(inst, xs, K, W)
    e_t, e_steps, h2d, d2h = time_e2e(form, x0, "fp64", device, barrier, reps=5)
    algo = 44 * m + 16 * n  # literals 12m, Xs/Xl read+write 32m, V read 8n + write 8n
    return {"value": m * done / (ms / 1000.0), "unit": "clause-updates/s",
            "ms_per_step": ms / K, "dtype": "f64",
            "resident": {"value": m * rsteps / (rms / 1000.0), "ms_per_step": rms / max(1, rsteps)},
            "e2e": {"value": m * e_steps / e_t, "unit": "clause-updates/s",
                    "h2d_bytes_per_step": h2d / E2E_STEPS, "d2h_bytes_per_step": d2h / E2E_STEPS},
            "roofline": roofline(algo, ms / K, kern,
                                 traffic=profiled_traffic("k_persist_fp64_n100k.md"))}


def large_line(K, W, device, ranks, barrier) -> dict:
    """Plain single formula at n = 1,000,000, m = 8,000,000 (FP32), whose per-step working set
    (2.3e8 algorithmic bytes) exceeds the 126 MB L2: the configuration where the step is
    bound by HBM."""
    import dmm_b200 as dmm

    n, m = LARGE_N, LARGE_N * 8
    f, _ = dmm.generate_planted(n, m, P0, P1, seed=LARGE_SEED)
    x0 = dmm.initial_state_uniform(f, LARGE_SEED + 1000)
    out = {"workload": f"planted 3-SAT n={n} m={m} r=8 p0=0.08 p1=0.46, one formula, FP32",
           "n": n, "m": m}
    with dmm.Instance(f, precision="fp32", device=device) as inst:
        kern = inst.step_kernel
        out["launch_form"], out["step_kernel"] = inst.launch_form, kern
        ms, done, _, xs = time_plain(inst, x0, K, W, ranks, barrier)
        rms, rsteps = time_resident(inst, xs, K, W)
    algo = 28 * m + 8 * n
    out.update({"value": m * done / (ms / 1000.0), "unit": "clause-updates/s",
                "ms_per_step": ms / K,
                "resident": {"value": m * rsteps / (rms / 1000.0),
                             "ms_per_step": rms / max(1, rsteps)},
                "roofline": roofline(algo, ms / K, KERNELS[kern],
                                     traffic=profiled_traffic(LARGE_PROFILES.get(kern, "")))})
    return out


def main():
    a = parse()
    if a.impl == "reference":
        run_reference_arm(a)
        return
    if a.prior_art_gpu:
        print(json.dumps(prior_art_gpu(a.steps, max(3, a.warmup))), flush=True)
        return
    if a.precision_study:
        from dmm_b200 import workloads as w

        r = w.precision_study(n=a.study_n, r=a.study_ratio, seeds=range(a.study_seeds),
                              max_steps=a.study_max_steps)
        print(json.dumps({"precision_study": r, "workload": f"planted 3-SAT n={a.study_n}, "
                          f"r={a.study_ratio:g}, p0=0.08, FP32 vs FP64 from the same initial "
                          "states"}), flush=True)
        return
    import torch

    import dmm_b200 as dmm

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        torch.cuda.set_device(local)
    ranks = Ranks(world, "nccl", f"cuda:{local}")
    barrier, max_over_ranks, sum_over_ranks = ranks.barrier, ranks.max, ranks.sum

    form, x0 = make_instance(rank)
    n, m = form.n, form.m
    K, W = a.steps, max(3, a.warmup)
    inst = dmm.Instance(form, precision="fp32", device=local)
    form_name, kernel_name = inst.launch_form, inst.step_kernel
    step_ms, steps_done, clocks, x0 = time_plain(inst, x0, K, W, ranks, barrier, local)
    t_max = max_over_ranks(step_ms)
    total_updates = sum_over_ranks(m * steps_done)
    value = total_updates / (t_max / 1000.0)

    # phase breakdown with one kernel per phase (same arithmetic, separate launches)
    tun = inst.tuning
    inst.set_tuning(launch_mode=1)
    inst.set_state(x0)
    inst.profile(W, FLUSH_BYTES)
    clause_ms, var_ms = inst.profile(K, FLUSH_BYTES)
    inst.set_tuning(**tun)

    # resident: the solver's own launch path (cooperative launches of steps_per_graph steps
    # each, no flush; this formula's 4.2e7-byte working set stays in the 126 MB L2)
    res_ms, res_steps = time_resident(inst, x0, K, W)
    resident_value = sum_over_ranks(m * res_steps) / (max_over_ranks(res_ms) / 1000.0)

    # end to end through the C ABI from pinned host buffers
    e2e_med, e2e_steps, h2d, d2h = time_e2e(form, x0, "fp32", local, barrier)
    e2e_t = max_over_ranks(e2e_med)
    e2e_value = sum_over_ranks(m * e2e_steps) / e2e_t

    algo_bytes = 28 * m + 8 * n  # per step: literals 12m, Xs/Xl read+write 16m, V 4n + 4n
    launch_ms = t_max / K  # one cooperative launch = one step

    cpu = None
    if rank == 0 and world == 1 and not a.no_cpu_baseline and (why := reference_missing()):
        cpu = {"unavailable": why}
    elif rank == 0 and world == 1 and not a.no_cpu_baseline:
        v, info = cpu_reference(CPU_SAMPLE_STEPS, 3, 1)
        cpu = {"value": v, "unit": "clause-updates/s", "cores": 1, "kind": "reference",
               "sample": f"{CPU_SAMPLE_STEPS} steps (after 3 untimed) of the same formula and "
                         "initial state, the unmodified dynex.cc right-hand side and Euler step "
                         "with its adaptive loop, 1 thread"}

    extras = {}
    if rank == 0 and world == 1 and not a.no_extras:
        extras["fp64"] = fp64_line(form, x0, K, W, local, ranks, barrier)
        pa = prior_art_child(K, W)
        if pa is not None:
            extras["prior_art_gpu"] = pa
        extras["large"] = large_line(K, W, local, ranks, barrier)
        extras.update(run_extras(local))
        if not a.no_study:
            from dmm_b200 import workloads as w

            extras["precision_study"] = w.precision_study(
                n=a.study_n, r=a.study_ratio, seeds=range(a.study_seeds),
                max_steps=a.study_max_steps)
            # at r = 8 every run solves before step 1000; the 1000-step horizon comes from a
            # formula below the threshold (r = 4.3), which keeps integrating
            extras["precision_study_r43"] = w.precision_study(
                n=a.study_n, r=4.3, seeds=range(8), max_steps=1000)

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "clause-updates/s", "n_gpus": world,
            "steps": K, "warmup": W, "ms_per_step": t_max / K, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "fp32", "data": "synthetic",
            "config": bench_config(world),
            "clocks": clocks,
            "e2e": {"value": e2e_value, "unit": "clause-updates/s",
                    "h2d_bytes_per_step": h2d / E2E_STEPS, "d2h_bytes_per_step": d2h / E2E_STEPS,
                    "path": f"dmm_instance_create + set_state + {E2E_STEPS} steps + assignment "
                            "readback, pinned host buffers"},
            "gpu_launches": K,
            "roofline": roofline(algo_bytes, launch_ms, KERNELS[kernel_name],
                                 traffic=profiled_traffic("k_staged_n100k.md"),
                                 note="traffic: ncu DRAM bytes of one launch of this kernel on "
                                      "this workload, read from the committed profile summary"),
            "tuning": inst.tuning, "launch_form": form_name,
            "phase_ms_per_step": {"k_clause": clause_ms / K, "k_var": var_ms / K,
                                  "note": "kernel-per-phase form, L2 flushed"},
            "resident": {"value": resident_value, "unit": "clause-updates/s",
                         "ms_per_step": res_ms / max(1, res_steps),
                         "note": "cooperative launches of several steps each (the solver's "
                                 "own launch path), no L2 flush"},
        }
        if cpu is not None:
            line["cpu_baseline"] = cpu
        line.update(extras)
        print(json.dumps(line), flush=True)
    inst.close()
    ranks.close()


if __name__ == "__main__":
    main()
