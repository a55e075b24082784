"""Throughput of the fused WCA flood step on B200.

Workload (config 2 of the benchmark set): a 4096 x 4096 grid at 90 m (16.8 M LAND
cells), fBm relief of 20 m amplitude, six Manning classes, 30 mm/h rain for
2 h and a north-edge point inflow (triangle peaking at 500 m^3/s at 3 h),
open south edge. A "step" is one WCA step over the whole grid. The timed
steps start from a warm state: 20 mm of water on every cell (what 40 minutes
of the storm leaves), as the reference's benchmarks start from a warm start.
Inputs are far larger than L2 (about 420 MB touched per step), so no L2
flush is needed between steps.

Metric: Gcell-updates/s = LAND cells x steps / time (the reference's mcups,
src/common/log.c:133-135). `value` is timed on the device with CUDA events
around K steps on the session stream; `e2e` is a whole config-2 run (6 h
simulated) through the reference-facing fca_cuda_run C-ABI with host
buffers, host<->device copies included. `cpu_baseline` is the reference's
own OpenMP core (compiled from its sources with its release flags) on a
bounded sample of the same workload on this host's cores.

--impl reference times that reference CPU implementation alone.
Multi-GPU: independent replicas, one per rank (the 4096^2 domain fits one
GPU; domains beyond one GPU run as row slabs, floodca_b200.slabs); value is
the whole-job aggregate, max-over-ranks time.
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
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "Gcell-updates/s"
# algorithmic bytes per cell-update: read z, h, n, hmax (4 B each), write h,
# hmax (4 B each); the generic layout also reads the mask (1 B), the all-LAND
# layout does not
BYTES_LAND_ONLY, BYTES_GENERIC = 24, 25


def warm_domain(n: int):
    from floodca_b200.profile_step import warm_config2
    return warm_config2(n)


def measured_peaks() -> dict:
    try:
        return json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except (OSError, ValueError):
        return {}


def profile_traffic() -> float | None:
    """DRAM bytes per step launch from the committed ncu summary, if any."""
    f = ROOT / "profiles" / "k_step_traffic.json"
    try:
        return float(json.loads(f.read_text())["dram_bytes_per_launch_4096"])
    except (OSError, ValueError, KeyError):
        return None


class ClockSampler:
    """nvidia-smi clock/throttle samples taken while the timed region runs."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.rows: list[list[str]] = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for ln in self.proc.stdout:
            self.rows.append([x.strip() for x in ln.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        sm = [float(r[1]) for r in self.rows if len(r) > 8 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) > 8 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows if len(r) > 8
                          for i, v in enumerate(r[5:9]) if v.lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(sm)}


# ---------------------------------------------------------------------------
# Reference CPU implementation (the OpenMP core compiled in oracle/_ref).

def reference_cpu(dom, p, steps: int, warmup: int, budget_s: float) -> dict:
    threads = os.cpu_count() or 1
    os.environ.setdefault("OMP_NUM_THREADS", str(threads))
    os.environ.setdefault("OMP_PROC_BIND", "close")
    os.environ.setdefault("OMP_PLACES", "cores")
    from oracle import refcore
    from floodca_b200.sim import Domain
    kind = refcore.shipped_kind()
    if not refcore.available(kind):
        return {"unavailable": f"oracle/_ref/libfcaref_{kind}.so missing (reference not built)"}
    # time one step on the full grid to size the sample within the budget
    run = refcore.RefRun(dom, p.with_(steps=0, T_sim=1e7), kind)
    t0 = time.perf_counter()
    run.step()
    t1 = time.perf_counter() - t0
    nr = dom.shape[0]
    rows = nr
    if t1 * (steps + warmup) > budget_s:
        rows = max(64, int(nr * budget_s / (t1 * (steps + warmup))))
    if rows < nr:
        sl = slice(0, rows)
        dom = Domain(z=dom.z[sl], mask=dom.mask[sl], n=dom.n[sl], C=dom.C[sl], Rday=dom.Rday[sl],
                     h=dom.h[sl], dx=dom.dx, hmax=dom.hmax[sl], tmax=None)
        run = refcore.RefRun(dom, p.with_(steps=0, T_sim=1e7), kind)
    for _ in range(warmup):
        run.step()
    t0 = time.perf_counter()
    for _ in range(steps):
        run.step()
    wall = time.perf_counter() - t0
    cells = int((dom.mask == 0).sum())
    return {"value": cells * steps / wall / 1e9, "cores": threads, "kind": "reference",
            "sample": f"{rows}x{dom.shape[1]} rows of the warm 4096^2 config-2 grid, {steps} steps "
                      f"after {warmup} warm-up, libfcaref_{kind} (reference src/common, -O3 "
                      f"{'-march=x86-64-v4' if kind.endswith('v4') else '-march=x86-64-v3'}, OpenMP)",
            "wall_s": wall, "steps": steps, "cells": cells}


def line_reference(args, n: int) -> dict:
    dom, p = warm_domain(n)
    r = reference_cpu(dom, p, args.steps, args.warmup, args.cpu_budget)
    base = {"metric": METRIC, "impl": "reference", "unit": "Gcell/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config_block(n, args.gpus)}
    if "unavailable" in r:
        return {"impl": "reference", "unavailable": r["unavailable"]}
    base.update(value=r["value"], ms_per_step=1e3 * r["wall_s"] / r["steps"],
                cpu_baseline={"value": r["value"], "unit": "Gcell/s", "cores": r["cores"],
                              "kind": "reference", "sample": r["sample"]},
                e2e={"value": r["value"], "unit": "Gcell/s", "h2d_bytes_per_step": 0,
                     "d2h_bytes_per_step": 0})
    return base


def config_block(n: int, gpus: int) -> dict:
    return {"workload": f"config-2 single domain {n}x{n}, 90 m, point inflow + 30 mm/h rain, "
                        "open south edge, warm start (20 mm), FP32 stencil / FP64 accumulation",
            "grid": [n, n], "K": 4, "U": 1, "precision": "f32-exact",
            "parallelism": f"replicas x{gpus}" if gpus > 1 else "single GPU",
            "l2": "inputs (~420 MB per step) larger than L2; no flush"}


def e2e_mass_error(r: dict) -> float:
    """|V + V_sea + V_bnd - V_rain - V0 - clamp| / (V_rain + V0) of a run
    through the drop-in ABI (the reference's diag.c:5-14)."""
    den = max(r["V_rain"] + r["V0"], 1e-30)
    return abs(r["V"] + r["V_sea"] + r["V_bnd"] - r["V_rain"] - r["V0"] - r["clamp_err"]) / den


# ---------------------------------------------------------------------------
# The ensemble half of the metric: a seeded config-4 subset batched against
# the same members one at a time through the same kernel.

ENSEMBLE_MEMBERS = 32


def ensemble_leg(math: str = "exact") -> dict:
    from floodca_b200 import ensemble as E
    allm = E.config4_members(256)
    members = allm[::len(allm) // ENSEMBLE_MEMBERS]
    tune = E.DEFAULT_TUNING
    try:
        table = json.loads(E.TUNING_FILE.read_text())
        tune = table.get(E._tuning_key(math), tune)
    except (OSError, ValueError):
        pass
    bat = E.run_batched(members, math, tune, window=0.0)
    one = E.run_one_at_a_time(members, math)
    same = all(a["step"] == b["step"] and a["t"] == b["t"]
               for a, b in zip(bat["stats"], one["stats"]))
    return {"workload": f"config 4 subset: {len(members)} members (every "
                        f"{len(allm) // len(members)}th of the seeded 256), side "
                        f"{min(m.side for m in members)}..{max(m.side for m in members)}, "
                        "8 h simulated, 20-150 mm/h for 0.5-4 h, own terrain and n scale each",
            "members": len(members),
            "batched_members_per_hour": bat["members_per_hour"],
            "one_at_a_time_members_per_hour": one["members_per_hour"],
            "multiple": bat["members_per_hour"] / one["members_per_hour"],
            "batched_wall_s": bat["wall_s"], "one_at_a_time_wall_s": one["wall_s"],
            "batched_gcell_steps_per_s": bat["cell_steps"] / bat["wall_s"] / 1e9,
            "one_at_a_time_gcell_steps_per_s": one["cell_steps"] / one["wall_s"] / 1e9,
            "members_steps_and_times_equal": same,
            "tuning": {k: tune[k] for k in ("cols_per_lane", "seg_rows_by_class")},
            "timing": "host wall around the runs with device synchronisation; terrain "
                      "generation and upload excluded (both arms)"}


# ---------------------------------------------------------------------------
# Per-configuration table: the same workloads on the GPU (sessions) and on the
# reference's OpenMP core with all host threads and with one.

TABLE_CONFIGS = {
    "C1": "config 1, 256x256, full run (2 h simulated)",
    "C2": "config 2, 4096x4096, warm, fixed step window",
    "C3": "config 3, 2048x2048, warm, fixed step window",
}


def _table_domain(name: str):
    from floodca_b200 import synth
    if name == "C1":
        return synth.config1()
    if name == "C2":
        return warm_domain(4096)
    dom, p = synth.config3()
    dom = dom.copy()
    dom.h = np.full(dom.shape, 0.02, np.float32)
    dom.hmax = dom.h.copy()
    return dom, p


def cpu_table_worker(name: str, steps: int) -> dict:
    """Runs in a child process so OMP_NUM_THREADS takes effect."""
    from oracle import refcore
    kind = refcore.shipped_kind()
    if not refcore.available(kind):
        return {"unavailable": "reference not built"}
    dom, p = _table_domain(name)
    cells = int((dom.mask == 0).sum())
    if name == "C1":
        t0 = time.perf_counter()
        r = refcore.run(dom, p, kind)
        wall = time.perf_counter() - t0
        return {"gcells": cells * r["step"] / wall / 1e9, "steps": r["step"], "wall_s": wall}
    run = refcore.RefRun(dom, p.with_(steps=0, T_sim=1e7), kind)
    run.step()
    t0 = time.perf_counter()
    for _ in range(steps):
        run.step()
    wall = time.perf_counter() - t0
    return {"gcells": cells * steps / wall / 1e9, "steps": steps, "wall_s": wall}


def config_table() -> dict:
    import torch
    from floodca_b200.sim import Session
    cores = os.cpu_count() or 1
    out = {"cores": cores, "rows": []}
    for name, desc in TABLE_CONFIGS.items():
        dom, p = _table_domain(name)
        land = int((dom.mask == 0).sum())
        s = Session(dom, p if name == "C1" else p.with_(T_sim=30 * 86400.0))
        st = torch.cuda.ExternalStream(s.stream())
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        if name == "C1":
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            s.run()
            torch.cuda.synchronize()
            wall = time.perf_counter() - t0
            steps = s.stats()["step"]
            gpu = land * steps / wall / 1e9
        else:
            s.advance(20)
            torch.cuda.synchronize()
            e0.record(st)
            s.advance(200)
            e1.record(st)
            e1.synchronize()
            steps = 200
            gpu = land * steps / (e0.elapsed_time(e1) / 1e3) / 1e9
        s.close()
        row = {"config": name, "workload": desc, "land_cells": land, "gpu_gcells": gpu,
               "gpu_timing": "host wall, whole run" if name == "C1" else "CUDA events, 200 steps"}
        for label, threads, k in (("cpu_omp", cores, 10), ("cpu_1thread", 1, 3)):
            env = dict(os.environ, OMP_NUM_THREADS=str(threads), OMP_PROC_BIND="close",
                       OMP_PLACES="cores")
            r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--cpu-worker", name,
                                str(k)], capture_output=True, text=True, env=env, timeout=900)
            try:
                row[label] = json.loads(r.stdout.strip().splitlines()[-1])
            except (IndexError, ValueError):
                row[label] = {"unavailable": r.stderr[-300:]}
        out["rows"].append(row)
    return out


# ---------------------------------------------------------------------------

def main() -> int:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=2000)
    ap.add_argument("--warmup", type=int, default=50)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--size", type=int, default=4096)
    ap.add_argument("--math", default="exact", choices=["exact", "fast"])
    ap.add_argument("--cpl", type=int, default=0)
    ap.add_argument("--cpu-budget", type=float, default=20.0,
                    help="seconds of CPU time for the reference baseline sample")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-ensemble", action="store_true")
    ap.add_argument("--config-table", action="store_true",
                    help="GPU vs reference CPU (all threads, one thread) on configs 1-3")
    ap.add_argument("--cpu-worker", nargs=2, metavar=("CONFIG", "STEPS"), help=argparse.SUPPRESS)
    args = ap.parse_args()
    if args.cpu_worker:
        print(json.dumps(cpu_table_worker(args.cpu_worker[0], int(args.cpu_worker[1]))))
        return 0
    if args.config_table:
        print(json.dumps(config_table(), indent=1))
        return 0
    args.warmup = max(3, args.warmup)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    n = args.size

    if args.impl == "reference":
        if rank == 0:
            print(json.dumps(line_reference(args, n)), flush=True)
        return 0

    import torch
    import torch.distributed as dist
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))

    from floodca_b200.sim import DropinGrid, Session

    dom, p = warm_domain(n)
    # keep the run going for all W+K steps (events of the storm still apply)
    pb = p.with_(T_sim=30 * 86400.0)
    sess = Session(dom, pb, precision="f32", math=args.math, cols_per_lane=args.cpl)
    info = sess.info()
    land = info["land_cells"]
    stream = torch.cuda.ExternalStream(sess.stream())
    # clocks are sampled from the warm-up to the end of the last GPU leg
    clk = ClockSampler(local).__enter__()
    sess.advance(args.warmup)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    fp0 = sess.stats()["dt_full_passes"]      # (launches k_volume: before the count)
    l0 = sess.launches()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(stream)
    sess.advance(args.steps)
    e1.record(stream)
    e1.synchronize()
    torch.cuda.synchronize()
    launches = sess.launches() - l0
    ms = e0.elapsed_time(e1)
    st = sess.stats()
    full_passes = st["dt_full_passes"] - fp0
    active = st["step"] == args.warmup + args.steps
    if world > 1:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
        dist.barrier()
    sess.close()

    value = world * land * args.steps / (ms / 1e3) / 1e9
    per_launch_s = ms / 1e3 / args.steps
    bytes_per_cell = BYTES_LAND_ONLY if info["land_only"] else BYTES_GENERIC
    alg_bytes = bytes_per_cell * land
    peaks = measured_peaks()
    peak = peaks.get("hbm_gbs")
    achieved = alg_bytes / per_launch_s / 1e9
    roof = {"bound": "hbm", "achieved": achieved, "peak": peak or 6650.0, "unit": "GB/s",
            "frac": achieved / (peak or 6650.0), "traffic": profile_traffic(),
            "peak_source": "measured" if peak else "fallback",
            "bytes_per_cell": bytes_per_cell,
            "kernel": "k_step_blk" if info["tma_rows"] else "k_step",
            "time": "CUDA events around the timed steps on the session stream: one step-kernel "
                    "launch per step; the only other kernel in the region is the full velocity "
                    "pass that the step tail-launches when its dt seed missed "
                    "(full_velocity_passes of them, about 0.2 ms each), so achieved "
                    "understates the step kernel's own rate by that share",
            "full_velocity_passes": int(full_passes)}

    out = {"metric": METRIC, "value": value, "unit": "Gcell/s", "n_gpus": world,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms / args.steps,
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
           "data": "synthetic", "config": config_block(n, world), "roofline": roof,
           "gpu_launches": int(launches),
           "all_steps_active": bool(active), "launch": info, "math": args.math}

    if not args.no_e2e:
        dom2, p2 = __import__("floodca_b200.synth", fromlist=["config2"]).config2(n=n)
        # one untimed run first (one-time costs of the process: module
        # loading, first allocations), then three timed runs; the median
        # wall time is reported (host-side copies and teardown vary by
        # a few hundred ms between runs on a shared host)
        DropinGrid(dom2, p2.with_(steps=20)).run()
        walls = []
        for _ in range(3):
            g = DropinGrid(dom2, p2)
            torch.cuda.synchronize()
            if world > 1:
                dist.barrier()
            t0 = time.perf_counter()
            rc = g.run()
            walls.append(time.perf_counter() - t0)
        res = g.result()
        wall = statistics.median(walls)
        if world > 1:
            t = torch.tensor([wall], device="cuda", dtype=torch.float64)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            wall = float(t.item())
        steps = res["step"]
        es = 4 * 7 + 1  # z h n C Rday hmax tmax (f32) + mask per cell
        out["e2e"] = {"value": world * land * steps / wall / 1e9, "unit": "Gcell/s",
                      "h2d_bytes_per_step": es * n * n / max(steps, 1),
                      "d2h_bytes_per_step": 12 * n * n / max(steps, 1),
                      "api": "fca_cuda_run (host buffers)",
                      "run": "config 2, 6 h simulated, without the point inflow (the reference "
                             "ABI has no inflow term)",
                      "steps": steps, "wall_s": wall, "timed_runs": 3,
                      "wall_s_each": walls, "statistic": "median", "rc": rc,
                      "E_mass": e2e_mass_error(res),
                      "t_h2d_s": g.tm.t_h2d, "t_d2h_s": g.tm.t_d2h}
    if not args.no_ensemble:
        out["ensemble"] = ensemble_leg(args.math)
    clk.__exit__(None, None, None)
    out["clocks"] = clk.summary()
    out["clocks"]["span"] = "warm-up, timed steps, end-to-end and ensemble legs"
    if rank == 0 and world == 1 and not args.no_cpu:
        # the same step and warm-up counts as the reference arm
        r = reference_cpu(dom, p, args.steps, args.warmup, args.cpu_budget)
        if "unavailable" not in r:
            out["cpu_baseline"] = {"value": r["value"], "unit": "Gcell/s", "cores": r["cores"],
                                   "kind": r["kind"], "sample": r["sample"]}
        else:
            out["cpu_baseline"] = r
    if world > 1:
        dist.destroy_process_group()
    if rank == 0:
        print(json.dumps(out), flush=True)
    return 0


if __name__ == "__main__":
    sys.exit(main())
