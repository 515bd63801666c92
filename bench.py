#!/usr/bin/env python
"""Throughput benchmark: 6-max 100BB MCCFR traversals/s on one or more B200s.

Contract: `python bench.py --gpus N --steps K --warmup W [--impl reference]`
prints ONE JSON line on rank 0.  A step is one training iteration of the
workload: N_players player-updates of `batch` traversals each (2^20 for the
6-max 100BB configuration).  `value` is whole-job traversals/s timed with CUDA
events on the trainer's stream over exactly K steps, max over ranks; `e2e` is the
same metric through the C-ABI train call from the host, host<->device copies
included.  Several GPUs run independent replicas (the trainer keeps one
device-resident table per GPU, no collective), so scaling is weak.

--impl reference times the reference path's CPU implementation (the C++
restatement of the reference traversal in oracle/, all host threads) on the
same workload, on rank 0 only.
"""
from __future__ import annotations

import argparse
import csv
import io
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WORKLOADS = {
    # name: (preset, overrides, traversals per player-update)
    "6max-100bb": ("PRESET_6MAX_100BB", {}, 1 << 20),
    "6max-100bb-refrule": ("PRESET_6MAX_100BB", {"sampling": 0, "max_depth": 64}, 1 << 20),
    "hu-20bb": ("PRESET_HU_20BB", {}, 1 << 16),
    "hu-20bb-refrule": ("PRESET_HU_20BB", {"sampling": 0}, 1 << 16),
    "ref8-6max": ("PRESET_REF8", {"num_players": 6, "table_log2": 27}, 1 << 18),
    "ref8-hu": ("PRESET_REF8", {"table_log2": 27}, 1 << 16),
}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--workload", choices=sorted(WORKLOADS), default="6max-100bb")
    ap.add_argument("--batch", type=int, default=0, help="traversals per player-update (0 = workload default)")
    ap.add_argument("--no-extras", action="store_true", help="skip the secondary measurements")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--table-log2", type=int, default=0, help="override the table capacity (profiling cases)")
    ap.add_argument("--key-bits", type=int, default=-1, help="override the hashed key width (profiling cases)")
    ap.add_argument("--hu-exploitability", type=int, default=0, metavar="ITERS",
                    help="only: train heads-up 20BB for ITERS iterations with each update rule and print the "
                         "exact best-response exploitability of both (a long run; one JSON line)")
    ap.add_argument("--br-flop-stride", type=int, default=1, help="with --hu-exploitability: flop-class stride")
    ap.add_argument("--curve", type=str, default="", metavar="I1,I2,...",
                    help="only: time single iterations at these points of one training run (one JSON line)")
    ap.add_argument("--form", type=int, default=-1, help="traversal form (0 auto, 1 lanes, 2 levels)")
    ap.add_argument("--c4-only", type=int, default=0, metavar="LOG2_HANDS",
                    help="only: the showdown microbench with 2^LOG2_HANDS 7-card hands and as many 6-seat deals "
                         "(one JSON line; profiling cases)")
    return ap.parse_args()


def make_config(L, workload: str, rank: int = 0):
    preset_name, over, batch = WORKLOADS[workload]
    cfg = L.preset(getattr(L, preset_name))
    for k, v in over.items():
        setattr(cfg, k, v)
    cfg.seed = int(cfg.seed) + rank  # independent replicas
    return cfg, batch


def traversal_form(cfg) -> str:
    """The kernels that a config's updates run: the default form walks while a path
    holds at most 31 decisions of the updating player (raise_cap + 1 per street, or
    the depth cut's nodes), and takes the level kernels for longer ones."""
    if cfg.sampling != 1:
        return "reference"
    if cfg.traversal_form == 0:
        decisions = min(cfg.max_depth, 4 * (cfg.raise_cap + 1)) if cfg.raise_cap > 0 else cfg.max_depth
        return "walk" if decisions < 32 else "levels"
    return "lanes" if cfg.traversal_form == 1 else "levels"


def apply_roofline(s0, s1, launches: int, peak: float, row_bytes: float = 420.0, wide_bytes: float = 96.0,
                   last: bool = False) -> dict:
    """The apply kernel's share of a step against the HBM roofline, at `row_bytes`
    per touched row and `wide_bytes` more per row whose second line was folded; rows
    counted on the device for the last player-update, over the mean time of a launch
    or, with `last`, the time of that update's own.  The defaults are a whole
    256-byte record read, 160 bytes of it written and a 4-byte list entry, plus 96
    bytes of accumulators."""
    ms = s1.last_apply_ms if last else (s1.apply_ms - s0.apply_ms) / max(1, launches)
    rows = int(s1.touched_last)
    wide = int(getattr(s1, "wide_rows_last", 0))
    nbytes = rows * row_bytes + wide * wide_bytes
    gbs = nbytes / (ms / 1e3) / 1e9 if ms > 0 else None
    return {"kernel": "k_apply", "kernel_ms_per_launch": ms, "touched_rows_last_update": rows,
            "wide_rows_last_update": wide, "bytes_per_launch": nbytes,
            "bytes_per_row": f"{row_bytes:.0f} + {wide_bytes:.0f} for rows whose second line was folded",
            "achieved": gbs, "unit": "GB/s", "frac": gbs / peak if gbs else None}


def over_ranks(ms: float, traversals: int, e2e_s: float, device) -> tuple[float, float, float]:
    """Whole-job figures from one replica's own: the slowest rank's device time
    and end-to-end wall time (MAX) and the traversals of all ranks (SUM).  With one
    rank, or no process group, a rank's own figures come back unchanged; several
    ranks all take the same two all-reduces in the same order."""
    import torch
    import torch.distributed as dist

    if not (dist.is_available() and dist.is_initialized()) or dist.get_world_size() == 1:
        return float(ms), float(traversals), float(e2e_s)
    t = torch.tensor([ms, e2e_s], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    n = torch.tensor([float(traversals)], dtype=torch.float64, device=device)
    dist.all_reduce(n, op=dist.ReduceOp.SUM)
    return float(t[0].item()), float(n[0].item()), float(t[1].item())


def describe(cfg, workload, batch) -> dict:
    kinds = {0: "fold", 1: "check", 2: "call", 3: "check/call", 4: "min-raise", 6: "all-in"}
    acts = []
    for a in range(cfg.num_actions):
        k = cfg.action_kind[a]
        acts.append(f"{cfg.action_num[a]}/{cfg.action_den[a]}pot" if k == 5 else kinds[k])
    return {
        "workload": workload,
        "players": cfg.num_players,
        "stack_bb": cfg.starting_stack / cfg.big_blind,
        "blinds": f"{cfg.small_blind}/{cfg.big_blind} chips",
        "actions": acts,
        "raise_cap": cfg.raise_cap,
        "buckets": [cfg.preflop_buckets, *cfg.postflop_buckets],
        "sampling": "external" if cfg.sampling == 1 else "reference (outcome at the updating player)",
        "table_rows": 1 << cfg.table_log2,
        "key_bits": cfg.key_bits if cfg.key_mode == 1 else 26,
        "traversals_per_update": batch,
        "seed": int(cfg.seed),
        "global_batch": batch * cfg.num_players,
        "l2": "working set > L2: 130 MB rank table + info-set table of several GB, no flush needed",
    }


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.out = ""

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.out, _ = self.proc.communicate(timeout=5)
            except Exception:
                self.proc.kill()
                self.out = ""

    def summary(self) -> dict:
        rows = [r for r in csv.reader(io.StringIO(self.out)) if len(r) >= 9]
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        smax = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].strip().lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": reasons, "samples": len(rows),
                "power_w_max": max((float(r[3]) for r in rows if r[3].strip().replace(".", "").isdigit()),
                                   default=None)}


def measured_peak() -> tuple[float, str]:
    p = ROOT / "MEASURED_PEAKS.json"
    try:
        return float(json.loads(p.read_text())["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def profiled_traffic(workload: str, form: str) -> dict | None:
    """DRAM bytes of the traversal kernels from a committed ncu summary
    (profiles/traffic.json, keyed "workload/form"), if one exists."""
    p = ROOT / "profiles" / "traffic.json"
    try:
        return json.loads(p.read_text()).get(f"{workload}/{form}")
    except Exception:
        return None


def _binding():
    sys.path.insert(0, str(ROOT / "oracle"))
    import binding

    return binding


def cpu_equal_work(rows: dict, cfg, iterations_done: int, batch: int, table, sample: int) -> dict:
    """The oracle (the reference path's C++ restatement) on all host cores, on
    exactly the trees the device walks next: the device's rows after
    `iterations_done` iterations are loaded into the oracle, which then runs
    traversals 0..sample-1 of update (iterations_done + 1, player 0), the same
    deals, draws and table reads as the device's first `sample` traversals of that
    update.  Returns traversals/s with the work per traversal it saw."""
    binding = _binding()
    threads = os.cpu_count() or 1
    orc = binding.Oracle(cfg, table)
    t0 = time.perf_counter()
    orc.import_rows(rows, iterations_done)
    load_s = time.perf_counter() - t0
    t0 = time.perf_counter()
    orc.step(iterations_done + 1, 0, sample, threads=threads)
    dt = time.perf_counter() - t0
    c = orc.counters()
    orc.close()
    return {"value": sample / dt, "unit": "traversals/s", "cores": threads, "kind": "port",
            "seconds": dt, "rows_loaded": int(rows["keys"].size), "load_seconds": load_s,
            "V_per_traversal": c["visits"] / sample, "U_per_traversal": c["updates"] / sample,
            "sample": (f"traversals 0..{sample - 1} of update (iteration {iterations_done + 1}, player 0) of the "
                       f"{batch}-traversal workload, on the device's {int(rows['keys'].size)} rows after iteration "
                       f"{iterations_done} loaded into the oracle: the trees the device walks next "
                       f"({c['visits'] / sample:.1f} node visits per traversal), {dt:.1f} s on {threads} threads, "
                       "update and fold included")}


# Traversals per player-update of the reference arm's own training run: a batch
# the CPU port trains through in seconds per iteration on the host's cores.
REFERENCE_ARM_BATCH = {"6max-100bb": 4096, "6max-100bb-refrule": 65536, "hu-20bb": 16384, "hu-20bb-refrule": 65536,
                       "ref8-6max": 65536, "ref8-hu": 65536}


def repo_libraries() -> list[str]:
    """Shared libraries of this repository mapped into the process
    (/proc/self/maps), relative to the repository root."""
    out = set()
    try:
        for line in Path("/proc/self/maps").read_text().splitlines():
            parts = line.split()
            if len(parts) >= 6 and parts[-1].endswith(".so") and parts[-1].startswith(str(ROOT)):
                out.add(os.path.relpath(parts[-1], ROOT))
    except OSError:
        pass
    return sorted(out)


def reference_arm(args, workload: str, world: int) -> dict:
    """The reference path's CPU implementation (the oracle, all host threads)
    training the workload's game from an empty table by itself: W iterations,
    then K timed iterations, each of N player-updates of a bounded batch.  It
    loads no device library: presets and the rank table come from the oracle."""
    import importlib

    binding = _binding()
    L = importlib.import_module("mccfr_b200.lib")  # struct definitions only; libmccfr.so is not loaded
    preset_name, over, batch = WORKLOADS[workload]
    cfg = binding.config_init(L.Config(), getattr(L, preset_name))
    for k, v in over.items():
        setattr(cfg, k, v)
    if args.table_log2:
        cfg.table_log2 = args.table_log2
    if args.key_bits >= 0:
        cfg.key_bits = args.key_bits
    b = args.batch or REFERENCE_ARM_BATCH.get(workload, 4096)
    threads = os.cpu_count() or 1
    table = binding.hand_table()
    orc = binding.Oracle(cfg, table)
    orc.train(args.warmup, b, threads=threads)
    c0 = orc.counters()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        orc.train(1, b, threads=threads)
    secs = time.perf_counter() - t0
    c1 = orc.counters()
    orc.close()
    trav = c1["traversals"] - c0["traversals"]
    v = trav / secs
    vpt = (c1["visits"] - c0["visits"]) / max(1, trav)
    upt = (c1["updates"] - c0["updates"]) / max(1, trav)
    metric = "6-max traversals/s" if cfg.num_players == 6 else "traversals/s"
    sample = (f"the oracle training the workload's game by itself from an empty table on {threads} threads: "
              f"{args.warmup} warm-up iterations, then {args.steps} timed iterations of {cfg.num_players} "
              f"player-updates x {b} traversals (iterations {args.warmup + 1}-{args.warmup + args.steps}); "
              f"{vpt:.1f} node visits and {upt:.2f} updating-player updates per traversal. Its trees are those "
              f"of a {b}-traversal run, larger than the device's at {batch} traversals per update (the device "
              "line's cpu_baseline times the oracle on the device's own trees)")
    return {
        "impl": "reference", "metric": metric, "value": v, "unit": "traversals/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": secs * 1e3 / max(1, args.steps),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {**describe(cfg, workload, batch), "parallelism": f"replicas{world}"},
        "cpu_baseline": {"value": v, "unit": "traversals/s", "cores": threads, "kind": "port", "sample": sample,
                         "V_per_traversal": vpt, "U_per_traversal": upt, "traversals_per_update": b},
        "e2e": {"value": v, "unit": "traversals/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "libraries_loaded": repo_libraries(),
    }


def iteration_curve(m, L, table, cfg, batch: int, points: list[int]) -> dict:
    """Traversals/s and work per traversal of single iterations along one
    training run of a fresh table: iteration i is timed alone (CUDA events on
    the trainer's stream) after iterations 1..i-1 ran untimed."""
    import torch

    tr = m.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(table)
    stream = torch.cuda.ExternalStream(tr.stream_ptr())
    out, done = [], 0
    t_start = time.perf_counter()
    for it in sorted(set(points)):
        if it - 1 > done:
            tr.train(it - 1 - done, batch, verbose=False)
            done = it - 1
        s0 = tr.stats()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        tr.train(1, batch, verbose=False, timed=True)
        e1.record(stream)
        e1.synchronize()
        done = it
        s1 = tr.stats()
        ms = e0.elapsed_time(e1)
        n = s1.traversals - s0.traversals
        out.append({"iteration": it, "traversals_per_s": n / (ms / 1e3), "ms": ms,
                    "V_per_traversal": (s1.node_visits - s0.node_visits) / n,
                    "U_per_traversal": (s1.traverser_updates - s0.traverser_updates) / n,
                    "traverse_ms_per_update": (s1.traverse_ms - s0.traverse_ms) / cfg.num_players,
                    "apply_ms_per_update": (s1.apply_ms - s0.apply_ms) / cfg.num_players,
                    "touched_rows_last_update": int(s1.touched_last)})
    tr.close()
    return {"points": out, "wall_s": time.perf_counter() - t_start, "traversals_per_update": batch,
            "form": int(cfg.traversal_form)}


def batched_same_table(m, L, table, args, plain_value) -> dict:
    """The headline 6-max table trained through the batched persistent form.
    The tuning is chosen on a scratch copy of the table; a fresh table then runs
    the same warm-up and timed iterations as the headline, so both time the
    same trees."""
    cfg, batch = make_config(L, args.workload)
    if args.batch:
        batch = args.batch
    scratch = m.GPUCFRTrainer(config=cfg)
    scratch.set_hand_table(table)
    sb = m.Batch([scratch], [batch])
    best = sb.autotune(max_candidates=16)
    sb.close()
    scratch.close()
    t = m.GPUCFRTrainer(config=cfg)
    t.set_hand_table(table)
    b = m.Batch([t], [batch])
    b.set_tuning(**best)
    b.train(args.warmup)
    s0 = b.stats()
    b.train(args.steps, timed=True)
    s1 = b.stats()
    n = s1.traversals - s0.traversals
    ms = s1.total_ms - s0.total_ms
    b.close()
    t.close()
    v = n / (ms / 1e3)
    return {"traversals_per_s": v, "vs_plain": v / plain_value, "tuning": best, "iterations": args.steps,
            "traverse_ms_per_iteration": (s1.traverse_ms - s0.traverse_ms) / args.steps,
            "note": "same table, seed, traversals per update and iterations as the headline; results are "
                    "bit-identical to plain training (tests/test_gpu_batched.py)"}


ACTION_SETS = {
    3: [(0, 0, 1), (3, 0, 1), (6, 0, 1)],
    4: [(0, 0, 1), (3, 0, 1), (5, 1, 1), (6, 0, 1)],
    5: [(0, 0, 1), (3, 0, 1), (5, 1, 2), (5, 1, 1), (6, 0, 1)],
    6: [(0, 0, 1), (3, 0, 1), (5, 1, 2), (5, 1, 1), (5, 2, 1), (6, 0, 1)],
}


def multitable_configs(L, n_tables=64, seed=2, scale=16):
    """Uneven tables: players U{2..6}, stacks U[10,200] BB, 3-6 actions, traversals
    per update round(LogNormal(14, 1)) / scale."""
    import numpy as np

    rng = np.random.default_rng(seed)
    out = []
    for i in range(n_tables):
        c = L.preset(L.PRESET_HU_20BB)
        c.num_players = int(rng.integers(2, 7))
        c.starting_stack = int(rng.integers(10, 201)) * c.big_blind
        na = int(rng.choice([3, 4, 5, 6]))
        c.num_actions = na
        for a, (k, num, den) in enumerate(ACTION_SETS[na]):
            c.action_kind[a], c.action_num[a], c.action_den[a] = k, num, den
        c.raise_cap = 3
        c.table_log2 = 22
        c.key_bits = 21
        c.seed = 1000 + i
        n = max(1024, int(round(rng.lognormal(14.0, 1.0) / scale)))
        out.append((c, n))
    return out


def time_table_graphs(m, L, make, counts, iters) -> float:
    """Wall-clock seconds of `iters` iterations of a fresh set of tables trained
    as one batch in the table-graph form (every table's own update kernels as a
    concurrent branch of one graph per iteration), after one untimed iteration."""
    import torch

    ts = make()
    g = m.Batch(ts, counts)
    g.set_tuning(form=L.BATCH_TABLE_GRAPHS)
    g.train(1)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    g.train(iters)
    torch.cuda.synchronize()
    secs = time.perf_counter() - t0
    g.close()
    for t in ts:
        t.close()
    return secs


def multitable(m, L, table, iters=2) -> dict:
    import torch

    specs = multitable_configs(L)
    def make():
        ts = []
        for c, _ in specs:
            t = m.GPUCFRTrainer(config=c)
            t.set_hand_table(table)
            ts.append(t)
        return ts
    # plain: each table's iteration on its own, one after another
    plain = make()
    for t, (c, n) in zip(plain, specs):
        t.train(1, n, verbose=False)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(iters):
        for t, (c, n) in zip(plain, specs):
            t.train(1, n, verbose=False)
    torch.cuda.synchronize()
    plain_s = time.perf_counter() - t0
    for t in plain:
        t.close()
    # tuning chosen on scratch tables; fresh tables then time the same iterations as plain
    scratch = make()
    sb = m.Batch(scratch, [n for _, n in specs])
    best = sb.autotune(max_candidates=16)
    sb.close()
    for t in scratch:
        t.close()
    batched = make()
    b = m.Batch(batched, [n for _, n in specs])
    b.set_tuning(**best)
    b.train(1)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    b.train(iters)
    torch.cuda.synchronize()
    batched_s = time.perf_counter() - t0
    b.close()
    for t in batched:
        t.close()
    graphs_s = time_table_graphs(m, L, make, [n for _, n in specs], iters)
    trav = iters * sum(n * c.num_players for c, n in specs)
    return {"tables": len(specs), "traversals_per_iteration": trav // iters,
            "plain_traversals_per_s": trav / plain_s, "batched_traversals_per_s": trav / batched_s,
            "speedup": plain_s / batched_s, "tuning": best,
            "table_graphs_traversals_per_s": trav / graphs_s, "table_graphs_speedup": plain_s / graphs_s,
            "workload": "64 tables, players U{2..6}, stacks U[10,200]BB, 3-6 actions, traversals/update "
                        "LogNormal(14,1)/16, seed 2; wall clock over iterations 2-3 of fresh tables; plain "
                        "(table after table), batched (one persistent launch per phase, autotuned) and "
                        "table_graphs (every table's own kernels as concurrent branches of one graph)"}


def batched_small_tables(m, L, table, n_tables=64, batch=4096, iters=3) -> dict:
    """The regime a multi-table kernel is for: 64 independent 6-max 100BB tables
    (2^20-row tables, 20-bit keys, seeds 100..163) of 4,096 traversals per
    player-update each.  Plain: every table's iteration on its own (one graph
    replay each), one table after another;
    batched: all 64 in one persistent traversal launch per phase; table graphs:
    every table's own update kernels as concurrent branches of one graph per
    iteration.  All over the same iterations of fresh tables, wall clock; rows
    are bit-identical between the forms (tests/test_gpu_batched.py)."""
    import torch

    def make():
        ts = []
        for i in range(n_tables):
            c = L.preset(L.PRESET_6MAX_100BB)
            c.table_log2, c.key_bits, c.seed = 20, 20, 100 + i
            t = m.GPUCFRTrainer(config=c)
            t.set_hand_table(table)
            ts.append(t)
        return ts

    plain = make()
    for t in plain:
        t.train(1, batch, verbose=False)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(iters):
        for t in plain:
            t.train(1, batch, verbose=False)
    torch.cuda.synchronize()
    plain_s = time.perf_counter() - t0
    for t in plain:
        t.close()
    scratch = make()
    sb = m.Batch(scratch, [batch] * n_tables)
    best = sb.autotune(max_candidates=16)
    sb.close()
    for t in scratch:
        t.close()
    batched = make()
    b = m.Batch(batched, [batch] * n_tables)
    b.set_tuning(**best)
    b.train(1)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    b.train(iters)
    torch.cuda.synchronize()
    batched_s = time.perf_counter() - t0
    b.close()
    for t in batched:
        t.close()
    graphs_s = time_table_graphs(m, L, make, [batch] * n_tables, iters)
    trav = iters * n_tables * batch * 6
    return {"tables": n_tables, "traversals_per_update": batch, "iterations": iters,
            "plain_traversals_per_s": trav / plain_s, "batched_traversals_per_s": trav / batched_s,
            "speedup": plain_s / batched_s, "tuning": best,
            "table_graphs_traversals_per_s": trav / graphs_s, "table_graphs_speedup": plain_s / graphs_s,
            "workload": "64 tables of 6-max 100BB, 4,096 traversals per player-update each, iterations 2-4 of "
                        "fresh tables, wall clock; plain, batched (persistent) and table_graphs forms"}


def serving_sweep(m, L, table, rates=(10, 30, 100, 300, 1000), n_requests=48) -> dict:
    """Re-solve serving at several Poisson arrival rates: p50/p99 latency (arrival
    to strategy on the host) and solves/s, continuous batching on one B200."""
    import importlib

    import numpy as np

    sv = importlib.import_module("mccfr_b200.serving")
    owner = m.GPUCFRTrainer(config=L.preset(L.PRESET_HU_20BB), table_log2=10)
    owner.set_hand_table(table)
    out = {}
    for rate in rates:
        rng = np.random.default_rng(4)
        reqs = [sv.make_request(rng, i) for i in range(n_requests)]
        for r, a in zip(reqs, sv.poisson_arrivals(rng, n_requests, rate)):
            r.arrival = float(a)
        srv = sv.ReSolveServer(owner, hbm_budget=32 << 30, traversals=1024, retire_workers=2)
        res = srv.run(reqs)
        line = {**sv.summarize(res), "rounds": srv.rounds, "tables_reused": srv.reused,
                **{k: round(v, 3) for k, v in srv.timing.items()}}
        srv.close()
        # the same trace on the plain trainer, one request at a time; equal strategies
        plain = sv.serve_plain(owner, reqs, traversals=1024)
        by_rid = {r.rid: r for r in res}
        same = sum(1 for r in plain if np.array_equal(r.keys, by_rid[r.rid].keys)
                   and np.array_equal(r.probs.view(np.uint32), by_rid[r.rid].probs.view(np.uint32)))
        line["plain_trainer"] = {**sv.summarize(plain), "strategies_bit_identical": f"{same}/{len(plain)}"}
        out[f"lambda_{rate}"] = line
    owner.close()
    out["workload"] = (f"{n_requests} requests per rate: turn/river board, 2-6 players, pot U[2,200]BB, "
                       "Dirichlet(0.5) ranges, 3-6 sizes drawn (at most 5 kept: fold, check/call, the sizes and "
                       "all-in fill the 8 action slots of a row) + all-in, 100BB stacks, seed 4. Budget unit: "
                       "iterations of the one-traversal-per-player form, log-uniform [2e3,5e4] = traversals per "
                       "player, spent 1024 per player-update; strategies exported by 2 retire workers beside the "
                       "rounds. plain_trainer: the same trace served one request at a time by train() in arrival "
                       "order")
    return out


def hu_subgame_exploitability(m, L, table, checkpoints=(10, 40, 160, 640), batch=2048) -> dict:
    """Exact FP64 best response of a heads-up river re-solve trained on the GPU
    by each update rule, at equal iterations (mccfr_exploitability)."""
    import numpy as np

    rng = np.random.default_rng(12)
    board = [int(c) for c in rng.permutation(52)[:5]]
    cards = np.array([(lo, hi) for hi in range(1, 52) for lo in range(hi)])
    blocked = np.isin(cards, board).any(axis=1)
    ranges = np.zeros((2, 1326))
    for p in range(2):
        idx = rng.permutation(np.flatnonzero(~blocked))[:200]
        ranges[p, idx] = rng.dirichlet(np.full(200, 1.0))
    ranges = ranges.astype(np.float32)
    owner = m.GPUCFRTrainer(config=L.preset(L.PRESET_HU_20BB), table_log2=10)
    owner.set_hand_table(table)
    out = {}
    for name, sampling in (("external", L.SAMPLING_EXTERNAL), ("reference_rule", L.SAMPLING_REFERENCE)):
        c = L.preset(L.PRESET_HU_20BB)
        c.starting_stack = 10000
        slots = [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_RAISE_POT, 1, 2), (L.ACT_RAISE_POT, 1, 1),
                 (L.ACT_ALL_IN, 0, 1)]
        c.num_actions = len(slots)
        for a, (k, n, d) in enumerate(slots):
            c.action_kind[a], c.action_num[a], c.action_den[a] = k, n, d
        c.raise_cap, c.max_depth, c.table_log2, c.key_bits, c.sampling = 2, 255, 18, 17, sampling
        tr = m.GPUCFRTrainer.subgame(c, 3, 1200, board, ranges)
        tr.share_hand_table(owner)
        done, curve = 0, []
        for k in checkpoints:
            tr.train(k - done, batch, verbose=False)
            done = k
            e = tr.exploitability()
            curve.append({"iterations": k, "mbb_per_game": e["mbb_per_game"], "br_seconds": round(e["seconds"], 3)})
        out[name] = curve
        tr.close()
    owner.close()
    out["workload"] = (f"heads-up river subgame, 100BB stacks, pot 12BB, 200-combo Dirichlet(1) ranges (seed 12), "
                       f"{{fold, check/call, 1/2 pot, pot, all-in}}, raise cap 2, {batch} traversals per update; "
                       "exact FP64 best response (mccfr_exploitability)")
    return out


# Exact counts of the 9 categories over all 133,784,560 seven-card hands, and
# the first rank of each category on the 1..7462 scale.
SEVEN_CARD_CATEGORIES = [23294460, 58627800, 31433400, 6461620, 6180020, 4047644, 3473184, 224848, 41584]
CATEGORY_START = [1, 1278, 4138, 4996, 5854, 5864, 7141, 7297, 7453, 7463]


def c4_showdown(m, L, table, total=1 << 28, chunk=1 << 24, deals6=1 << 24) -> dict:
    """Showdown microbench, both parts seeded by Philox seed 3 on the device.
    7-card: `total` uniform 7-card hands (mccfr_deal_eval7: drawn and ranked in
    one kernel, 7 dependent gathers = 28 B of rank-table reads per hand); the
    category frequencies are checked against the exact counts.  6-seat:
    `deals6` deals of training's 6-player deal (update 1, player 0) with the
    board walked once for all seats (mccfr_showdown_masks: 5 + 2 x 6 gathers =
    68 B per deal) and 6-bit winner masks; seat symmetry and the split rate are
    checked.  Kernel time from the library's CUDA events."""
    import ctypes

    import numpy as np
    import torch

    lib = L.load()
    peak, kind = measured_peak()
    cfg = L.preset(L.PRESET_6MAX_100BB)
    cfg.seed, cfg.table_log2 = 3, 10
    t = m.GPUCFRTrainer(config=cfg)
    t.set_hand_table(table)
    ranks = torch.empty(chunk, dtype=torch.int16, device="cuda")
    hist = torch.zeros(7463, dtype=torch.int64, device="cuda")
    ms_total = 0.0
    torch.cuda.synchronize()
    for stream in range(total // chunk):
        ms = ctypes.c_float()
        L.check(lib.mccfr_deal_eval7(t.handle, stream, chunk, ctypes.c_void_p(ranks.data_ptr()), ctypes.byref(ms)))
        ms_total += ms.value
        hist += torch.bincount(ranks.to(torch.int64) & 0xFFFF, minlength=7463)[:7463]
    h = hist.cpu().numpy()
    n = (total // chunk) * chunk
    obs = np.array([h[CATEGORY_START[i]:CATEGORY_START[i + 1]].sum() for i in range(9)], dtype=np.float64)
    p = np.array(SEVEN_CARD_CATEGORIES, dtype=np.float64) / 133784560.0
    z = (obs / n - p) / np.sqrt(p * (1 - p) / n)
    evals = n / (ms_total / 1e3)
    # 6-seat shared-board showdown of training's deals
    masks = torch.empty(deals6, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ms6 = ctypes.c_float()
    L.check(lib.mccfr_showdown_masks(t.handle, 1, 0, deals6, ctypes.c_void_p(masks.data_ptr()), ctypes.byref(ms6)))
    mk = masks.to(torch.int64)
    wins = [int(((mk >> q) & 1).sum().item()) for q in range(6)]
    pop = sum(((mk >> q) & 1) for q in range(6))
    split = float((pop > 1).double().mean().item())
    bad = int(((mk == 0) | (mk >= 64)).sum().item())
    t.close()
    deals_s = deals6 / (ms6.value / 1e3)
    return {"hands": n, "hand_evals_per_s": evals, "kernel_ms": ms_total,
            "gather_gbs": 28.0 * evals / 1e9, "gather_frac_of_hbm_peak": 28.0 * evals / 1e9 / peak,
            "category_max_abs_z": float(np.abs(z).max()), "invalid_ranks": int(h[0]),
            "six_seat": {"deals": deals6, "kernel_ms": ms6.value, "deals_per_s": deals_s,
                         "hand_evals_per_s": 6 * deals_s, "gather_gbs": 68.0 * deals_s / 1e9,
                         "seat_wins": wins, "split_rate": split, "invalid_masks": bad},
            "workload": "Philox seed 3 on the device. 7-card: 2^28 hands in 16 calls of 2^24 (stream = call "
                        "index), k_deal_eval7 draws and ranks each hand (7 dependent gathers into the 130 MB rank "
                        "table). 6-seat: 2^24 deals of training's 6-player deal (iteration 1, player 0), "
                        "k_showdown_masks (board walked once, 2 gathers per seat, winner/split mask per deal); "
                        "both bit-exact with the oracle in tests/test_gpu_showdown.py"}


def reference_gpu(m, L, table, iters: int = 20) -> dict:
    """The reference's own GPU trainer (poker_cuda/src/cfr_gpu.cu compiled
    unchanged for sm_100a, oracle/_ref/libref_gpu.so) on this box, in a child
    process, beside this trainer's reference rule on the same game: the
    reference's benchmark configurations (main.cpp:380-398; players and blinds of
    scripts/carc_train.sh:75-80), `iters` iterations from a fresh trainer.  Its
    own figure is the rate its training loop prints (cfr_gpu.cu:1368-1377,
    after allocation and graph capture); ours is CUDA-event time of the same
    iterations after the same start."""
    import re
    import tempfile

    import torch

    lib_path = ROOT / "oracle" / "_ref" / "libref_gpu.so"
    if not lib_path.exists():
        return {"unavailable": "the reference's GPU trainer was not built (its sources were absent at build time)"}
    out = {}
    with tempfile.TemporaryDirectory() as d:
        table_file = Path(d) / "handranks.dat"
        table.tofile(table_file)
        for players, batch in ((6, 262144), (6, 65536), (2, 65536)):
            r = subprocess.run([sys.executable, str(ROOT / "oracle" / "ref_gpu_run.py"), "time", str(players),
                                str(iters), str(batch), str(table_file)], capture_output=True, text=True, timeout=900)
            line = {"returncode": r.returncode}
            mdone = re.search(r"\(([\d.]+)M hands/sec\)", r.stdout)
            if mdone:
                line["reference_loop_traversals_per_s"] = float(mdone.group(1)) * 1e6
            for ln in r.stdout.splitlines():
                if ln.startswith("{"):
                    line["reference_benchmark_mode_traversals_per_s"] = json.loads(ln)["traversals_per_s"]
            cfg = L.preset(L.PRESET_REF8)
            cfg.num_players = players
            t = m.GPUCFRTrainer(config=cfg)
            t.set_hand_table(table)
            t.train(1, batch, verbose=False)  # graph capture, as the reference's loop figure excludes it
            st = torch.cuda.ExternalStream(t.stream_ptr())
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            t.train(iters - 1, batch, verbose=False)
            e1.record(st)
            e1.synchronize()
            t.close()
            ours = (iters - 1) * batch * players / (e0.elapsed_time(e1) / 1e3)
            line["ours_traversals_per_s"] = ours
            if "reference_loop_traversals_per_s" in line:
                line["ours_over_reference"] = ours / line["reference_loop_traversals_per_s"]
            out[f"{players}p_batch{batch}"] = line
    out["workload"] = (f"the reference's game: stack 1000, blinds 10/20, 8 action slots, 64/128 buckets, its update "
                       f"rule (outcome sampling at the updating player), {iters} iterations of a fresh trainer")
    return out


def hu_full_exploitability(m, L, table, iters: int, stride: int) -> dict:
    """Heads-up 20BB from the blinds: both update rules trained for `iters`
    iterations of 65,536 traversals per player-update, then the exact best
    response of each average strategy (all 1,755 flop classes unless a stride
    is given)."""
    out = {"iterations": iters, "traversals_per_update": 1 << 16, "flop_stride": stride}
    for wl in ("hu-20bb", "hu-20bb-refrule"):
        cfg, batch = make_config(L, wl)
        tr = m.GPUCFRTrainer(config=cfg)
        tr.set_hand_table(table)
        t0 = time.perf_counter()
        tr.train(iters, batch, verbose=False)
        st = tr.stats()
        train_s = time.perf_counter() - t0
        e = tr.exploitability(flop_stride=stride, verbose=True)
        out[wl] = {"train_seconds": train_s, "traversals": st.traversals, "rows_used": st.rows_used,
                   "traversals_per_s": st.traversals / train_s, **e}
        tr.close()
        print(json.dumps({wl: out[wl]}), file=sys.stderr, flush=True)
    a, b = out["hu-20bb"]["mbb_per_game"], out["hu-20bb-refrule"]["mbb_per_game"]
    out["external_over_reference_rule"] = a / b
    return out


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    import __graft_entry__ as ge

    if args.impl == "reference":
        if rank != 0:
            return
        # the checker libraries only: this arm loads no product library
        ge._build_module().build_oracle()
        ge.load_package()
        print(json.dumps(reference_arm(args, args.workload, world)), flush=True)
        return

    ge.build()
    m = ge.load_package()
    L = m.lib
    cfg, batch = make_config(L, args.workload, rank)
    if args.batch:
        batch = args.batch
    if args.table_log2:
        cfg.table_log2 = args.table_log2
    if args.key_bits >= 0:
        cfg.key_bits = args.key_bits
    if args.form >= 0:
        cfg.traversal_form = args.form
    metric = "6-max traversals/s" if cfg.num_players == 6 else "traversals/s"

    import torch
    import torch.distributed as dist

    torch.cuda.set_device(local_rank)
    if world > 1:
        backend = "nccl" if torch.cuda.is_available() else "gloo"
        from datetime import timedelta
        dist.init_process_group(backend, timeout=timedelta(seconds=300))
    cfg.device = local_rank
    table = L.hand_table()
    if args.c4_only:
        if rank == 0:
            n = 1 << args.c4_only
            print(json.dumps({"c4_showdown": c4_showdown(m, L, table, total=n, chunk=min(n, 1 << 24), deals6=n)}),
                  flush=True)
        return
    if args.curve:
        if rank == 0:
            pts = [int(x) for x in args.curve.split(",") if x.strip()]
            print(json.dumps({"workload": args.workload, **iteration_curve(m, L, table, cfg, batch, pts)}),
                  flush=True)
        return
    if args.hu_exploitability:
        if rank == 0:
            print(json.dumps(hu_full_exploitability(m, L, table, args.hu_exploitability, args.br_flop_stride)),
                  flush=True)
        return
    tr = m.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(table)

    # warm-up (graph capture happens here)
    tr.train(args.warmup, batch, verbose=False)
    s0 = tr.stats()
    stream = torch.cuda.ExternalStream(tr.stream_ptr(), device=local_rank)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local_rank) as clocks:
        ev0.record(stream)
        tr.train(args.steps, batch, verbose=False, timed=True)
        ev1.record(stream)
        ev1.synchronize()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    s1 = tr.stats()
    ms = ev0.elapsed_time(ev1)
    trav = s1.traversals - s0.traversals
    visits = s1.node_visits - s0.node_visits
    updates = s1.traverser_updates - s0.traverser_updates
    launches = args.steps * cfg.num_players
    trav_ms = s1.traverse_ms - s0.traverse_ms

    levels = None
    if cfg.sampling == 1 and cfg.traversal_form != 1:
        try:
            levels = tr.level_counts()
        except Exception as e:  # noqa: BLE001
            levels = {"error": str(e)}

    # the table after the timed region: the oracle's CPU baseline walks the same
    # trees as the device's next update (taken before the e2e steps run it)
    cpu_rows = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            cpu_rows = tr.export_rows()
        except Exception as e:  # noqa: BLE001
            cpu_rows = e
    cpu_iterations = args.warmup + args.steps

    rows_used = tr.rows_used()
    tr.close()  # frees its HBM for the end-to-end trainer

    # e2e through the C ABI: a fresh trainer of the same config runs the same warm-up
    # untimed, then the timed region's K iterations again, one host call per
    # iteration (schedule H2D inside, stats D2H read): identical work to `value`
    te = m.GPUCFRTrainer(config=cfg)
    te.set_hand_table(table)
    te.train(args.warmup, batch, verbose=False)
    e0 = te.stats()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e2e_steps = max(1, args.steps)
    for _ in range(e2e_steps):
        te.train(1, batch, verbose=False)
        st = te.stats()
    e2e_s = time.perf_counter() - t0
    e2e_same_work = (st.node_visits - e0.node_visits) == visits if args.steps > 0 else None
    te.close()

    ms_max, total, e2e_s_max = over_ranks(ms, trav, e2e_s, f"cuda:{local_rank}")
    value = total / (ms_max / 1e3)
    e2e_value = world * e2e_steps * batch * cfg.num_players / e2e_s_max

    peak, peak_kind = measured_peak()
    bytes_per_launch = (40.0 * visits + 96.0 * updates) / launches
    kernel_ms = trav_ms / launches if trav_ms > 0 else None
    achieved = bytes_per_launch / (kernel_ms / 1e3) / 1e9 if kernel_ms else None
    has_levels = isinstance(levels, dict) and "seeds" in levels
    nlev = len(levels["seeds"]) if has_levels else 0
    form_name = traversal_form(cfg)
    tr_prof = profiled_traffic(args.workload, form_name)
    traffic = None
    if tr_prof and "dram_bytes_per_node_visit" in tr_prof:
        traffic = tr_prof["dram_bytes_per_node_visit"] * (visits / launches)
    elif tr_prof and "dram_bytes_per_traversal" in tr_prof:
        traffic = tr_prof["dram_bytes_per_traversal"] * (trav / launches)
    # traversal and apply per update; one deal per update, or one per iteration when
    # an iteration's deals are few
    deals = 1 if batch * cfg.num_players <= 1 << 18 else cfg.num_players
    traversal_launches = 1
    if form_name == "levels":
        kernel_name = ("k_level_expand + k_level_dfs + k_level_showdown + k_level_back (the traversal of one "
                       "player-update)")
        traversal_launches = 2 * nlev + 1  # nlev expand levels, dfs, showdown, nlev - 1 back levels
    else:
        kernel_name = {"walk": "k_walk", "lanes": "k_traverse_es", "reference": "k_path"}[form_name]
    launches_per_iteration = deals + cfg.num_players * (traversal_launches + 1)

    out = {
        "metric": metric, "value": value, "unit": "traversals/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {**describe(cfg, args.workload, batch), "parallelism": f"replicas{world}"},
        "e2e": {"value": e2e_value, "unit": "traversals/s", "h2d_bytes_per_step": 16,
                "d2h_bytes_per_step": 44,
                "iterations": (f"{args.warmup + 1}-{args.warmup + e2e_steps} of a fresh trainer of the same config "
                               "after the same warm-up: the timed region's iterations, one C-ABI train call each"),
                "same_node_visits_as_timed_region": e2e_same_work},
        "gpu_launches": int(args.steps * launches_per_iteration),
        "clocks": clocks.summary(),
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": (achieved / peak) if achieved else None, "traffic": traffic, "peak_kind": peak_kind,
                     "kernel": kernel_name, "form": form_name,
                     "kernel_ms_per_launch": kernel_ms,
                     "traffic_source": tr_prof.get("source") if tr_prof else None,
                     "algorithmic_bytes": "40*V + 96*U per launch (V node visits, U updating-player updates)",
                     "V_per_traversal": visits / max(1, trav), "U_per_traversal": updates / max(1, trav)},
        # k_apply: a row's first 128-byte line read, its counters and sums written (192 B); for a row of
        # the updating player its accumulators read and zeroed and its regrets and strategy written, but
        # most of them leave the sums as they are (160 more); the strategy weights of off-mask visits
        # read and zeroed (128 more).  The last update's rows over the last update's time.
        "apply": apply_roofline(s0, s1, launches, peak, row_bytes=192.0, wide_bytes=160.0, last=True),
        "table": {"rows_used": rows_used, "capacity": int(s1.table_capacity),
                  "load": rows_used / max(1, s1.table_capacity), "record_bytes": 256,
                  "span_gb": s1.table_capacity * 256 / 1e9},
        "levels_last_update": levels,
        "node_visits_per_s": visits / (ms / 1e3) * world,
        "hand_evals_per_s": (s1.hand_evals - s0.hand_evals) / (ms / 1e3) * world,
    }

    if rank == 0 and world == 1 and not args.no_extras:
        # secondary measurements: one that fails is recorded as its error, the
        # headline figures above are kept either way
        # secondary measurements after a CUDA error would run on a poisoned
        # context: the first such error is recorded and the rest are skipped
        extras = {}
        poisoned = []

        def extra(name, fn):
            if poisoned:
                extras[name] = {"skipped": f"a CUDA error in {poisoned[0]} came first"}
                return
            try:
                extras[name] = fn()
            except Exception as e:  # noqa: BLE001
                extras[name] = {"error": f"{type(e).__name__}: {e}"}
                if getattr(e, "status", None) == 2 or "CUDA" in str(e):
                    poisoned.append(name)

        def refrule_rate(wl):
            c2, b2 = make_config(L, wl)
            t2 = m.GPUCFRTrainer(config=c2)
            try:
                t2.set_hand_table(table)
                t2.train(3, b2, verbose=False)
                a0 = t2.stats()
                st2 = torch.cuda.ExternalStream(t2.stream_ptr(), device=local_rank)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(st2)
                t2.train(5, b2, verbose=False, timed=True)
                e1.record(st2)
                e1.synchronize()
                a1 = t2.stats()
                ms2 = e0.elapsed_time(e1)
                n2 = a1.traversals - a0.traversals
                return {"traversals_per_s": n2 / (ms2 / 1e3), "batch": b2, "iterations": 5,
                        "traverse_kernel_ms": (a1.traverse_ms - a0.traverse_ms) / (5 * c2.num_players),
                        "apply_kernel_ms": (a1.apply_ms - a0.apply_ms) / (5 * c2.num_players)}
            finally:
                t2.close()

        extra("batched_same_table", lambda: batched_same_table(m, L, table, args, value))
        extra("c3_multitable", lambda: multitable(m, L, table))
        extra("batched_small_tables", lambda: batched_small_tables(m, L, table))
        extra("resolve_serving", lambda: serving_sweep(m, L, table))
        extra("hu_subgame_exploitability", lambda: hu_subgame_exploitability(m, L, table))
        extra("c4_showdown", lambda: c4_showdown(m, L, table))
        extra("reference_gpu", lambda: reference_gpu(m, L, table))
        for wl in ("ref8-6max", "6max-100bb-refrule"):
            if wl != args.workload:
                extra(wl, lambda wl=wl: refrule_rate(wl))
        out["extras"] = extras

    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            if isinstance(cpu_rows, Exception):
                raise cpu_rows
            out["cpu_baseline"] = cpu_equal_work(cpu_rows, cfg, cpu_iterations, batch, table,
                                                 min(batch, 1 << 20))
        except Exception as e:  # noqa: BLE001
            out["cpu_baseline"] = {"value": None, "unit": "traversals/s", "error": f"{type(e).__name__}: {e}"}
        cpu_rows = None
    if rank == 0:
        print(json.dumps(out), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
