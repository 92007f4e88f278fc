#!/usr/bin/env python
"""Benchmark: full length-2 enumeration of the 6502 superoptimizer on B200.

One step = one pass of the equivalence-checking path over the whole
length-2 workload: all 7,633,612 pruned length-2 targets x all 2,863
length-1 candidates (21,855,031,156 pair-checks) through QuickCheck ->
MidCheck -> full ExhaustiveCheck, dead-flags 0x00, CUDA-pipeline semantics.
The metric is pair-checks/s of the whole job.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl engine|reference]
  python bench.py --workload len3            # 4,096 length-3 targets x length-1+2 candidates x 4 masks
  python bench.py --workload stoke           # STOKE time-to-proof, uniform proposal
  python bench.py --workload stoke-learned   # the same with the trained 50/50 mixed proposal
  python bench.py --workload gemm            # the proposal's tcgen05 bf16 GEMM, TFLOP/s

With N > 1 (torchrun) the target list is split strided across ranks (no
collective on the data path; the fixed job is shared, "scaling": "strong").
--impl reference times the reference's own CPU implementation of the path
(its host code built from its sources, oracle/_ref) on the host cores.
"""
import argparse
import csv
import ctypes
import io
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "6502-optimizer_b200"))

import numpy as np  # noqa: E402

PAIRS_PER_TARGET = 2863
WORKLOAD = "len2-enumerate-full"


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)), int(os.environ.get("LOCAL_RANK", 0))


class ClockSampler:
    """nvidia-smi clocks during the timed region (median SM MHz under load)."""
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu):
        self.gpu = gpu
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None

    def start(self):
        """Starts sampling every 50 ms and returns once the first sample is in
        (nvidia-smi takes a while to start; a timed region of a few tens of
        milliseconds would otherwise end before the first sample)."""
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.QUERY}",
                                       "--format=csv,noheader,nounits", "-lms", "50"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None
            return
        t_end = time.time() + 5.0
        while time.time() < t_end and self.p.poll() is None:
            try:
                with open(self.f.name) as g:
                    if "\n" in g.read():
                        break
            except OSError:
                break
            time.sleep(0.01)

    def stop(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        if not self.p:
            return out
        self.p.terminate()
        try:
            self.p.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.p.kill()
        self.f.flush()
        self.f.seek(0)
        rows = [r for r in csv.reader(io.StringIO(self.f.read())) if len(r) >= 9]
        os.unlink(self.f.name)
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in rows:
            for name, v in zip(names, r[5:9]):
                if v.strip().lower() == "active":
                    reasons.add(name)
        out.update(sm_mhz=statistics.median(sm) if sm else None, sm_max_mhz=max(mx) if mx else None,
                   reasons=sorted(reasons), samples=len(rows))
        return out


def cpu_model():
    """The host CPU's model name and logical core count (from /proc/cpuinfo)."""
    name = None
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    name = line.split(":", 1)[1].strip()
                    break
    except OSError:
        pass
    return {"model": name, "logical_cores": os.cpu_count() or 1}


def cpu_reference_rate(targets, budget_targets, nthreads):
    """The reference's own CPU path (oracle/_ref, else the C restatement) on a
    strided sample of the workload's targets; returns pair-checks/s.  The
    reference's host pipeline sweeps 32 representative values per register
    once a pair reads three or more (its cpu_exhaustive_check has no full
    sweep), so it does at most the work of the engine's full sweep."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    stride = max(1, len(targets) // budget_targets)
    sample = np.ascontiguousarray(targets[::stride][:budget_targets])
    t0 = time.perf_counter()
    if oracle.ref_available():
        oracle.ref_search(sample, dead=0, nthreads=nthreads)
        kind = "reference"
    else:
        oracle.search_cuda(sample, dead=0, sweep=oracle.SWEEP_REFERENCE, nthreads=nthreads)
        kind = "port"
    dt = time.perf_counter() - t0
    return len(sample) * PAIRS_PER_TARGET / dt, kind, len(sample), stride, dt


def oracle_targets(first=0, last=2863):
    """All pruned length-2 targets, enumerated by the oracle's restatement of
    the reference's enumeration and ShouldPrune (no engine code involved)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle
    return oracle.enumerate_targets(2, first, last)


REF_SWEEP_NOTE = ("reference: 32 representative values per register for pairs reading >= 3 extra registers "
                  "(cpu_exhaustive_check, the reference's only CPU sweep); engine: all 256 values")


def run_reference(args):
    """The reference's own host pipeline (oracle/_ref: h_fingerprint,
    h_midcheck, should_prune, cpu_exhaustive_check built from its sources)
    on a strided sample of the length-2 workload, all host threads.  Nothing
    of the engine is loaded: the targets come from the oracle."""
    rank, world, _ = dist_env()
    if world > 1:
        import torch.distributed as dist
        import datetime
        dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=120))
        if rank != 0:
            dist.barrier()
            dist.destroy_process_group()
            return
    targets = oracle_targets(args.first_op, args.last_op)
    nthreads = os.cpu_count() or 1
    per_step = args.ref_sample
    for _ in range(args.warmup):
        cpu_reference_rate(targets, max(8, per_step // 8), nthreads)
    rates, secs, kind, stride = [], 0.0, None, 1
    for _ in range(args.steps):
        rate, kind, n, stride, dt = cpu_reference_rate(targets, per_step, nthreads)
        rates.append(rate)
        secs += dt
    value = len(rates) * per_step * PAIRS_PER_TARGET / secs
    cpu = cpu_model()
    workload = WORKLOAD if (args.first_op, args.last_op) == (0, 2863) else \
        f"len2-enumerate-first-ops-{args.first_op}-{args.last_op}"
    line = {"metric": "pair-checks/s", "value": value, "unit": "pair-checks/s", "impl": "reference",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1000 * secs / max(len(rates), 1), "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "u8", "data": "synthetic (exhaustive enumeration)",
            "config": {"workload": workload, "targets": int(len(targets)), "candidates": PAIRS_PER_TARGET,
                       "dead_flags": "0x00", "semantics": "cuda-pipeline",
                       "sweep": "reference (the only sweep the reference's CPU path has)",
                       "engine_sweep": "full", "reference_sweep": "reduced for >= 3 extra registers",
                       "sweep_note": REF_SWEEP_NOTE,
                       "sample": f"every {stride}th target, {per_step} targets per step"},
            "cpu_baseline": {"value": value, "unit": "pair-checks/s", "cores": nthreads, "kind": kind,
                             "cpu": cpu["model"],
                             "sample": f"{per_step} targets (every {stride}th) x 2863 candidates per step, "
                                       "reduced sweep for >= 3 extra registers"},
            "e2e": {"value": value, "unit": "pair-checks/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
        dist.destroy_process_group()


def load_profile_figures():
    """Per-kernel figures of the committed ncu summary profiles/traffic.txt:
    DRAM bytes per full-workload launch (dram__bytes_read.sum +
    dram__bytes_write.sum), the issue-slot utilisation
    (smsp__issue_active.avg.pct_of_peak_sustained_active) and the lane
    instructions executed per unit of work of the same capture.  Lines:
    `kernel bytes issue_active lane_instructions`; `# source:` names the
    capture."""
    p = os.path.join(ROOT, "profiles", "traffic.txt")
    out, source = {}, None
    if os.path.exists(p):
        for line in open(p):
            if line.startswith("# source:"):
                source = line.split(":", 1)[1].strip()
                continue
            parts = line.split()
            if len(parts) >= 2 and not line.startswith("#") and parts[1].isdigit():
                out[parts[0]] = {"traffic": int(parts[1]),
                                 "issue_active": float(parts[2]) if len(parts) > 2 else None,
                                 "lane_insts": float(parts[3]) if len(parts) > 3 else None}
    return out, source


# The stages of a search as its events bracket them, each kernel with the
# statistic that counts its units of work.
STAGE_KERNELS = {
    "qc": (("k_qc_join", "targets"), ("k_expand", "mid_hits")),
    "exhaustive": (("k_small", "exh_passed"), ("k_exhaustive", "exh_passed"), ("k_exh_items", "exh_items")),
}


def stage_roofline(stats, stage_ms, figs, peak_lane_ops):
    """The longest stage against the integer issue rate: lane instructions its
    kernels executed (per unit of work from the profiles, times this run's
    units) over its measured time."""
    stage = max(STAGE_KERNELS, key=lambda k: stage_ms[k])
    kernels = STAGE_KERNELS[stage]
    known = all(k in figs and figs[k]["lane_insts"] is not None for k, _ in kernels)
    done = sum(figs[k]["lane_insts"] * stats[unit] for k, unit in kernels) if known else None
    achieved = done / (stage_ms[stage] / 1e3) if known and stage_ms[stage] > 0 else None
    return {"bound": "int-issue", "kernel": "+".join(k for k, _ in kernels),
            "achieved": achieved / 1e12 if achieved is not None else None, "peak": peak_lane_ops / 1e12, "unit": "Tlane-op/s",
            "frac": achieved / peak_lane_ops if achieved is not None else None,
            "kernel_ms_per_step": stage_ms[stage],
            "traffic": sum(figs[k]["traffic"] for k, _ in kernels) if all(k in figs for k, _ in kernels) else None,
            "traffic_unit": "DRAM bytes per launch (one 2^21-target pass), summed over the kernels named",
            "algorithmic": "lane instructions executed: " + ", ".join(f"{k} per {u}" for k, u in kernels) +
                           " from the profiles, times this run's counts",
            "issue_active_from_profile": {k: figs[k]["issue_active"] for k, _ in kernels
                                          if k in figs and figs[k]["issue_active"] is not None}}


def run_engine(args):
    import torch
    rank, world, local = dist_env()
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    torch.cuda.set_device(local)
    import m6502
    from m6502 import inst, _lib
    from m6502.distributed import shard_indices

    all_targets = inst.enumerate_targets(2, args.first_op, args.last_op)
    shard = np.ascontiguousarray(all_targets[shard_indices(len(all_targets), rank, world)])
    n = len(shard)
    eng = m6502.Engine(device=local)
    # the scheduling knobs for this device: the tuning cache if one exists,
    # else timed now (m6502_autotune), before anything is measured
    tune_path = os.environ.get("M6502_TUNE_CACHE") or os.path.expanduser(
        "~/.cache/m6502/bench-tune-" + "".join(c if c.isalnum() else "_" for c in
                                              torch.cuda.get_device_properties(local).name) + ".txt")
    if args.tune == "default":
        eng.tune = _lib.TUNE_DEFAULT
        tuned, tune_ms, tune_source = eng.tune, 0.0, "default"
    else:
        tuned, tune_ms = eng.autotune(cache_path=tune_path, force=args.tune == "force")
        tune_source = "timed" if tune_ms > 0 else "cache"
    stream = torch.cuda.ExternalStream(eng.stream, device=local)
    d_targets = torch.from_numpy(shard.view(np.int16)).to(f"cuda:{local}")
    flush = torch.empty(512 << 20, dtype=torch.uint8, device=f"cuda:{local}")   # > 126 MB L2
    sweep = _lib.SWEEP_FULL if args.sweep == "full" else _lib.SWEEP_REFERENCE

    def step_device():
        return eng.search(None, dead_flags=0, semantics=_lib.SEM_CUDA, sweep=sweep,
                          device_ptr=(d_targets.data_ptr(), n, 2), cap=1 << 21)

    def barrier():
        if dist:
            dist.barrier()

    rules = None
    for _ in range(args.warmup):   # each result held, as in the timed loop, so the page-locked
        rules, _ = step_device()   # rule buffers it needs are allocated before timing
    clocks = ClockSampler(local)
    clocks.start()
    total_ms, stats = 0.0, []
    for _ in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        rules, st = step_device()
        e1.record(stream)
        torch.cuda.synchronize()
        total_ms += e0.elapsed_time(e1)
        stats.append(st)
        barrier()
    clk = clocks.stop()
    # e2e: the public C-ABI call with pinned host targets in and host rules out
    pinned = torch.from_numpy(shard.view(np.int16)).pin_memory()
    host_targets = pinned.numpy().view(np.uint16)
    e2e_ms, e2e_rules = 0.0, 0
    r2 = None
    for _ in range(args.warmup):
        r2, _ = eng.search(host_targets, dead_flags=0, semantics=_lib.SEM_CUDA, sweep=sweep, cap=1 << 21)
    for _ in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        r2, _ = eng.search(host_targets, dead_flags=0, semantics=_lib.SEM_CUDA, sweep=sweep, cap=1 << 21)
        e1.record(stream)
        torch.cuda.synchronize()
        e2e_ms += e0.elapsed_time(e1)
        e2e_rules = len(r2)
        barrier()
    times = torch.tensor([total_ms, e2e_ms], dtype=torch.float64, device=f"cuda:{local}")
    counts = torch.tensor([n, len(rules)], dtype=torch.float64, device=f"cuda:{local}")
    if dist:
        dist.all_reduce(times, op=dist.ReduceOp.MAX)
        dist.all_reduce(counts, op=dist.ReduceOp.SUM)
    total_ms, e2e_ms = float(times[0]), float(times[1])
    total_targets, total_rules = int(counts[0]), int(counts[1])
    pairs_per_step = total_targets * PAIRS_PER_TARGET
    value = pairs_per_step * args.steps / (total_ms / 1000.0)
    e2e_value = pairs_per_step * args.steps / (e2e_ms / 1000.0)

    if rank == 0:
        s0 = stats[-1]
        K = len(stats)
        avg = lambda k: sum(s[k] for s in stats) / K  # noqa: E731
        props = torch.cuda.get_device_properties(local)
        sms = props.multi_processor_count
        f_mhz = clk["sm_mhz"] or clk["sm_max_mhz"] or 1965.0
        peak_lane_ops = sms * 128 * f_mhz * 1e6       # 32-bit integer lanes per SM per clock
        exh_ms = avg("ms_exhaustive") + avg("ms_exh_items")
        qc_ms = avg("ms_qc")
        exh_achieved = s0["exh_algo_ops"] / (exh_ms / 1e3) if exh_ms > 0 else 0.0
        qc_algo = 13 * s0["pairs"] + 13 * (7 + 24) * s0["qc_hits"]
        qc_achieved = qc_algo / (qc_ms / 1e3) if qc_ms > 0 else 0.0
        stages = {"fingerprint_ms": avg("ms_fingerprint"), "qc_mid_ms": qc_ms,
                  "exhaustive_ms": avg("ms_exhaustive"), "exh_items_ms": avg("ms_exh_items"),
                  "emit_ms": avg("ms_emit")}
        figs, figs_source = load_profile_figures()
        roof = stage_roofline(s0, {"qc": qc_ms, "exhaustive": exh_ms}, figs, peak_lane_ops)
        roof.update({
            "peak_basis": f"{sms} SMs x 128 int32 lanes x {f_mhz:.0f} MHz (median SM clock sampled)",
            # the fixed convention: every pair costs its QuickCheck, every accepted
            # pair its whole product sweep; neither the join nor the cones do that
            # work, so these figures exceed the peak and are not a utilisation
            "convention": {"qc_achieved": qc_achieved / 1e12, "exhaustive_achieved": exh_achieved / 1e12,
                           "qc_algorithmic": "13 ops/pair + 31x13 ops per QC hit (QC+MidCheck)",
                           "exhaustive_algorithmic": "accepted pairs x 2^(9+8k) states x (10 ops/instruction + 3)",
                           "note": "emulation-equivalent, not a utilisation"},
            "profile_source": figs_source})
        line = {
            "metric": "pair-checks/s", "value": value, "unit": "pair-checks/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps,
            "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (exhaustive enumeration of all length-2 targets)",
            "config": {"workload": WORKLOAD if (args.first_op, args.last_op) == (0, 2863)
                       else f"len2-enumerate-first-ops-{args.first_op}-{args.last_op}",
                       "targets": total_targets, "candidates": PAIRS_PER_TARGET,
                       "pairs_per_step": pairs_per_step, "dead_flags": "0x00",
                       "sweep": args.sweep, "semantics": "cuda-pipeline", "exh_mode": "cones",
                       "parallelism": f"strided target shards x{world}",
                       "l2": "512 MB buffer written between timed steps"},
            "len2_wall_s": total_ms / args.steps / 1000.0,
            "cuda_graph_replayed": bool(s0.get("graph_replays", 0)),
            "rules": total_rules,
            "stage_counts": {k: s0[k] for k in ("qc_hits", "mid_hits", "exh_checked", "exh_passed", "rules",
                                                  "exh_states", "exh_items", "exh_probe_rejects")},
            "stages_ms": stages,
            "roofline": roof,
            "clocks": {"sm_mhz": clk["sm_mhz"], "sm_max_mhz": clk["sm_max_mhz"], "reasons": clk["reasons"]},
            "e2e": {"value": e2e_value, "unit": "pair-checks/s", "h2d_bytes_per_step": int(shard.nbytes),
                    "d2h_bytes_per_step": int(e2e_rules * 16 + 8 * 16 * s0["passes"])},
            # per pass: opcode check, QC join, expansion, small cones, exhaustive, work
            # items, emit (the join computes the targets' outputs itself, so no
            # fingerprint launch)
            "gpu_launches": int(7 * s0["passes"] * args.steps),
        }
        line["config"]["tuning"] = dict(tuned, source=tune_source, calibration_ms=tune_ms,
                                        trace=m6502.Engine.tune_trace(tune_path) if args.tune != "default" else [])
        if world == 1 and not args.no_mask_ff:
            line["mask_ff"] = mask_ff_run(eng, stream, d_targets, n, sweep)
        if world == 1 and not args.no_stoke:   # configs 4 and 5, beside the headline
            main, extra = stoke_compare(eng, args, learned=True)
            line["stoke"] = {"config": stoke_config(args, True), "learned": main, **extra}
        if world == 1 and not args.no_cpu_baseline:
            rate, kind, ns, stride, dt = cpu_reference_rate(all_targets, args.cpu_sample, os.cpu_count() or 1)
            line["cpu_baseline"] = {"value": rate, "unit": "pair-checks/s", "cores": os.cpu_count() or 1,
                                    "kind": kind, "cpu": cpu_model()["model"],
                                    "sample": f"{ns} targets (every {stride}th of the workload) "
                                    f"x 2863 candidates, {dt:.1f} s",
                                    "sweep": REF_SWEEP_NOTE}
        print(json.dumps(line), flush=True)
    eng.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def mask_ff_run(eng, stream, d_targets, n, sweep):
    """The same enumeration at dead-flags 0xFF (every flag dead): 482 M pairs
    survive MidCheck and go to ExhaustiveCheck.  The rules are counted on the
    device, not copied out.  One warm-up run, then one run timed with CUDA
    events on the engine's stream."""
    import torch
    from m6502 import _lib

    def run():
        return eng.search(None, dead_flags=0xFF, semantics=_lib.SEM_CUDA, sweep=sweep,
                          device_ptr=(d_targets.data_ptr(), n, 2), count_only=True)
    run()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    nrules, st = run()
    e1.record(stream)
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    return {"dead_flags": "0xFF", "ms": ms, "pair_checks_per_s": n * PAIRS_PER_TARGET / (ms / 1e3),
            "rules": nrules, "qc_hits": st["qc_hits"], "mid_hits": st["mid_hits"],
            "exh_checked": st["exh_checked"], "exh_passed": st["exh_passed"],
            "exh_probe_rejects": st["exh_probe_rejects"], "exh_states": st["exh_states"],
            "exh_items": st["exh_items"],
            "stages_ms": {"qc_mid_ms": st["ms_qc"], "exhaustive_ms": st["ms_exhaustive"],
                          "exh_items_ms": st["ms_exh_items"], "emit_ms": st["ms_emit"]},
            "note": "rules counted on the device (M6502_COUNT_ONLY), not copied to the host"}


def stoke_once(eng, targets, args, model=None):
    """One STOKE run over the 512-target set; returns the per-target summary
    and the stats.  Same seeds for every proposal."""
    from m6502 import _lib
    kw = dict(chains_per_target=128, steps=args.stoke_steps, steps_per_epoch=args.stoke_epoch,
              first_epoch=args.stoke_first_epoch, seed=2, cost=_lib.COST_HAMMING, sweep=_lib.SWEEP_FULL,
              stop_on_proof=True)
    if model is not None:
        kw.update(model=model, learned_frac=args.stoke_learned_frac, uniform_chains=args.stoke_uniform_chains)
    res, proofs, st = eng.stoke(targets, **kw)
    times = sorted(r["first_proof_ms"] for r in res if r["first_proof_ms"] >= 0)
    steps = sorted(r["first_proof_step"] for r in res if r["first_proof_ms"] >= 0)
    q = lambda xs, f: xs[int(f * (len(xs) - 1))] if xs else None  # noqa: E731
    summary = {"median_ms": statistics.median(times) if times else None,
               "p75_ms": q(times, 0.75), "p90_ms": q(times, 0.9),
               "median_steps": statistics.median(steps) if steps else None,
               "p75_steps": q(steps, 0.75), "p90_steps": q(steps, 0.9),
               "proved": len(times), "censored": len(targets) - len(times),
               "proofs": st["proofs"], "candidates": st["candidates"], "verified": st["verified"],
               "undecided": st["undecided"], "epochs": st["epochs"],
               "chain_steps_per_s": st["steps"] / (st["ms_device"] / 1e3) if st["ms_device"] else None,
               "ms_device": st["ms_device"], "ms_chains": st["ms_chains"], "ms_verify": st["ms_verify"]}
    return res, summary


def hard_target_speedup(res_u, res_l, min_steps, budget):
    """Median ratio of first-proof steps (uniform / learned) over the targets
    uniform STOKE needed at least min_steps for; an unproved target counts at
    the step budget, and targets neither proposal proved are left out."""
    ratios = []
    for ru, rl in zip(res_u, res_l):
        su = ru["first_proof_step"] if ru["first_proof_ms"] >= 0 else budget
        sl = rl["first_proof_step"] if rl["first_proof_ms"] >= 0 else budget
        if su < min_steps or (ru["first_proof_ms"] < 0 and rl["first_proof_ms"] < 0):
            continue
        ratios.append((su + 1) / (sl + 1))
    return {"targets": len(ratios), "min_uniform_steps": min_steps,
            "median_step_ratio": statistics.median(ratios) if ratios else None}


def hard_target_times(res_u, res_l, first_epoch, ms_u, ms_l):
    """Time-to-proof on the targets uniform STOKE did not prove within its
    first epoch (the same seeds make that epoch identical under both
    proposals, since the model is first used in the second).  A target a
    proposal never proved counts at that run's whole device time (censored,
    so its true time is at least that); targets neither proved are left
    out.  Returns both medians, their ratio and the median per-target
    ratio."""
    tu, tl, ratios, cens_u, cens_l = [], [], [], 0, 0
    for ru, rl in zip(res_u, res_l):
        if ru["first_proof_ms"] >= 0 and ru["first_proof_step"] < first_epoch:
            continue
        if ru["first_proof_ms"] < 0 and rl["first_proof_ms"] < 0:
            continue
        a = ru["first_proof_ms"] if ru["first_proof_ms"] >= 0 else ms_u
        b = rl["first_proof_ms"] if rl["first_proof_ms"] >= 0 else ms_l
        cens_u += ru["first_proof_ms"] < 0
        cens_l += rl["first_proof_ms"] < 0
        tu.append(a)
        tl.append(b)
        ratios.append(a / b if b > 0 else None)
    ratios = [r for r in ratios if r is not None]
    mu, ml = (statistics.median(tu) if tu else None), (statistics.median(tl) if tl else None)
    return {"targets": len(tu), "definition": f"uniform first proof at step >= {first_epoch} or never",
            "median_ms_uniform": mu, "median_ms_learned": ml,
            "speedup_median_ms": mu / ml if mu and ml else None,
            "median_per_target_ratio": statistics.median(ratios) if ratios else None,
            "censored_uniform": cens_u, "censored_learned": cens_l}


def stoke_compare(eng, args, learned):
    """The 512-target STOKE workload (seed 2) with the uniform proposal and,
    when `learned`, with the 50/50 mixed proposal of a model first trained on
    the GPU (training targets seed 20, validation seed 22, disjoint draws).
    Returns (summary of the main run, extra keys)."""
    from m6502 import inst, _lib
    from m6502.proposal import train_proposal
    targets = inst.draw_targets(2, 4, 8, 512, reject_pruned=False)
    # warm-up at full size (every device buffer allocated before the timed runs)
    eng.stoke(targets, chains_per_target=128, steps=4 * args.stoke_first_epoch, steps_per_epoch=args.stoke_epoch,
              first_epoch=args.stoke_first_epoch, seed=1, cost=_lib.COST_HAMMING, sweep=_lib.SWEEP_FULL,
              stop_on_proof=True)
    model, train_info, train_s = None, None, None
    if learned:
        t0 = time.perf_counter()
        model, train_info = train_proposal(eng, inst.draw_targets(20, 4, 8, 2048, reject_pruned=False),
                                           inst.draw_targets(22, 4, 8, 64, reject_pruned=False),
                                           steps=3000, chunk=500)
        train_s = time.perf_counter() - t0
    res_u, uni = stoke_once(eng, targets, args)
    extra = {}
    if not learned:
        return uni, extra
    res_l, lrn = stoke_once(eng, targets, args, model)
    extra["uniform"] = uni
    extra["train"] = dict(train_info, seconds=train_s)
    if uni["median_ms"] and lrn["median_ms"]:
        extra["speedup_median_ms"] = uni["median_ms"] / lrn["median_ms"]
    if uni["median_steps"] is not None and lrn["median_steps"] is not None:
        extra["speedup_median_steps"] = (uni["median_steps"] + 1) / (lrn["median_steps"] + 1)
    extra["hard_targets"] = hard_target_times(res_u, res_l, args.stoke_first_epoch, uni["ms_device"],
                                              lrn["ms_device"])
    extra["hard_targets_steps"] = hard_target_speedup(res_u, res_l, 1000, args.stoke_steps)
    model.close()
    return lrn, extra


def run_stoke(args):
    """STOKE benchmark workloads on 512 seeded targets of length 4..8 (seed 2),
    128 chains each (65,536 chains), Hamming cost over the 32 MidCheck
    vectors, temperature 1.0 -> 0.1; every shorter zero-cost best is proved on
    the GPU (full sweep).  Metric: median time-to-proof over the proved
    targets.  `stoke`: the uniform proposal.  `stoke-learned`: the 50/50
    mixed proposal of a model trained first on the GPU, reported beside a
    uniform run with the same seeds."""
    import torch
    import m6502
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    eng = m6502.Engine(device=local)
    learned = args.workload == "stoke-learned"
    clocks = ClockSampler(local)
    clocks.start()
    main, extra = stoke_compare(eng, args, learned)
    clk = clocks.stop()
    line = {"metric": "STOKE time-to-proof (median over proved targets)", "value": main["median_ms"], "unit": "ms",
            "higher_is_better": False, "n_gpus": 1, "steps": args.stoke_steps, "warmup": 1,
            "dtype": "u8", "data": "synthetic (512 seeded random targets, length 4-8, seed 2)",
            "config": stoke_config(args, learned),
            "clocks": {"sm_mhz": clk["sm_mhz"], "sm_max_mhz": clk["sm_max_mhz"], "reasons": clk["reasons"]}}
    line.update(main)
    line.update(extra)
    print(json.dumps(line), flush=True)
    eng.close()


def stoke_config(args, learned):
    return {"workload": "stoke-512x128" + ("-learned" if learned else ""), "targets": 512,
            "chains_per_target": 128, "steps_per_chain": args.stoke_steps,
            "steps_per_epoch": args.stoke_epoch, "first_epoch": args.stoke_first_epoch,
            "cost": "hamming over 32 vectors + bytes + cycles/100", "temperature": "1.0 -> 0.1",
            "proposal": (f"portfolio: {args.stoke_uniform_chains} of every 8 chains of a target uniform, the "
                         f"others mixed {args.stoke_learned_frac:.2f} learned + uniform (model from the second "
                         f"epoch on)" if learned else "uniform"),
            "sweep": "full", "stop_on_proof": True}


def run_gemm(args):
    """The learned proposal's dense-layer kernel (tcgen05 bf16 GEMM, fp32
    accumulate in TMEM) against the measured cuBLAS bf16 peak of this pool
    (MEASURED_PEAKS.json, burst figure): a square problem (--gemm-n), then
    the proposal network's own layer shapes at its largest batch (65,536
    chain rows: 448 -> 512, 512 -> 512, 512 -> 384, and the weight gradient
    512 x 512 over K = 65,536 rows).  One JSON line per shape."""
    import torch
    import m6502
    from m6502.mlp import gemm_bf16, gemm_bf16_timed
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    shapes = [(args.gemm_n, args.gemm_n, args.gemm_n)]
    if args.gemm_shapes:
        shapes += [tuple(int(v) for v in s.split("x")) for s in args.gemm_shapes.split(",")]
    peaks = {}
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            peaks = json.load(f)
    except OSError:
        pass
    peak = peaks.get("bf16_tflops", 1590.0)
    eng = m6502.Engine(device=local)
    g = torch.Generator(device=f"cuda:{local}").manual_seed(0)
    for (M, N, K) in shapes:
        a = torch.randn(M, K, device=f"cuda:{local}", generator=g).to(torch.bfloat16)
        b = torch.randn(N, K, device=f"cuda:{local}", generator=g).to(torch.bfloat16)
        for _ in range(max(args.warmup, 3)):
            c = gemm_bf16(eng, a, b)
        torch.cuda.synchronize()
        ref = a[:256].float() @ b.float().T
        err = float((c[:256] - ref).abs().max() / ref.abs().max())
        # short problems: repeat so that the timed region spans ~100 ms
        flop = 2.0 * M * N * K
        reps = max(args.steps, int(min(2000, max(1, 1e14 / flop))))
        clocks = ClockSampler(local)
        clocks.start()
        # back-to-back launches on the engine's stream, timed there by CUDA events
        _, ms = gemm_bf16_timed(eng, a, b, reps)
        clk = clocks.stop()
        tflops = flop / (ms / 1e3) / 1e12
        square = M == N == K
        line = {"metric": "bf16 GEMM TFLOP/s (tcgen05, TMA, 128x256 tiles)", "value": tflops, "unit": "TFLOP/s",
                "higher_is_better": True, "n_gpus": 1, "steps": reps, "warmup": max(args.warmup, 3),
                "ms_per_step": ms, "dtype": "bf16", "data": "synthetic (seeded normal)",
                "config": {"workload": f"gemm-{M}" if square else f"gemm-mlp-{M}x{N}x{K}", "M": M, "N": N, "K": K,
                           "output": "fp32, written to HBM (the MLP's layers fuse bias/ReLU instead)"},
                "roofline": {"bound": "tensor", "achieved": tflops, "peak": peak, "unit": "TFLOP/s",
                             "frac": tflops / peak, "peak_source": "measured" if peaks else "fallback"},
                "max_rel_err_vs_fp32": err,
                "clocks": {"sm_mhz": clk["sm_mhz"], "sm_max_mhz": clk["sm_max_mhz"], "reasons": clk["reasons"]}}
        print(json.dumps(line), flush=True)
        del a, b, c
    eng.close()


def go_checked_pairs(targets, rules, dead, nc2=True):
    """Distinct (target, candidate) pairs the Go worker decides before it
    stops (worker.go:122-176: every candidate of each length it tries, up to
    and including the first pass), from the rule set.  Under a dead-flags
    mask the masked pass walks the same Go order again; a pair both passes
    examine is counted once, so each target counts the longer of its two
    walks."""
    from m6502 import inst, _lib
    go_tab = inst.insn_table(_lib.SEM_GO)
    rank = {int(x): i for i, x in enumerate(go_tab)}
    n1, n2 = len(go_tab), len(go_tab) ** 2 if nc2 else 0
    win = {}
    for r in rules:
        c = [int(x) for x in r["cand"][:r["cand_len"]]]
        kind = 1 if (dead and int(r["dead_flags"])) else 0
        rk = rank[c[0]] + 1 if len(c) == 1 else n1 + rank[c[0]] * n1 + rank[c[1]] + 1
        win[(int(r["target"]), kind)] = rk
    total = 0
    for t in range(len(targets)):
        total += max(win.get((t, kind), n1 + n2) for kind in range(2 if dead else 1))
    return total


def run_len3(args):
    """Batched length-3 workload: 4,096 seeded length-3 targets (seed 1), each
    searched against all length-1 (2,863) and length-2 (8,196,769) candidates
    under dead-flags masks 0x00, 0x01, 0xC3, 0xFF, Go-worker semantics (first
    passing candidate per length in Go order), full sweep by default.  One
    step = the four masks.  Metric: pair-checks/s, counting the distinct
    pairs the Go worker decides before it stops."""
    import torch
    import m6502
    from m6502 import inst, _lib
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    from concurrent.futures import ThreadPoolExecutor
    masks = (0x00, 0x01, 0xC3, 0xFF)
    sweep = _lib.SWEEP_FULL if args.len3_sweep == "full" else _lib.SWEEP_REFERENCE
    targets = np.asarray(inst.draw_targets(1, 3, 3, 4096), dtype=np.uint16)
    # one engine context (stream, buffers, key tables) per mask, driven from
    # its own host thread, so the four searches run concurrently on the GPU
    engines = [m6502.Engine(device=local) for _ in masks]
    tuned, _ = engines[0].autotune()
    for e in engines[1:]:
        e.tune = tuned
    streams = [torch.cuda.ExternalStream(e.stream, device=local) for e in engines]
    fork = torch.cuda.Stream(device=local)
    pool = ThreadPoolExecutor(len(masks))
    d_targets = torch.from_numpy(targets.view(np.int16)).to(f"cuda:{local}")
    flush = torch.empty(512 << 20, dtype=torch.uint8, device=f"cuda:{local}")

    def one(i, device):
        m = masks[i]
        if device:
            return engines[i].search(None, dead_flags=m, semantics=_lib.SEM_GO, sweep=sweep, max_cand_len=2,
                                     device_ptr=(d_targets.data_ptr(), len(targets), 3), cap=2 * len(targets) + 16)
        return engines[i].search(targets, dead_flags=m, semantics=_lib.SEM_GO, sweep=sweep, max_cand_len=2,
                                 cap=2 * len(targets) + 16)

    def step(device=True):
        return list(pool.map(lambda i: one(i, device), range(len(masks))))

    def timed_step(device=True):
        """Device time of one step: an event on a fork stream that every
        engine stream waits for, and a join event after all four."""
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record(fork)
        for st_ in streams:
            st_.wait_event(start)
        out = step(device)
        for st_ in streams:
            ev = torch.cuda.Event()
            ev.record(st_)
            fork.wait_event(ev)
        stop.record(fork)
        torch.cuda.synchronize()
        return out, start.elapsed_time(stop)

    # the first step builds each mask's sorted key table of the 8.2 M length-2
    # candidates (164 MB each) and records the passes as CUDA graphs; later
    # steps reuse both
    torch.cuda.synchronize()
    _, first_ms = timed_step()
    for _ in range(max(args.warmup, 1) - 1):
        step()
    # The register-cap variant of the exhaustive kernel is chosen on this
    # workload (four searches share the SMs here, unlike the single search
    # the device-wide tuning times): each candidate's passes are recorded by
    # one untimed step, then two steps are timed; all of it in the warm-up.
    len3_trace = []
    for minb in (4, 3, 2):
        knobs = dict(tuned, exh_minb=minb)
        for e in engines:
            e.tune = knobs
        step()
        len3_trace.append({"exh_minb": minb, "ms": min(timed_step()[1] for _ in range(2))})
    best = min(len3_trace, key=lambda r: r["ms"])["exh_minb"]
    tuned = dict(tuned, exh_minb=best)
    for e in engines:
        e.tune = tuned
    step()
    clocks = ClockSampler(local)
    clocks.start()
    ms, res = [], None
    for _ in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        res, t = timed_step()
        ms.append(t)
    e2e_ms = []
    for _ in range(args.steps):   # host targets in, host rules out, through the C ABI
        flush.fill_(1)
        torch.cuda.synchronize()
        _, t = timed_step(device=False)
        e2e_ms.append(t)
    clk = clocks.stop()
    pairs = sum(go_checked_pairs(targets, rules, m) for m, (rules, _) in zip(masks, res))
    all_pairs = sum(st["pairs"] for _, st in res)
    t_ms = statistics.median(ms)
    per_mask = {f"0x{m:02X}": {"rules": int(len(rules)), "qc_hits": st["qc_hits"], "exh_checked": st["exh_checked"],
                               "exh_passed": st["exh_passed"], "exh_undecided": st["exh_undecided"],
                               "exh_states": st["exh_states"], "exh_items": st["exh_items"], "ms": st["ms_device"],
                               "ms_qc": st["ms_qc"], "ms_exhaustive": st["ms_exhaustive"],
                               "ms_exh_items": st["ms_exh_items"], "ms_emit": st["ms_emit"]}
                for m, (rules, st) in zip(masks, res)}
    line = {"metric": "pair-checks/s", "value": pairs / (t_ms / 1e3), "unit": "pair-checks/s",
            "n_gpus": 1, "steps": args.steps, "warmup": max(args.warmup, 1), "ms_per_step": t_ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (4,096 seeded length-3 targets, seed 1)",
            "config": {"workload": "len3-x-len1+len2-4masks", "targets": len(targets),
                       "candidates": 2863 + 2863 * 2863, "masks": [f"0x{m:02X}" for m in masks],
                       "semantics": "go worker (first pass per candidate length)", "sweep": args.len3_sweep,
                       "tuning": dict(tuned, exh_minb_source="timed on this workload in the warm-up",
                                      exh_minb_trace=len3_trace),
                       "l2": "flushed between steps (512 MB write)",
                       "schedule": "one engine context per mask, the four searches concurrent on four streams; "
                                   "each search pass one CUDA graph with device-settled Go-order rounds",
                       "key_tables": "built by the first step (first_step_ms) and cached: not in the timed steps"},
            "first_step_ms": first_ms,
            "pairs_go_counted": pairs, "pairs_counting": "distinct (target, candidate) pairs per mask",
            "pairs_decided": all_pairs, "per_mask": per_mask,
            "e2e": {"value": pairs / (statistics.median(e2e_ms) / 1e3), "unit": "pair-checks/s",
                    "h2d_bytes_per_step": int(targets.nbytes) * len(masks),
                    "d2h_bytes_per_step": int(sum(len(r) for r, _ in res)) * 16},
            "clocks": {"sm_mhz": clk["sm_mhz"], "sm_max_mhz": clk["sm_max_mhz"], "reasons": clk["reasons"]}}
    if not args.no_cpu_baseline:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle
        nthreads = os.cpu_count() or 1
        sample = targets[::64][:64]
        t0 = time.perf_counter()
        cpu_pairs = 0
        for m in masks:
            _, st = oracle.search_go(sample, dead=m, max_cand_len=2, nthreads=nthreads)
            cpu_pairs += st["pairs"]
        dt = time.perf_counter() - t0
        line["cpu_baseline"] = {"value": cpu_pairs / dt, "unit": "pair-checks/s", "cores": nthreads, "kind": "port",
                                "sample": f"{len(sample)} targets (every 64th) x 4 masks, oracle Go worker "
                                          f"(reduced sweep, both passes counted), {dt:.1f} s"}
    print(json.dumps(line), flush=True)
    pool.shutdown()
    for e in engines:
        e.close()


def main():
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["engine", "reference"], default="engine")
    ap.add_argument("--sweep", choices=["full", "reference"], default="full")
    ap.add_argument("--cpu-sample", type=int, default=1500, help="targets in the CPU baseline sample")
    ap.add_argument("--ref-sample", type=int, default=600, help="targets per reference-arm step")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-mask-ff", action="store_true", help="skip the dead-flags 0xFF run of the default line")
    ap.add_argument("--no-stoke", action="store_true", help="skip the STOKE runs (configs 4, 5) of the default line")
    ap.add_argument("--len3-sweep", choices=["full", "reference"], default="full",
                    help="ExhaustiveCheck sweep of the length-3 workload")
    ap.add_argument("--tune", choices=["auto", "force", "default"], default="auto",
                    help="scheduling knobs: the device's tuning cache or a timed tuning (auto), a new timed "
                         "tuning (force), or the built-in defaults")
    ap.add_argument("--workload", choices=["len2", "len3", "stoke", "stoke-learned", "gemm"], default="len2")
    ap.add_argument("--gemm-n", type=int, default=8192, help="GEMM workload: M = N = K")
    ap.add_argument("--gemm-shapes", default="65536x512x448,65536x512x512,65536x384x512,512x512x65536",
                    help="GEMM workload: further MxNxK shapes after the square one (empty: none)")
    ap.add_argument("--first-op", type=int, default=0,
                    help="length-2 workload: first instructions [first-op, last-op) of the CUDA-order table "
                         "(a subset, for small profiler captures)")
    ap.add_argument("--last-op", type=int, default=2863)
    ap.add_argument("--stoke-steps", type=int, default=1000000, help="steps per chain (STOKE workload)")
    ap.add_argument("--stoke-epoch", type=int, default=2000, help="steps between proof rounds (STOKE workload)")
    ap.add_argument("--stoke-learned-frac", type=float, default=0.5,
                    help="share of replace / insert moves the learned proposal draws")
    ap.add_argument("--stoke-uniform-chains", type=int, default=4,
                    help="learned STOKE: of every 8 chains of a target, how many keep the uniform proposal")
    ap.add_argument("--stoke-first-epoch", type=int, default=64,
                    help="steps of the first STOKE epoch; epochs double up to --stoke-epoch")
    args = ap.parse_args()
    if args.workload in ("stoke", "stoke-learned"):
        run_stoke(args)
    elif args.workload == "len3":
        run_len3(args)
    elif args.workload == "gemm":
        run_gemm(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_engine(args)


if __name__ == "__main__":
    main()
