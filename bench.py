"""Benchmark of the EDDY permutation test on GB300: gene-set x permutation
units per second, exact edges.

Workload (one gene set, the largest single-GPU configuration the metric is
quoted on): 200 genes x 1000 samples (classes 400/600), -mp 4, the -r 10000
permutation test; synthetic seeded data of the "precision stress" workload
(eddy_gpu/synth.py config 4: every gene loads on one latent factor, so the
pair tests sit near the Bonferroni edge threshold; the measured near-threshold
fractions are reported in `config`).  One step = `--units` permutations of
that set (default 10000: the whole -r 10000 run).

  value  device time of the hot path with the set resident in HBM (CUDA
         events on the library's launching stream around K steps; labellings
         generated on the device from the counter stream).
  e2e    the same units through the public C ABI per step: the matrix and
         labels copied from pinned host memory, the set added, eddy_run
         (iteration 0 with its networks, the permutations, the beta fit) and
         the JS values read back.
  cpu_baseline  the oracle (CPU restatement of the reference kernels, FP64,
         OpenMP over units, or inside a unit when units are fewer than
         threads) on a bounded sample of the same units.
  precision  edge decisions of every network, node-summed BDeu, JS, U and
         the pDDN of one eddy_run, against the FP64 oracle on that sample.

`--impl reference` runs the reference's algorithm on the host cores (the
oracle port: the reference's own hot path exists only as CUDA kernels; its
CPU build here runs under a thread emulator and is not a performance arm)
on the same workload, each step a bounded sample of units.
Multi-GPU: every rank processes its own permutation indices (weak scaling,
no collective on the data path); timing is the max over ranks.
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

ROOT = os.path.dirname(os.path.abspath(__file__))
for _p in (os.path.join(ROOT, "eddy-gpu_gb300"), os.path.join(ROOT, "oracle")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import numpy as np  # noqa: E402

METRIC = "gene-set x permutations/sec, batched FP32 vs plain FP64 on one GB300, exact edges"
UNIT = "units/s"
WORKLOAD = ("config 4 (precision stress): one 200-gene set x 1000 samples (400/600), -mp 4, "
            "permutations of -r 10000")


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return d.get("hbm_gbs", 6800.0), d.get("bf16_tflops", 1900.0), "measured"
    return 6800.0, 1900.0, "fallback"


def required_bytes(g, n):
    """Per-unit bytes the network stages (k_units: networks, dedup, BDeu,
    normalisation and JS) cannot do without when everything else stays on
    chip: the decision masks read and cleared, the labelling's mask, and the
    JS, unique count and status written."""
    return 2 * 4 * (g * (g - 1) // 2) + 8 * ((n + 63) // 64) + 16


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    def __init__(self, index=0):
        self.index = index
        self.rows = []  # (host time, fields)
        self.proc = None
        self.window = None

    def mark(self, t0, t1):
        """Restricts the summary to samples taken in [t0, t1] (host clock)."""
        self.window = (t0, t1)

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={q}", "--format=csv,noheader,nounits", "-lms", "50",
                 "-i", str(self.index)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9:
                self.rows.append((time.perf_counter(), parts))

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        rows = [r for t, r in self.rows
                if self.window is None or self.window[0] <= t <= self.window[1] + 0.06]
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        self_rows = rows
        sm = [float(r[1]) for r in self_rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self_rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self_rows for i in range(4)
                          if r[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(self_rows)}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def cpu_sample(w, genes, seed, first, count, threads):
    """Oracle (FP64, the reference's algorithm) on `count` units; returns
    (units/s, seconds)."""
    import oracle
    lab = oracle.counter_labels(seed, 0, w.labels, first + count)[first:first + count]
    prm = oracle.params(mp=w.flags["mp"], pw=w.flags["pw"])
    t0 = time.perf_counter()
    js, U = oracle.units(w.data[genes], lab, None, prm, threads=threads)
    dt = time.perf_counter() - t0
    return count / dt, dt, js, U


def precision_vs_oracle(eddy_gpu, oracle, w, genes, seed, labs, ojs, oU):
    """The GPU against the FP64 oracle on the sampled labellings: one
    eddy_run over them (the unpermuted labelling and the permutations of
    the counter stream) for JS, U and pDDN; every edge decision of every
    network and the node-summed BDeu of every unique network for the first
    two labellings."""
    mp, pw = w.flags["mp"], w.flags["pw"]
    prm = oracle.params(mp=mp, pw=pw)
    R = labs.shape[0]
    ctx = eddy_gpu.Context(max_parents=mp, prior_weight=pw, permutations=R,
                           rng=eddy_gpu.RNG_COUNTER, seed=seed, keep_networks=True)
    ctx.load_matrix(w.data, w.labels)
    sid = ctx.add_set(genes)
    ctx.run()
    gjs, gU = ctx.js(sid)
    summ = ctx.summary(sid)
    rc, _, _, opd = oracle.pddn(ojs)
    data = w.data[genes]
    tests = agree = 0
    bdeu_err = 0.0
    ids_equal = True
    for r in range(min(2, R)):
        o = oracle.unit(data, labs[r], None, prm)
        e = ctx.debug_edges(sid, labs[r])
        tests += e.size
        agree += int((e == o["edges"]).sum())
        d = ctx.debug_unit(sid, labs[r], min(mp, 3))
        ids_equal &= bool(np.array_equal(d["ids"], o["unique_ids"]))
        od = o["out5"].sum(axis=2)
        if d["dist"].shape == od.shape:
            bdeu_err = max(bdeu_err, float(np.max(np.abs(d["dist"] - od) / np.abs(od))))
        else:
            bdeu_err = float("inf")
    ctx.close()
    rel = np.abs(gjs - ojs) / np.maximum(np.abs(ojs), 1e-300)
    return {"oracle_units": int(R),
            "edge_decisions_compared": int(tests),
            "edge_decision_agreement": agree / max(tests, 1),
            "unique_ids_equal": ids_equal,
            "unique_networks_equal": bool(np.array_equal(gU, oU)),
            "bdeu_max_rel_err": bdeu_err,
            "js_max_rel_err": float(np.max(rel)),
            "pddn": summ["pddn"], "pddn_oracle": opd,
            "pddn_rel_err": (abs(summ["pddn"] - opd) / abs(opd)) if rc == 0 and opd else None}


def run_reference(args, rank, world):
    """Reference arm: the reference's hot path on the host cores (oracle
    port), same workload and metric; rank 0 only."""
    if rank != 0:
        return
    from eddy_gpu import synth
    import oracle
    oracle.build(ref=False)
    w = synth.make(4, seed=0)
    genes = w.sets[0][1]
    threads = os.cpu_count() or 1
    per_step = args.ref_units
    for i in range(args.warmup):
        cpu_sample(w, genes, 4242, 1 + i * per_step, per_step, threads)[:2]
    t0 = time.perf_counter()
    done = 0
    for i in range(args.steps):
        cpu_sample(w, genes, 4242, 1 + (args.warmup + i) * per_step, per_step, threads)
        done += per_step
    dt = time.perf_counter() - t0
    v = done / dt
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT,
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * dt / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": WORKLOAD + f"; a bounded sample of {per_step} "
                       "permutations per step", "units_per_step": per_step},
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                             "sample": f"{per_step} permutations per step x {args.steps} steps"},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_multiset(args, rank, world, local):
    """Configs 3 and 5: many gene sets of uneven size, -r iterations each on
    the counter stream (labellings drawn on the device).  `value`: one
    eddy_run over all sets, which packs the sets of each contingency-kernel
    choice into shared batches (a batch holds the units of several sets);
    `per_set_value`: the same units set by set (one eddy_run_permutations
    call per set).  Prints its own JSON line."""
    import torch

    torch.cuda.set_device(local)
    import build as _build
    _build.build()
    import eddy_gpu
    from eddy_gpu import synth
    w = synth.make(args.workload, seed=0, n_sets=args.sets)
    R = args.perms or w.flags["r"]
    ctx = eddy_gpu.Context(max_parents=w.flags["mp"], prior_weight=w.flags["pw"], permutations=R,
                           rng=eddy_gpu.RNG_COUNTER, seed=77, device=local, keep_networks=False)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.load_matrix(w.data, w.labels)

    def add_all():
        ctx.clear_sets()
        return [ctx.add_set(genes, prior) for _, genes, prior in w.sets]

    # warm-up: one full run (tunes every size class once)
    add_all()
    ctx.run()
    torch.cuda.synchronize()
    sids = add_all()
    t0 = time.perf_counter()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    ctx.run()
    e1.record(stream)
    torch.cuda.synchronize()
    wall = time.perf_counter() - t0
    ms = e0.elapsed_time(e1)
    t = ctx.timing()
    # the units the run needed: iteration 0 of every set, and the
    # permutations of the sets whose iteration-0 JS is finite (a set stops
    # at a non-finite one, main.cu:1431-1435, as the reference's does)
    iters = [ctx.summary(s)["iterations"] for s in sids]
    units = int(sum(iters))
    stop0 = sum(1 for s, it in zip(sids, iters) if it == 1 and R > 1)
    # the same units set by set: one eddy_run_permutations call per set
    sids = add_all()
    torch.cuda.synchronize()
    f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for sid, it in zip(sids, iters):
        ctx.run_permutations(sid, 0, it)
    f1.record(stream)
    torch.cuda.synchronize()
    ms_per_set = f0.elapsed_time(f1)
    sizes = [len(gn) for _, gn, _ in w.sets]
    line = {"metric": METRIC, "value": units / (ms / 1e3), "unit": UNIT, "n_gpus": 1,
            "workload": f"config {args.workload}: {len(sids)} sets (sizes {min(sizes)}-"
                        f"{max(sizes)}, median {int(np.median(sizes))}) x {R} iterations "
                        f"(counter stream), {w.data.shape[0]} genes x {w.data.shape[1]} samples",
            "wall_units_per_s": units / wall, "units": units, "sets": len(sids),
            "sets_per_s": len(sids) / (ms / 1e3), "ms": ms, "launches": t["launches"],
            "stage_ms": {"k_operands+k_pairs_mma": t["ms_gemm"], "k_general+k_exact": t["ms_decide"],
                         "k_units": t["ms_units"], "k_units_js": t["ms_js"]},
            "sets_stopped_at_iteration0": stop0,
            "sets_with_all_iterations": sum(1 for it in iters if it == R),
            "per_set_value": units / (ms_per_set / 1e3),
            "batching_speedup": ms_per_set / ms}
    print(json.dumps(line), flush=True)
    ctx.close()


def run_ours(args, rank, world, local):
    import torch
    import torch.distributed as dist

    torch.cuda.set_device(local)
    if world > 1 and not dist.is_initialized():
        dist.init_process_group("nccl" if torch.cuda.is_available() else "gloo")
    import build as _build
    _build.build()
    import eddy_gpu
    from eddy_gpu import synth

    w = synth.make(4, seed=0)
    genes = w.sets[0][1]
    g, n = len(genes), w.data.shape[1]
    mp, pw = w.flags["mp"], w.flags["pw"]
    B = args.units
    seed = 4242
    ctx = eddy_gpu.Context(max_parents=mp, prior_weight=pw, permutations=B,
                           rng=eddy_gpu.RNG_COUNTER, seed=seed, device=local, keep_networks=False)
    # the library launches on this stream; the timing events are recorded on it
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.load_matrix(w.data, w.labels)
    sid = ctx.add_set(genes)
    # each rank its own permutation indices
    base = 1 + rank * (args.warmup + args.steps + 1) * B

    u_mean = []

    def step(i):
        js, U = ctx.run_permutations(sid, base + i * B, B)
        u_mean.append(float(np.mean(U)))
        t = ctx.timing()
        return t

    # clocks sampled from before the warm-up; summarised over the timed region
    clk = ClockSampler(local).__enter__()
    for i in range(args.warmup):
        step(i)
    # timed region: barrier + synchronize on both sides, events on the stream
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    acc = {"ms_pairs": 0.0, "ms_units": 0.0, "launches": 0, "ms_gemm": 0.0, "ms_decide": 0.0,
           "ms_networks": 0.0, "ms_js": 0.0}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    h0 = time.perf_counter()
    e0.record(stream)
    for i in range(args.steps):
        t = step(args.warmup + i)
        for k in acc:
            acc[k] += t[k]
    e1.record(stream)
    torch.cuda.synchronize()
    clk.mark(h0, time.perf_counter())
    clk.__exit__()
    ms = e0.elapsed_time(e1)
    stats = ctx.stats()  # decision counters of the last timed step
    if world > 1:
        dist.barrier()
        tt = torch.tensor([ms], device="cuda")
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        ms = float(tt.item())
    total_units = B * args.steps * world
    value = total_units / (ms / 1e3)

    # the plain FP64 form on the same GPU: every table decided by the
    # reference's FP64 formula (no FP32 fast path, no filter); short sample
    fp64 = None
    if not args.no_fp64:
        os.environ["EDDY_DECISIONS"] = "fp64"
        ctx.clear_sets()
        sid64 = ctx.add_set(genes)
        Bf = max(128, B // 8)
        ctx.run_permutations(sid64, base, Bf)  # warm-up
        torch.cuda.synchronize()
        f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        ctx.run_permutations(sid64, base + Bf, Bf)
        f1.record(stream)
        torch.cuda.synchronize()
        fms = f0.elapsed_time(f1)
        del os.environ["EDDY_DECISIONS"]
        ctx.clear_sets()
        fp64 = {"value": Bf / (fms / 1e3), "unit": UNIT, "units": Bf,
                "form": "same pipeline, every table decided in FP64 (reference formula), "
                        "no FP32 fast path, no leave-one-out filter"}

    # end to end through the public API with host buffers
    data_pinned = torch.from_numpy(w.data).pin_memory().numpy()
    labels_pinned = torch.from_numpy(w.labels).pin_memory().numpy()
    ectx = eddy_gpu.Context(max_parents=mp, prior_weight=pw, permutations=B,
                            rng=eddy_gpu.RNG_COUNTER, seed=seed + 1 + rank, device=local,
                            keep_networks=True)

    def e2e_step():
        ectx.clear_sets()
        ectx.load_matrix(data_pinned, labels_pinned)
        s = ectx.add_set(genes)
        ectx.run()
        js, U = ectx.js(s)
        return ectx.summary(s)

    for _ in range(max(1, args.warmup)):
        e2e_step()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    launches_e2e = 0
    for _ in range(args.steps):
        e2e_step()
        launches_e2e += ectx.timing()["launches"]
    torch.cuda.synchronize()
    e2e_s = time.perf_counter() - t0
    if world > 1:
        tt = torch.tensor([e2e_s], device="cuda")
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        e2e_s = float(tt.item())
    e2e_value = B * args.steps * world / e2e_s
    W = (n + 63) // 64
    h2d = w.data.size + n + 8 * B
    d2h = 16 * B

    if rank != 0:
        return
    hbm, bf16, peak_kind = load_peaks()
    U_mean = float(np.mean(u_mean[-args.steps:]))
    bu = required_bytes(g, n)
    c = g * (g - 1) // 2
    # a step's units run as equal batches of at most 2^28 / (2 c) units (the
    # library's general-path queue holds every table of a batch): one launch
    # of each kernel per batch
    batches = -(-B // min(32768, (1 << 28) // (2 * c)))
    launches_per_kernel = args.steps * batches
    Bl = B / batches  # units per launch
    traffic_info = {}
    tf = os.path.join(ROOT, "profiles", "traffic_config4.json")
    if os.path.exists(tf):
        with open(tf) as f:
            traffic_info = json.load(f)
    # contingency GEMM + decisions on the tensor cores: useful GEMM work is
    # 2 x (cells x c pairs) x n samples per unit (0/1 e4m3, FP32 accumulate),
    # with 4 counted cells per table when the set has no missing value (the
    # epilogue derives the other five from the genes' class counts) and 9
    # otherwise; the dense e4m3 peak is twice the measured dense bf16 one
    core = bool(np.isin(w.data[np.asarray(genes)], (-1, 0, 1)).all()) and \
        os.environ.get("EDDY_PAIR_LAYOUT") != "full"
    cells = 4 if core else 9
    # each kernel's own device time (CUDA events between the launches on
    # the library's stream): operands + contraction; then the decisions the
    # epilogue's bound leaves (k_general + k_exact) apart
    k1_ms = acc["ms_gemm"] / launches_per_kernel
    # algorithmic work of the contraction: 2 (3g)^2 n_A per unit (the class-A
    # Gram matrix of the genes' state indicators); the GEMM the kernel runs
    # is smaller: 2 x cells x c x n per unit
    nA = int((np.asarray(w.labels) == 0).sum())
    k1_flops = 2.0 * (3 * g) ** 2 * nA * Bl
    k1_gemm = 2.0 * cells * c * n * Bl
    e4m3 = 2.0 * bf16
    k1 = {"kernel": "k_pairs_mma", "bound": "tensor", "achieved": k1_flops / (k1_ms / 1e3) / 1e12,
          "peak": e4m3, "unit": "TFLOP/s", "ms_per_launch": k1_ms,
          "algorithmic_flops_per_launch": k1_flops,
          "layout": f"{cells} counted cells per table",
          "gemm_flops_per_launch": k1_gemm,
          "gemm_frac": k1_gemm / (k1_ms / 1e3) / 1e12 / e4m3,
          "traffic": traffic_info.get("k_pairs_mma_bytes_per_unit", 0) * Bl or None,
          "units_per_launch": Bl,
          "ncu_sm_throughput_pct": traffic_info.get("k_pairs_mma_sm_throughput_pct"),
          "ncu_tensor_pipe_pct": traffic_info.get("k_pairs_mma_tensor_pipe_pct")}
    k1["frac"] = k1["achieved"] / e4m3
    # networks, dedup, BDeu, JS: bound by the SMs' issue slots, not by bytes
    # (which are reported beside it): warp instructions per unit as ncu counts
    # them, against four a cycle and SM at the sampled clock
    k2_ms = acc["ms_units"] / launches_per_kernel
    insts = traffic_info.get("k_units_warp_instructions_per_unit", 0) * Bl
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    issue = 4.0 * sms * (clk.summary().get("sm_mhz") or 2070.0) / 1e3
    k2 = {"kernel": "k_units", "bound": "issue", "achieved": insts / (k2_ms / 1e3) / 1e9,
          "peak": issue, "unit": "G warp instructions/s", "ms_per_launch": k2_ms,
          "warp_instructions_per_launch": insts, "required_bytes_per_launch": bu * Bl,
          "required_bytes_hbm_frac": bu * Bl / (k2_ms / 1e3) / 1e9 / hbm,
          "unique_networks_per_unit": U_mean, "units_per_launch": Bl,
          "traffic": traffic_info.get("k_units_bytes_per_unit", 0) * Bl or None,
          "ncu_sm_throughput_pct": traffic_info.get("k_units_sm_throughput_pct"),
          "ncu_issue_active_pct": traffic_info.get("k_units_issue_active_pct")}
    k2["frac"] = k2["achieved"] / issue
    dom = k1 if k1_ms >= k2_ms else k2
    roofline = dict(dom)
    roofline["peak_source"] = (f"2 x MEASURED_PEAKS.json bf16_tflops ({peak_kind}): the GEMM "
                               "runs e4m3 operands, whose dense peak is twice the bf16 one"
                               if dom is k1 else "four warp instructions a cycle and SM at the sampled clock")
    cpu = None
    precision = {"tables": int(stats["tables"]), "filtered": int(stats["filtered"]),
                 "exact_rechecks": int(stats["exact_rechecks"])}
    # near-threshold share of the pair tests: the unpermuted labelling and
    # the sampled permutations (host numpy; a property of the workload)
    import oracle
    R_s = args.cpu_units + 1
    labs = oracle.counter_labels(seed, 0, w.labels, R_s)
    near = synth.near_threshold(w.data[genes], labs)
    if world == 1 and not args.no_cpu:
        try:
            cu, cs, ojs, oU = cpu_sample(w, genes, seed, 0, R_s, os.cpu_count() or 1)
            cpu = {"value": cu, "unit": UNIT, "cores": os.cpu_count() or 1, "kind": "port",
                   "sample": f"{R_s} labellings of the same set: the unpermuted one and "
                             f"{args.cpu_units} permutations ({cs:.1f} s)"}
            precision.update(precision_vs_oracle(eddy_gpu, oracle, w, genes, seed, labs, ojs, oU))
        except Exception as e:  # pragma: no cover - reported, not hidden
            cpu = {"value": None, "unit": UNIT, "cores": 0, "kind": "port", "sample": f"failed: {e}"}
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u8/i32 counts, f32 decisions + f64 rechecks",
            "data": "synthetic (seeded, shapes of the precision-stress workload)",
            "config": {"workload": WORKLOAD, "units_per_step": B, "genes": g, "samples": n,
                       "max_parents": mp, "rng": "counter (Philox-4x32-10, on device)",
                       "near_threshold": {
                           "p_band": near["p_band"], "chi2_band": near["chi2_band"],
                           "tests": near["tests"],
                           "definition": "share of (pair, class) tests of the unpermuted labelling "
                                         "and the sampled permutations whose Bonferroni-adjusted p is "
                                         "within +-20% of 0.05 (p_band), or whose chi-square is within "
                                         "+-20% of the critical chi-square (chi2_band)"},
                       "l2": "per-launch working set (decision masks + per-unit scratch) "
                             f"~{(Bl * c * 4 + 1.5e9) / 1e9:.2f} GB > L2"},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h},
            "gpu_launches": acc["launches"],
            "stage_ms": {"k_operands+k_pairs_mma": acc["ms_gemm"],
                         "k_general+k_exact": acc["ms_decide"], "k_units": acc["ms_units"],
                         "k_units_js": acc["ms_js"], "steps": args.steps},
            "roofline": roofline,
            "kernels": {"k_pairs_mma": k1, "k_units": k2},
            "clocks": clk.summary(),
            "plain_fp64_form": fp64,
            "vs_plain_fp64": (value / world / fp64["value"]) if fp64 else None,
            "precision": precision,
            "cpu_baseline": cpu}
    print(json.dumps(line), flush=True)
    ctx.close()
    ectx.close()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--units", type=int, default=10000, help="permutations per step")
    ap.add_argument("--cpu-units", type=int, default=8, help="permutations in the CPU sample")
    ap.add_argument("--ref-units", type=int, default=2,
                    help="permutations per step of the reference arm")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--workload", type=int, default=4, choices=[3, 4, 5],
                    help="3 or 5: multi-set sample (prints its own line)")
    ap.add_argument("--sets", type=int, default=100)
    ap.add_argument("--perms", type=int, default=0)
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    rank, world, local = dist_env()
    if args.impl == "reference":
        run_reference(args, rank, world)
    elif args.workload != 4:
        run_multiset(args, rank, world, local)
    else:
        run_ours(args, rank, world, local)


if __name__ == "__main__":
    main()
