"""Benchmark: harmonic-mean GTEPS over 64 roots on a seeded RMAT scale-24 graph.

One "step" is one pass of the hot path over one batch of synthetic input: a
BFS from each of 64 roots (lcg(0) picker of hybrid_bfs_main.cc:136-144) on a
seeded RMAT scale-24 graph (A=.57 B=.19 C=.19 D=.05, edge factor 16,
deduplicated, symmetrised; int64 offsets, uint32 ids), generated on the
device.  Per root, time covers run_* only, as in the reference
(hybrid_bfs_main.cc:267-282): clear() is outside, the source setup inside,
and so is the writing of every root's results (int32 depths and int64
parents, caller ids, the reference's encoding: run_beamer leaves parent_
complete).  TEPS = count_num_traversed_edges() / time; the metric is the
harmonic mean of the per-root GTEPS (combined.cc:124-128).  A batched group's
time is spread evenly over its roots.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (torchrun, one rank per GPU) every rank runs an independent
replica on its own 64 roots (lcg(rank)); there is no collective on the data
path.  value = N x harmonic mean over all ranks' roots, timed as the max over
ranks.

--impl reference times the reference's own CPU build (oracle/_ref/hybrid_bfs,
the unmodified hybrid_bfs sources compiled as a Cilk serial elision: 1 core)
on the same graph, written as an el64 file by a child process, over a
bounded sample of roots (8 per step).
"""
from __future__ import annotations

import argparse
import json
import os
import re
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "harmonic-mean GTEPS over 64 roots, RMAT scale 24, learned vs plain switch, 1 B200"
UNIT = "GTEPS"
SCALE = 24
EDGE_FACTOR = 16
GRAPH_SEED = 24
NUM_ROOTS = 64
REF_BIN = os.path.join(ROOT, "oracle", "_ref", "hybrid_bfs")
REF_CC_BIN = os.path.join(ROOT, "oracle", "_ref", "components")


def hmean(x):
    x = np.asarray(x, np.float64)
    return float(len(x) / np.sum(1.0 / x))


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle samples while the timed region runs."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.thread.join(timeout=2)

    def summary(self):
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = max(mx, float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx or None,
                "reasons": sorted(reasons), "samples": len(sm)}


def reduce_over_ranks(step_ms: float, value: float, e2e: float, device=None):
    """Replicas: every rank ran its own roots.  The step time is the slowest
    rank's; the whole-job throughput is world x the slowest rank's (so a
    fast rank cannot hide a slow one).  One all_reduce(MAX); `device` is the
    rank's GPU under NCCL, None (CPU tensors) under gloo."""
    import torch
    import torch.distributed as dist
    world = dist.get_world_size()
    t = torch.tensor([step_ms, -value, -e2e], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t[0]), world * -float(t[1]), world * -float(t[2])


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def reference_cpu_run(el64_path: str, trials: int, timeout: float):
    """Runs the reference CLI (serial elision, one core) and returns the
    per-trial (edges, ms) it prints (hybrid_bfs_main.cc:297-301)."""
    cmd = [REF_BIN, "--graph_filename", el64_path, "--algorithm", "beamer_hybrid",
           "--num_trials", str(trials)]
    try:
        cmd = ["taskset", "-c", str(max(0, (os.cpu_count() or 1) - 1))] + cmd
        out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                             timeout=timeout).stdout
    except (subprocess.TimeoutExpired, FileNotFoundError, OSError) as e:
        return None, str(e)
    rows = [(int(a), float(b)) for a, b in
            re.findall(r"Traversed (\d+) edges in ([0-9.]+) ms", out)]
    return rows, out[-400:]


REF_ROOTS_PER_STEP = 8
# B200 HBM3e nominal bandwidth (HGX figure), reported beside the measured peak
HBM_NOMINAL_GBS = 7700.0


def workload_config(desc: str, num_roots: int, scale, graph_seed: int, n: int, m: int) -> dict:
    """The `config` object of a graph workload: what was run, nothing about
    how.  Both arms print the same object for the same workload."""
    return {
        "workload": f"{desc}, {num_roots} roots per step",
        "scale": scale, "edge_factor": EDGE_FACTOR if scale else None, "graph_seed": graph_seed,
        "num_vertices": n, "num_edges": m, "roots": num_roots, "root_seed": 0,
        "l2": "inputs larger than L2 (CSR %.2f GB), and L2 flushed (512 MB write) before "
              "each way's runs on the GPU" % ((8 * (n + 1) + 8 * m) / 1e9),
    }


def write_graph_el64(path: str, scale: int) -> int:
    """Writes the benchmark graph as an el64 file from a child process, so
    the process that times the reference maps none of this repository's
    native code.  Returns the child's exit code."""
    code = ("import sys; sys.path.insert(0, %r); import beedrill_b200 as bd; "
            "g = bd.Graph.rmat(%d, %d, seed=%d); g.write_el64(%r); "
            "print(g.num_vertices(), g.num_edges())" % (ROOT, scale, EDGE_FACTOR, GRAPH_SEED, path))
    out = subprocess.run([sys.executable, "-c", code], stdout=subprocess.PIPE,
                         stderr=subprocess.STDOUT, text=True, timeout=1800)
    return out.returncode, out.stdout.strip().splitlines()[-1:] or [""]


def impl_reference(args):
    """The reference's own CPU build (oracle/_ref/hybrid_bfs: the unmodified
    hybrid_bfs sources compiled as a Cilk serial elision, one pinned core)
    on the benchmark graph.  One step = a bounded sample of the workload:
    REF_ROOTS_PER_STEP roots of the lcg(0) sequence, in the order the GPU
    arm takes them (warm-up steps first)."""
    world, rank, local = dist_setup()
    if rank != 0:
        return 0
    if not os.path.exists(REF_BIN):
        print(json.dumps({"impl": "reference", "unavailable":
                          "oracle/_ref/hybrid_bfs was not built (reference sources absent at build time)"}))
        return 0
    with tempfile.TemporaryDirectory(dir=os.environ.get("BD_TMP", None)) as tmp:
        path = os.path.join(tmp, f"rmat{SCALE}.el64")
        rc, last = write_graph_el64(path, SCALE)
        if rc != 0:
            print(json.dumps({"impl": "reference",
                              "unavailable": f"graph generation failed: {last[0][-200:]}"}))
            return 0
        n, m = (int(x) for x in last[0].split())
        trials = (args.warmup + args.steps) * REF_ROOTS_PER_STEP
        t0 = time.time()
        rows, tail = reference_cpu_run(path, trials, timeout=3000)
        wall = time.time() - t0
    if not rows or len(rows) < trials:
        print(json.dumps({"impl": "reference", "unavailable": f"reference run failed: {tail}"}))
        return 0
    timed = rows[args.warmup * REF_ROOTS_PER_STEP:]
    gteps = [e / (ms * 1e-3) / 1e9 for e, ms in timed]
    value = hmean(gteps)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": float(np.sum([ms for _, ms in timed]) / args.steps),
        "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "i64", "data": "synthetic",
        "config": workload_config(f"rmat-scale{SCALE}-ef{EDGE_FACTOR} seed {GRAPH_SEED}",
                                  NUM_ROOTS, SCALE, GRAPH_SEED, n, m),
        "run": {"results": "parent_ complete per root (the reference's run_beamer)",
                "roots_per_step": REF_ROOTS_PER_STEP,
                "parallelism": "host CPU, 1 pinned core (serial elision; rank 0 only)"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": 1, "kind": "reference",
                         "sample": f"each step {REF_ROOTS_PER_STEP} lcg(0) roots of the "
                                   f"{NUM_ROOTS}-root workload: {len(timed)} timed roots after "
                                   f"{args.warmup * REF_ROOTS_PER_STEP} warm-up roots, "
                                   f"reference serial-elision build on 1 pinned core; process "
                                   f"wall {wall:.0f} s incl. el64 load + graph build"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


DEFAULT_MODES = "plain,learned,batched,batched_rule,plain_traversal,batched_traversal"

WORKLOADS = {
    # the headline: RMAT scale 24, 64 roots
    "rmat24": {"kind": "rmat", "scale": 24, "roots": 64},
    # plain Beamer, one root per launch, at scale 22
    "rmat22": {"kind": "rmat", "scale": 22, "roots": 64},
    # 256 roots in four 64-lane groups of one captured launch
    "rmat20-256": {"kind": "rmat", "scale": 20, "roots": 256},
    # the largest single-GPU case (materialized rows of 64 roots take 51.5 GB,
    # so only the batched way keeps every root's results)
    "rmat26": {"kind": "rmat", "scale": 26, "roots": 64, "modes": "batched,plain_traversal"},
    # graphs inside the learned policies' training range (scales 16-18),
    # seeds the trainer never used: 64-root batches, learned vs rule
    "policy16-18": {"kind": "policy_set", "scales": (16, 17, 18), "seeds": (7001, 7002, 7003)},
    # high-diameter contrast: 4096 x 4096 grid, 1% of its edges deleted
    "grid4096": {"kind": "grid", "rows": 4096, "cols": 4096, "delete": 0.01, "roots": 64,
                 "modes": "plain,batched,batched_rule"},
    # 512 independent RMAT graphs (scales 10-18, edge factors 4-32), one root each
    "packed512": {"kind": "packed", "graphs": 512},
    # connected components (components.cc) on the same RMAT scale-24 graph
    "components24": {"kind": "components", "scale": 24, "cpu_scale": 20},
}


def packed_parts(bd, count: int, order: int):
    """The packed-graphs workload: seeded scales 10-18 and edge factors
    4-32, graph i generated with seed 5000 + i, root lcg(i) of graph i."""
    rng = np.random.default_rng(512)
    scales = rng.integers(10, 19, count)
    factors = rng.integers(4, 33, count)
    return [bd.Graph.rmat(int(s), int(f), seed=5000 + i, order=order)
            for i, (s, f) in enumerate(zip(scales, factors))]


def bench_packed(args, w, bd, order, local):
    """512 graphs packed into one CSR: one multi-source launch over all of
    them ("batched") against one launch per graph on its own CSR ("plain").
    GTEPS = sum of m_c over all graphs / time of the step."""
    t_gen = time.time()
    parts = packed_parts(bd, w["graphs"], order)
    g, base = bd.Graph.concat(parts)
    gen_s = time.time() - t_gen
    roots = np.array([int(p.pick_roots(i, 1)[0]) + int(base[i]) for i, p in enumerate(parts)],
                     np.int64)
    n, m = g.num_vertices(), g.num_edges()
    multi = bd.HybridBFS(g)
    singles = [bd.HybridBFS(p) for p in parts]

    import torch
    flush_buf = torch.empty(512 << 20, dtype=torch.uint8, device=f"cuda:{local}")

    def flush_l2():  # > the 126 MB L2, before each way's runs
        flush_buf.fill_(1)
        torch.cuda.synchronize(local)

    def one_step():
        flush_l2()
        t0 = time.perf_counter()
        multi.clear()
        st = multi.run_multi(roots)
        edges = multi.count_num_traversed_edges()
        wall_multi = (time.perf_counter() - t0) * 1e3
        ms_multi = st.ms
        flush_l2()
        t0 = time.perf_counter()
        ms_single, edges_single = 0.0, 0
        for i, (h, p) in enumerate(zip(singles, parts)):
            h.clear()
            ms_single += h.run(int(roots[i] - base[i])).ms
            edges_single += h.count_num_traversed_edges()
        wall_single = (time.perf_counter() - t0) * 1e3
        return {"batched": (ms_multi, edges, wall_multi), "plain": (ms_single, edges_single, wall_single)}

    for _ in range(args.warmup):
        one_step()
    runs = []
    with ClockSampler(local) as clocks:
        for _ in range(args.steps):
            runs.append(one_step())
    modes = {}
    for name in ("batched", "plain"):
        ms = np.array([r[name][0] for r in runs])
        edges = np.array([r[name][1] for r in runs])
        wall = np.array([r[name][2] for r in runs])
        modes[name] = {"gteps": float(edges.sum() / (ms.sum() * 1e-3) / 1e9),
                       "e2e_gteps": float(edges.sum() / (wall.sum() * 1e-3) / 1e9),
                       "ms_per_step": float(ms.mean()), "edges": int(edges[0])}
    if modes["batched"]["edges"] != modes["plain"]["edges"]:
        raise RuntimeError("packed and per-graph runs disagree on m_c")
    head = modes["batched"]
    peak, peak_kind = peaks()
    # one pass over the packed CSR plus every vertex's depth and parent
    b_alg = 8.0 * (n + 1) + 8.0 * m + 12.0 * n
    achieved = b_alg / (head["ms_per_step"] * 1e-3) / 1e9
    line = {
        "metric": f"aggregate GTEPS, {w['graphs']} packed RMAT graphs (scales 10-18), one root each, 1 B200",
        "value": head["gteps"], "unit": UNIT, "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": head["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
        "config": {"workload": args.workload, "graphs": w["graphs"], "num_vertices": n,
                   "num_edges": m, "adjacency_order": args.order,
                   "l2": "inputs larger than L2 (CSR %.2f GB)" % ((8 * (n + 1) + 8 * m) / 1e9),
                   "graph_build_s": round(gen_s, 2), "parallelism": "1 GPU"},
        "modes": {k: {kk: vv for kk, vv in v.items() if kk != "edges"} for k, v in modes.items()},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": None, "peak_kind": peak_kind,
                     "note": "B_alg = 8(n+1) + 8m + 12n per multi-source launch"},
        "e2e": {"value": head["e2e_gteps"], "unit": UNIT, "h2d_bytes_per_step": 8 * len(roots),
                "d2h_bytes_per_step": 8,
                "note": "public API calls per step: clear, run_multi (root upload), m_c download"},
        # clear and search: of the packed graph, and of each part
        "gpu_launches": args.steps * (2 + 2 * len(parts)),
        "clocks": clocks.summary(),
    }
    print(json.dumps(line))
    multi.close()
    for h in singles:
        h.close()
    return 0


def reference_components_run(el64_path: str, trials: int, timeout: float):
    """Runs the reference's components CLI (serial elision, one pinned core)
    and returns per-trial (components, iterations, ms) (components_main.cc:180-181)."""
    cmd = ["taskset", "-c", str(max(0, (os.cpu_count() or 1) - 1)), REF_CC_BIN,
           "--graph_filename", el64_path, "--num_trials", str(trials)]
    try:
        out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                             timeout=timeout).stdout
    except (subprocess.TimeoutExpired, FileNotFoundError, OSError) as e:
        return None, str(e)
    rows = [(int(a), int(b), float(c)) for a, b, c in
            re.findall(r"Found (\d+) components in (\d+) iterations \(([0-9.]+) ms", out)]
    return rows, out[-400:]


def bench_components(args, w, bd, local):
    """Connected components of the RMAT scale-24 graph.  One step = one
    components run (labels, sizes, count).  GTEPS = iterations x edges / time
    as the reference prints it (components_main.cc:179); one iteration here.
    The CPU baseline is the reference's own components build on a scale-20
    graph of the same generator (its label propagation would take minutes at
    scale 24 on one core)."""
    import torch
    scale = args.scale or w["scale"]
    t_gen = time.time()
    g = bd.Graph.rmat(scale, EDGE_FACTOR, seed=GRAPH_SEED if scale == SCALE else scale)
    gen_s = time.time() - t_gen
    n, m = g.num_vertices(), g.num_edges()
    cc = bd.Components(g)
    flush_buf = torch.empty(512 << 20, dtype=torch.uint8, device=f"cuda:{local}")

    def flush_l2():  # > the 126 MB L2 before every timed run
        flush_buf.fill_(1)
        torch.cuda.synchronize(local)

    labels = np.empty(n, np.int64)
    lab_ptr = labels.ctypes.data_as(bd.ctypes.POINTER(bd.ctypes.c_int64))
    for _ in range(args.warmup):
        flush_l2()
        cc.run()
    ok = cc.check()
    ms, wall, counts = [], [], set()
    with ClockSampler(local) as clocks:
        for _ in range(args.steps):
            flush_l2()
            t0 = time.perf_counter()
            st = cc.run()
            if bd.lib().bd_components_get_labels(cc._h, lab_ptr) != 0:
                raise RuntimeError("label copy failed")
            wall.append((time.perf_counter() - t0) * 1e3)
            ms.append(st.ms)
            counts.add(st.num_components)
    if not ok or len(counts) != 1:
        raise RuntimeError("components check failed or counts differ between runs")
    ms_step = float(np.mean(ms))
    value = m / (ms_step * 1e-3) / 1e9
    e2e = m / (float(np.mean(wall)) * 1e-3) / 1e9
    peak, peak_kind = peaks()
    b_alg = 8.0 * (n + 1) + 8.0 * m + 4.0 * n + 16.0 * n
    achieved = b_alg / (ms_step * 1e-3) / 1e9
    cpu = None
    if not args.no_cpu_baseline and os.path.exists(REF_CC_BIN):
        cs = w["cpu_scale"]
        gs = bd.Graph.rmat(cs, EDGE_FACTOR, seed=cs)
        ms_cpu = None
        with tempfile.TemporaryDirectory(dir=os.environ.get("BD_TMP", None)) as tmp:
            path = os.path.join(tmp, f"rmat{cs}.el64")
            gs.write_el64(path)
            rows, _ = reference_components_run(path, 2, timeout=600)
        if rows:
            ms_cpu = rows[-1][2]
            cpu = {"value": gs.num_edges() / (ms_cpu * 1e-3) / 1e9, "unit": UNIT, "cores": 1,
                   "kind": "reference",
                   "sample": f"reference components build (serial elision, 1 pinned core) on "
                             f"RMAT scale {cs} (seed {cs}): {rows[-1][0]} components, "
                             f"{rows[-1][1]} label-propagation iterations, {ms_cpu:.0f} ms; "
                             f"value = edges / time (its own printout multiplies by iterations)"}
        gs.close()
    line = {
        "metric": f"connected components, edges / run time, RMAT scale {scale}, 1 B200",
        "value": value, "unit": UNIT, "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "u32", "data": "synthetic",
        "config": {"workload": args.workload, "scale": scale, "edge_factor": EDGE_FACTOR,
                   "num_vertices": n, "num_edges": m, "components": counts.pop(),
                   "l2": "flushed (512 MB write) before every run; CSR %.2f GB" %
                         ((8 * (n + 1) + 8 * m) / 1e9),
                   "graph_build_s": round(gen_s, 2), "check": ok, "parallelism": "1 GPU"},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": None, "peak_kind": peak_kind,
                     "note": "B_alg = 8(n+1) + 4*2m + 4n (forest) + 16n (labels, sizes) per run"},
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 8 * n,
                "note": "public API per step: run, then the int64 labels copied to the host"},
        "cpu_baseline": cpu,
        # hooks, three merges, four flattens, two probes, walk, two for heavy lists, labels
        "gpu_launches": 14 * args.steps,
        "clocks": clocks.summary(),
    }
    print(json.dumps(line))
    cc.close()
    g.close()
    return 0


def bench_policy_set(args, w, bd, order, local):
    """Held-out graphs of the learned policies' training range (RMAT A=.57
    B=C=.19 D=.05, edge factor 16, graph seeds the trainer never used), one
    64-root batch each, with the learned push/pull policy ("batched") and
    with the rule alone ("batched_rule").  GTEPS = sum of m_c over all
    roots of all graphs / sum of the batch times."""
    from beedrill_b200 import policy as P
    import torch
    flush_buf = torch.empty(512 << 20, dtype=torch.uint8, device=f"cuda:{local}")

    def flush_l2():  # > the 126 MB L2, before each batch
        flush_buf.fill_(1)
        torch.cuda.synchronize(local)

    pol = P.Policy.load(P.BATCHED_PATH)
    graphs = []
    for scale in w["scales"]:
        for seed in w["seeds"]:
            g = bd.Graph.rmat(scale, EDGE_FACTOR, 0.57, 0.19, 0.19, 0.05, seed + 10 * scale,
                              order=order)
            learned, rule = bd.BatchedBFS(g, 64), bd.BatchedBFS(g, 64)
            pol.install(learned)
            graphs.append((g, g.pick_roots(seed, 64), learned, rule))
    totals = {"batched": [0.0, 0], "batched_rule": [0.0, 0]}
    dirs = {}
    with ClockSampler(local) as clocks:
        for step in range(args.warmup + args.steps):
            for g, roots, learned, rule in graphs:
                for name, h in (("batched", learned), ("batched_rule", rule)):
                    flush_l2()
                    st = h.run(roots)
                    if step >= args.warmup:
                        totals[name][0] += st.ms
                        totals[name][1] += int(h.counts()[0].sum())
                        dirs.setdefault(name, []).append(h.directions())
    modes = {k: {"gteps": e / (ms * 1e-3) / 1e9, "ms_per_step": ms / args.steps}
             for k, (ms, e) in totals.items()}
    line = {
        "metric": "aggregate GTEPS, 64-root batches on 9 held-out RMAT graphs (scales 16-18), "
                  "learned push/pull policy vs rule, 1 B200",
        "value": modes["batched"]["gteps"], "unit": UNIT, "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": modes["batched"]["ms_per_step"],
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32",
        "data": "synthetic",
        "config": {"workload": args.workload, "scales": list(w["scales"]),
                   "graph_seeds": [s + 10 * sc for sc in w["scales"] for s in w["seeds"]],
                   "roots": 64, "adjacency_order": args.order,
                   "l2": "L2 flushed (512 MB write) before each batch", "parallelism": "1 GPU"},
        "modes": modes,
        "directions": {k: sorted(set(v)) for k, v in dirs.items()},
        # clear, init, traversal and per-lane counts of each batch
        "gpu_launches": args.steps * 2 * len(graphs) * 4,
        "clocks": clocks.summary(),
    }
    print(json.dumps(line))
    for g, _, learned, rule in graphs:
        learned.close()
        rule.close()
        g.close()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="rmat24", choices=sorted(WORKLOADS),
                    help="rmat24 is the headline; the others are the remaining evaluation cases")
    ap.add_argument("--scale", type=int, default=None, help="override the RMAT scale")
    ap.add_argument("--modes", default=None,
                    help="subset of plain,learned,batched,batched_rule,plain_traversal,"
                         "batched_traversal to run (default: the workload's set; profiling "
                         "runs use one, to hold only that handle on the device)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-roots", type=int, default=8)
    ap.add_argument("--order", default="hub", choices=["insertion", "sorted", "degree", "hub"],
                    help="adjacency order / numbering the kernels run on (same results for all)")
    args = ap.parse_args()
    if args.impl == "reference":
        return impl_reference(args)

    world, rank, local = dist_setup()
    import beedrill_b200 as bd
    if world > 1:
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=600))
    bd.lib().bd_set_device(local)

    w = dict(WORKLOADS[args.workload])
    order = {"insertion": bd.ORDER_INSERTION, "sorted": bd.ORDER_SORTED,
             "degree": bd.ORDER_DEGREE, "hub": bd.ORDER_HUB}[args.order]
    if w["kind"] == "packed":
        if world > 1:
            raise SystemExit("packed512 runs on one GPU")
        return bench_packed(args, w, bd, order, local)
    if w["kind"] == "policy_set":
        if world > 1:
            raise SystemExit("policy16-18 runs on one GPU")
        return bench_policy_set(args, w, bd, order, local)
    if w["kind"] == "components":
        if world > 1:
            raise SystemExit("components24 runs on one GPU")
        return bench_components(args, w, bd, local)
    num_roots = w["roots"]
    t_gen = time.time()
    if w["kind"] == "rmat":
        scale = args.scale or w["scale"]
        g = bd.Graph.rmat(scale, EDGE_FACTOR, seed=GRAPH_SEED if scale == SCALE else scale,
                          order=order)
        graph_seed = GRAPH_SEED if scale == SCALE else scale
        desc = f"rmat-scale{scale}-ef{EDGE_FACTOR} seed {graph_seed}"
        metric = METRIC if (scale == SCALE and num_roots == NUM_ROOTS) else \
            f"harmonic-mean GTEPS over {num_roots} roots, RMAT scale {scale}, 1 B200"
    else:
        scale = None
        graph_seed = 0
        g = bd.Graph.grid(w["rows"], w["cols"], w["delete"], graph_seed, order=order)
        desc = f"grid {w['rows']}x{w['cols']}, {w['delete']:.0%} of edges deleted, seed {graph_seed}"
        metric = f"harmonic-mean GTEPS over {num_roots} roots, {desc}, 1 B200"
    gen_s = time.time() - t_gen
    n, m = g.num_vertices(), g.num_edges()
    roots = g.pick_roots(rank, num_roots)

    # CPU baseline: the reference's own build on a bounded sample of the same
    # workload (rank 0, N = 1), run after the GPU's timed region, not beside it.
    el64 = None
    tmpdir = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline and os.path.exists(REF_BIN) \
            and m <= 300_000_000:
        tmpdir = tempfile.TemporaryDirectory(dir=os.environ.get("BD_TMP", None))
        el64 = os.path.join(tmpdir.name, "graph.el64")
        g.write_el64(el64)

    # The ways of running the roots.  Materialized (what a caller gets: every
    # root's int32 depths and int64 parents in caller ids and the reference's
    # encoding, in device memory, when the step ends):
    #   plain         one launch per root, Beamer alpha=15 / beta=18
    #   learned       one launch per root, the learned top-down/bottom-up policy
    #   batched       64 roots per group, one captured launch, learned push/pull
    #   batched_rule  the same under the alpha rule alone
    # Traversal only (results left in the kernels' own form, as before):
    #   plain_traversal, batched_traversal
    want = [x for x in (args.modes or w.get("modes", DEFAULT_MODES)).split(",") if x]
    from beedrill_b200 import policy as P
    import torch
    dev = f"cuda:{local}"
    handles = {}
    if any(x in want for x in ("plain", "plain_traversal")):
        handles["plain"] = bd.HybridBFS(g, alg="beamer_hybrid")
    if "learned" in want and os.path.exists(P.DEFAULT_PATH):
        handles["learned"] = bd.HybridBFS(g, alg="learned")
        P.Policy.load().install(handles["learned"])
    for name, mat, pol in (("batched", True, True), ("batched_rule", True, False),
                           ("batched_traversal", False, True)):
        if name in want:
            handles[name] = bd.BatchedBFS(g, num_roots, materialize=mat)
            if pol and os.path.exists(P.BATCHED_PATH):
                P.Policy.load(P.BATCHED_PATH).install(handles[name])
    out_depth = out_parent = None
    if any(x in want for x in ("plain", "learned")):
        out_depth = torch.empty((num_roots, n), dtype=torch.int32, device=dev)
        out_parent = torch.empty((num_roots, n), dtype=torch.int64, device=dev)
    groups = (num_roots + 63) // 64

    # A 512 MB write (> the 126 MB L2) before each way's runs, so that no
    # way starts with another's graph or state in cache.
    flush_buf = torch.empty(512 << 20, dtype=torch.uint8, device=dev)

    def flush_l2():
        flush_buf.fill_(1)
        torch.cuda.synchronize(local)

    def run_way(name):
        if name in ("plain", "learned"):
            h = handles[name]
            ms, edges, reached, _ = h.run_many_into(roots, out_depth.data_ptr(),
                                                    out_parent.data_ptr())
            return ms, edges, reached
        if name == "plain_traversal":
            ms, edges, reached, _ = handles["plain"].run_many(roots, with_reached=True)
            return ms, edges, reached
        h = handles[name]
        st = h.run(roots)
        m_c, n_c = h.counts()
        return np.full(num_roots, st.ms / num_roots), m_c, n_c

    order_run = [x for x in ("plain", "learned", "plain_traversal", "batched", "batched_rule",
                             "batched_traversal")
                 if x in want and (x in handles or x == "plain_traversal" and "plain" in handles)]

    def one_step():
        out = {}
        for name in order_run:
            flush_l2()
            out[name] = run_way(name)
        return out

    # e2e: the public call a user makes, host buffers in and out: roots
    # uploaded by the call, the run, m_c / n_c read back, and every root's
    # parent array (int64, n entries) copied to pinned host memory.
    e2e_ways = [x for x in ("batched", "plain") if x in order_run]
    rows_bytes = 8 * n * num_roots
    host_rows = torch.empty((num_roots if rows_bytes <= (16 << 30) else 1, n), dtype=torch.int64,
                            pin_memory=True) if e2e_ways else None

    def e2e_step(name):
        flush_l2()
        t0 = time.perf_counter()
        if name == "batched":
            h = handles[name]
            h.run(roots)
            m_c, _ = h.counts()
            for i in range(num_roots):
                row = host_rows[i % host_rows.shape[0]]
                h.parents_to(i, row.data_ptr())
        else:
            _, m_c, _, _ = handles["plain"].run_many_into(roots, out_depth.data_ptr(),
                                                          out_parent.data_ptr())
            if host_rows.shape[0] == num_roots:
                host_rows.copy_(out_parent, non_blocking=False)
            else:
                for i in range(num_roots):
                    host_rows[0].copy_(out_parent[i], non_blocking=False)
        torch.cuda.synchronize(local)
        return m_c, (time.perf_counter() - t0) * 1e3

    for _ in range(args.warmup):
        one_step()
        for name in e2e_ways:
            e2e_step(name)

    def barrier():
        if world > 1:
            dist.barrier()

    barrier()
    torch.cuda.synchronize(local)
    runs, e2e_runs = [], {name: [] for name in e2e_ways}
    with ClockSampler(local) as clocks:
        for _ in range(args.steps):
            runs.append(one_step())
        for _ in range(args.steps):
            for name in e2e_ways:
                e2e_runs[name].append(e2e_step(name))
    torch.cuda.synchronize(local)
    barrier()

    def summarize(name):
        ms = np.concatenate([r[name][0] for r in runs])
        edges = np.concatenate([r[name][1] for r in runs])
        reached = np.concatenate([r[name][2] for r in runs])
        gteps = edges / (ms * 1e-3) / 1e9
        step_ms = float(np.mean([r[name][0].sum() for r in runs]))
        if name.startswith("batched"):
            # one shared CSR pass per 64-root group, plus every root's depth
            # and parent outputs, spread evenly over the group's roots
            per_root = np.zeros(len(reached))
            for s0 in range(0, len(reached), num_roots):
                for g0 in range(0, num_roots, 64):
                    lo, hi = s0 + g0, s0 + min(g0 + 64, num_roots)
                    b = 8.0 * (n + 1) + 8.0 * m + 12.0 * reached[lo:hi].sum()
                    per_root[lo:hi] = b / (hi - lo)
            b_alg = per_root
        else:
            b_alg = 8.0 * (n + 1) + 8.0 * edges + 12.0 * reached
        out = {"gteps": hmean(gteps), "step_ms": step_ms, "ms": ms, "edges": edges,
               "reached": reached, "b_alg": b_alg}
        if name in e2e_runs:
            per = [m_c / (wall / num_roots * 1e-3) / 1e9 for m_c, wall in e2e_runs[name]]
            out["e2e"] = hmean(np.concatenate(per))
            out["e2e_step_ms"] = float(np.mean([w for _, w in e2e_runs[name]]))
        return out

    modes = {name: summarize(name) for name in runs[0]}
    first = next(iter(modes.values()))
    if not all(np.array_equal(modes[k]["edges"], first["edges"]) for k in modes):
        raise RuntimeError("modes disagree on m_c")
    # the headline: the learned + batched way with results materialized,
    # else the best materialized way that ran, else the best of the rest
    best = max(modes, key=lambda k: (k == "batched", "traversal" not in k, modes[k]["gteps"]))
    head = modes[best]
    value_rank, step_ms = head["gteps"], head["step_ms"]
    e2e_rank = head.get("e2e", 0.0)
    if world > 1:
        step_ms, value, e2e_value = reduce_over_ranks(step_ms, value_rank, e2e_rank, device=dev)
    else:
        value, e2e_value = value_rank, e2e_rank

    # roofline of the headline way over its timed launches: the algorithmic
    # bytes B_alg (one CSR pass per group + every root's int32 depth and
    # int64 parent of each reached vertex) over the device time of the groups, which covers
    # the traversal kernel, the per-lane counts and the result rows
    achieved = float(head["b_alg"].sum() / (head["ms"].sum() * 1e-3) / 1e9)
    peak, peak_kind = peaks()
    traffic = None
    tpath = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(tpath):
        with open(tpath) as f:
            traffic = json.load(f).get(f"{args.workload}-{best}", {}).get("bytes_per_launch")
    kernels = {}
    if "batched" in modes and "batched_traversal" in modes:
        t_all = modes["batched"]["step_ms"] / groups
        t_trav = modes["batched_traversal"]["step_ms"] / groups
        rows = 12.0 * n * min(num_roots, 64)
        kernels = {
            "traversal_ms_per_group": t_trav,
            "traversal_GBps_csr_pass": (8.0 * (n + 1) + 8.0 * m) / (t_trav * 1e-3) / 1e9,
            "result_rows_ms_per_group": t_all - t_trav,
            "result_rows_GBps_written": rows / max(t_all - t_trav, 1e-9) / 1e6 if t_all > t_trav
            else None,
            "note": "traversal = the batched_traversal way's group time; result rows = the "
                    "difference to the materialized way (12 B x n x 64 written per group)",
        }
    ms = head["ms"]
    bi, bo = 8 * num_roots, 16 * num_roots + 8 * n * num_roots
    line = {
        "metric": metric, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": step_ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
        "config": workload_config(desc, num_roots, scale, graph_seed, n, m),
        "run": {
            "mode": best,
            "results": "materialized: every root's int32 depths and int64 parents (caller ids, "
                       "reference encoding) in device memory when the step ends"
                       if "traversal" not in best else "traversal only",
            "parallelism": f"replicas x{world} (rank r takes lcg(r) roots)" if world > 1
            else "1 GPU",
            "graph_build_s": round(gen_s, 2),
            "adjacency_order": args.order,
        },
        "modes": {k: {kk: vv for kk, vv in (("gteps", v["gteps"]), ("ms_per_step", v["step_ms"]),
                                             ("e2e_gteps", v.get("e2e")),
                                             ("e2e_ms_per_step", v.get("e2e_step_ms")))
                      if vv is not None}
                  for k, v in modes.items()},
        "plain_beamer_gteps": modes["plain"]["gteps"] if "plain" in modes else None,
        "learned_gteps": modes["learned"]["gteps"] if "learned" in modes else None,
        "batched_gteps": modes["batched"]["gteps"] if "batched" in modes else None,
        "per_root_ms": {"min": float(ms.min()), "median": float(np.median(ms)), "max": float(ms.max())},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": traffic,
                     "peak_kind": peak_kind,
                     "peak_nominal": HBM_NOMINAL_GBS, "frac_nominal": achieved / HBM_NOMINAL_GBS,
                     "note": ("B_alg per 64-root group = 8(n+1) + 8m + 12 sum n_c" if best.startswith("batched")
                              else "B_alg = 8(n+1) + 8 m_c + 12 n_c per root") +
                             " over the device time of the " + best + " way (traffic: ncu DRAM "
                             "bytes of the launches of one group or root, profiles/traffic.json)",
                     "kernels": kernels or None},
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": bi,
                "d2h_bytes_per_step": bo,
                "note": f"public API per step ({best if best in e2e_runs else 'none'}): the run "
                        "(roots uploaded by the call), m_c / n_c read back, and every root's int64 "
                        "parent array copied to pinned host memory"},
        # kernels per root (clear, search with its source setup and counters, result
        # rows) or per group (clear, init, traversal, per-lane counts, result rows);
        # the e2e passes launch the same kernels again
        "gpu_launches": args.steps * (
            sum({"plain": 3 * num_roots, "learned": 3 * num_roots, "plain_traversal": 2 * num_roots,
                 "batched": 5 * groups, "batched_rule": 5 * groups,
                 "batched_traversal": 4 * groups}[x] for x in order_run)
            + sum({"batched": 5 * groups, "plain": 3 * num_roots}[x] for x in e2e_ways)),
        "clocks": clocks.summary(),
    }
    if el64 is not None:
        t0 = time.time()
        rows, tail = reference_cpu_run(el64, args.cpu_roots, timeout=1200)
        wall = time.time() - t0
        if rows:
            cg = [e / (t * 1e-3) / 1e9 for e, t in rows]
            line["cpu_baseline"] = {
                "value": hmean(cg), "unit": UNIT, "cores": 1, "kind": "reference",
                "sample": f"{len(rows)} lcg(0) roots of the same graph, reference serial-elision "
                          f"build (oracle/_ref/hybrid_bfs) pinned to 1 core, after the GPU's "
                          f"timed region; wall {wall:.0f} s incl. el64 load + graph build"}
        else:
            line["cpu_baseline"] = {"value": None, "unit": UNIT, "cores": 1, "kind": "reference",
                                    "sample": f"failed: {tail}"}
        tmpdir.cleanup()
    if rank == 0:
        print(json.dumps(line))
    for h in handles.values():
        h.close()
    if world > 1:
        dist.destroy_process_group()
    return 0

if __name__ == "__main__":
    sys.exit(main())
