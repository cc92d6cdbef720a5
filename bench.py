#!/usr/bin/env python
"""Benchmark: colorings/sec of color-coding tree-template counting on B200.

Default workload (N=1): the 12-vertex tree (path v0..v7, pendants v8@v2,
v9@v4, v10@v5, v11@v10) on an R-MAT scale-20, edge-factor-8 graph
(a,b,c = 0.57,0.19,0.19, seed 1; symmetrised, deduplicated), FP32 count
tables, 16 colorings per step (coloring c seeded srand(7 + c)).

  value     colorings/sec over all ranks, CUDA-event time of the counting
            launches on the library's stream, inputs resident in HBM.
  e2e       the same metric through the public C ABI per step: device graph
            built from pinned host CSC arrays (H2D copy inside the timed
            region), all colorings counted, raw counts read back (D2H);
            W untimed warm-up steps first, as for value.
  roofline  the dominant step (gather and product kernels of one
            sub-template): compulsory bytes divided by its CUDA-event
            duration, against MEASURED_PEAKS.json.
  cpu_baseline  the reference's own CPU code (its CountMat::colorCounting,
            built from the reference sources into oracle/_ref/) on the host
            cores, on the first two colorings the GPU timed, same graph: its
            raw counts give rel_err_vs_reference.

--impl reference runs the reference's stock CLI (oracle/_ref/sc-nec-ncc.bin)
alone on rank 0 on the same text edge list (one coloring per step) and prints
its line.  The graphs are written by subgraph_b200.synth (numpy only), so
that arm never loads this project's library.
Multi-GPU (torchrun): every rank counts its own colorings of the same graph
(independent replicas, weak scaling); the only exchange is the max of the
step times and a gather of the counts.
"""
from __future__ import annotations

import argparse
import json
import os
import re
import shutil
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

TEMPLATES = {
    "p3": (3, [(0, 1), (1, 2)]),
    "tree5": (5, [(0, 1), (1, 2), (2, 3), (1, 4)]),
    "spider7": (7, [(0, 1), (1, 2), (0, 3), (3, 4), (0, 5), (5, 6)]),
    "tree12": (12, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (5, 6), (6, 7), (2, 8), (4, 9), (5, 10), (10, 11)]),
}
WORKLOADS = {
    # the 12-vertex tree on R-MAT scale 20, edge factor 8: 16 colorings per step
    "tree12_rmat20_ef8": dict(scale=20, ef=8, template="tree12", per_step=16, seed=7),
    "p3_rmat16_ef16": dict(scale=16, ef=16, template="p3", per_step=1, seed=7),
    "tree5_rmat20_ef6": dict(scale=20, ef=6, template="tree5", per_step=10, seed=7),
    "spider7_rmat21_ef8": dict(scale=21, ef=8, template="spider7", per_step=64, seed=7),
    # the 12-vertex tree on R-MAT scale 18: the same kernels on a case small
    # enough for full ncu captures (about 2 GB of tables, still above L2)
    "tree12_rmat18_ef8": dict(scale=18, ef=8, template="tree12", per_step=1, seed=7),
}
# a seeded stream of 256 jobs, each a random tree of 3-10 vertices (uniform
# Pruefer sequence, smallest-leaf decoding, edges in decode order) on one of
# three R-MAT graphs (scales 16, 18, 20, edge factor 8): one coloring per job,
# the jobs of a graph spread over CUDA streams (--persistent: one persistent
# job-queue launch per graph and wave)
MIXED = dict(jobs=256, stream_seed=5, scales=(16, 18, 20), ef=8, seed=7)
WORKLOADS["mixed256_rmat16_18_20_ef8"] = dict(mixed=True, per_step=MIXED["jobs"], template="random 3-10",
                                              scale="16/18/20", ef=8, seed=7)
DEFAULT_WORKLOAD = "tree12_rmat20_ef8"


def prufer_tree(n, rng):
    """Edges of the labelled tree of a uniform random Pruefer sequence."""
    if n == 2:
        return [(0, 1)]
    seq = [rng.randrange(n) for _ in range(n - 2)]
    deg = [1] * n
    for a in seq:
        deg[a] += 1
    edges = []
    for a in seq:
        leaf = min(i for i in range(n) if deg[i] == 1)
        edges.append((leaf, a))
        deg[leaf] -= 1
        deg[a] -= 1
    u, v = [i for i in range(n) if deg[i] == 1]
    edges.append((u, v))
    return edges


def mixed_jobs():
    import random
    rng = random.Random(MIXED["stream_seed"])
    jobs = []
    for j in range(MIXED["jobs"]):
        n = rng.randint(3, 10)
        jobs.append((rng.randrange(len(MIXED["scales"])), n, prufer_tree(n, rng), MIXED["seed"] + j))
    return jobs
METRIC = "colorings/sec"


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, index: int):
        self.path = tempfile.mktemp(suffix=".csv")
        self.proc = None
        self.index = index

    def __enter__(self):
        if shutil.which("nvidia-smi"):
            q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
                 "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.proc or not os.path.exists(self.path):
            return None
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


def graph_file(scale: int, ef: int) -> str:
    """The workload's R-MAT graph as a text edge list (numpy generator, cached)."""
    from subgraph_b200 import synth
    return synth.rmat_file(scale, ef, seed=1)


def build_graph(w):
    """Host CSC of the workload's graph, read from its text file by the
    library's EdgeList (EdgeList.cpp:34-116 semantics)."""
    import subgraph_b200 as sg
    path = graph_file(w["scale"], w["ef"])
    el = sg.EdgeList(path)
    csc = sg.CSCGraph()
    csc.createFromEdgeListFile(el.getNumVertices(), el.getNumEdges(), el.getSrcList(), el.getDstList())
    return path, csc


def write_template(workdir: str, n: int, edges) -> str:
    tpath = os.path.join(workdir, "template.fascia")
    with open(tpath, "w") as f:
        f.write(f"{n}\n{len(edges)}\n" + "".join(f"{a} {b}\n" for a, b in edges))
    return tpath


def reference_cli(gpath: str, n: int, edges, iters: int, threads: int, workdir: str):
    """The reference's stock CLI (built from its sources, oracle/_ref/sc-nec-ncc.bin)
    on a text edge list: argv graph template iterations threads load_binary=0
    write_binary=0 isPruned=1 useSPMM=1.  Returns seconds per coloring (its
    "Time for count per iter" line, which covers the counting loop only) or
    None when the binary is missing or fails."""
    exe = os.path.join(ROOT, "oracle", "_ref", "sc-nec-ncc.bin")
    if not os.path.exists(exe):
        return None
    tpath = write_template(workdir, n, edges)
    env = dict(os.environ, OMP_NUM_THREADS=str(threads))
    r = subprocess.run([exe, gpath, tpath, str(iters), str(threads), "0", "0", "1", "1"],
                       capture_output=True, text=True, env=env, cwd=workdir, timeout=3600)
    m = re.search(r"Time for count per iter:\s*([0-9.eE+-]+)", r.stdout)
    if r.returncode == 0 and m:
        return float(m.group(1))
    log("reference CLI failed:", r.returncode, r.stderr[-500:])
    return None


def reference_counts(gpath: str, n: int, edges, seed: int, ncol: int, threads: int, workdir: str):
    """The reference's CountMat::colorCounting (oracle/_ref/ref_oracle, linked
    from the reference's own objects) for colorings srand(seed) ..
    srand(seed + ncol - 1) on the same text edge list: (raw counts, seconds of
    each coloring), or None when the harness is missing."""
    from oracle import oracle as O
    if not O.ref_available():
        return None
    tpath = write_template(workdir, n, edges)
    R = O.run_ref(gpath, tpath, ncol, seed, os.path.join(workdir, "ref_out"), threads=threads, light=True)
    return R["raw"], R["times"]


def run_reference_arm(args, w):
    """Rank 0 runs the reference's stock CLI: W warm-up colorings in one run, then
    K timed colorings (one per step) in another; ms_per_step is its time per
    coloring."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    n, edges = TEMPLATES[w["template"]]
    gpath = graph_file(w["scale"], w["ef"])
    with tempfile.TemporaryDirectory() as tmp:
        if args.warmup > 0:
            reference_cli(gpath, n, edges, args.warmup, threads, tmp)
        sec = reference_cli(gpath, n, edges, args.steps, threads, tmp)
    if sec is None:
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/sc-nec-ncc.bin is missing or failed "
                                                               "(build it with oracle/build_ref.sh)"}), flush=True)
        return
    value = 1.0 / sec
    line = {
        "metric": METRIC, "value": value, "unit": "colorings/s", "impl": "reference", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1000.0, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp32", "data": "synthetic",
        "config": config_of(args, w),
        "step": "one coloring of the workload per step (the GPU arm's step is colorings_per_step colorings); "
                "the metric is per coloring in both arms",
        "cpu_baseline": {"value": value, "unit": "colorings/s", "cores": threads, "kind": "reference",
                         "sample": f"{args.steps} colorings timed by the reference CLI's own counter after a "
                                   f"{args.warmup}-coloring warm-up run, {threads} OpenMP threads, text edge "
                                   f"list input"},
        "e2e": {"value": value, "unit": "colorings/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_mixed(args):
    """The mixed-template job stream: every step counts all jobs once."""
    import numpy as np
    import torch

    import subgraph_b200 as sg
    jobs = mixed_jobs()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    cfg = {"workload": args.workload, "jobs": MIXED["jobs"], "templates": "random trees of 3-10 vertices",
           "graphs": "rmat scales 16/18/20 edge factor 8 seed 1", "stream_seed": MIXED["stream_seed"],
           "form": ("persistent job queue per graph" if args.persistent
                    else f"job streams per graph ({args.batch or 8} CUDA streams)"), "tables": "fp32", "sums": "fp64",
           "l2": "inputs larger than L2 at scales 18 and 20"}
    paths = [graph_file(sc, MIXED["ef"]) for sc in MIXED["scales"]]
    if args.impl == "reference":
        if rank != 0:
            return
        # the reference CLI on a bounded sample: the first jobs of the stream, one coloring each
        t_tot, done = 0.0, 0
        cores = os.cpu_count() or 1
        with tempfile.TemporaryDirectory() as tmp:
            for gi, n, edges, seed in jobs:
                if t_tot > 20.0 or done >= 32:
                    break
                sec = reference_cli(paths[gi], n, edges, 1, cores, tmp)
                if sec is None:
                    print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/sc-nec-ncc.bin is missing "
                                                                           "or failed"}), flush=True)
                    return
                t_tot += sec
                done += 1
        value = done / t_tot
        kind = "reference"
        print(json.dumps({"metric": METRIC, "value": value, "unit": "colorings/s", "impl": "reference",
                          "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
                          "ms_per_step": MIXED["jobs"] / value * 1000.0, "higher_is_better": True, "scaling": "weak",
                          "vs_baseline": None, "dtype": "fp32", "data": "synthetic", "config": cfg,
                          "cpu_baseline": {"value": value, "unit": "colorings/s", "cores": cores, "kind": kind,
                                           "sample": f"the first {done} jobs of the stream, one coloring each"},
                          "e2e": {"value": value, "unit": "colorings/s", "h2d_bytes_per_step": 0,
                                  "d2h_bytes_per_step": 0}}), flush=True)
        return
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    graphs = []
    for path in paths:
        el = sg.EdgeList(path)
        csc = sg.CSCGraph()
        csc.createFromEdgeListFile(el.getNumVertices(), el.getNumEdges(), el.getSrcList(), el.getDstList())
        graphs.append(csc)
    dgs = [csc.device_graph(local) for csc in graphs]
    tmpls = [sg.Graph(n, e) for _, n, e, _ in jobs]
    by_graph = [[j for j, job in enumerate(jobs) if job[0] == gi] for gi in range(len(graphs))]

    launches = [0]

    def step():
        ms, lat = 0.0, np.zeros(len(jobs))
        raw = np.zeros(len(jobs))
        for gi, idx in enumerate(by_graph):
            if not idx:
                continue
            r, l, st = sg.count_jobs(dgs[gi], [tmpls[j] for j in idx], [jobs[j][3] for j in idx],
                                     return_latency=True, return_stats=True, persistent=args.persistent,
                                     streams=args.batch)
            raw[idx], lat[idx] = r, l + ms   # the graphs run one after the other
            ms += st["device_ms"]
            launches[0] += st["kernel_launches"]
        return ms, lat, raw

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    launches[0] = 0
    tot, lats = 0.0, []
    with Clocks(local) as clk:
        torch.cuda.nvtx.range_push("timed")
        for _ in range(args.steps):
            ms, lat, raw = step()
            tot += ms
            lats.append(lat)
        torch.cuda.nvtx.range_pop()
    clocks = clk.summary()
    value = world * len(jobs) * args.steps / (tot / 1000.0)
    lat = np.concatenate(lats)
    # the plain form: each job on its own, one after the other
    plain_ms = 0.0
    for j, (gi, n, e, seed) in enumerate(jobs):
        _, st = sg.count(dgs[gi], tmpls[j], 1, seed, return_stats=True)
    for j, (gi, n, e, seed) in enumerate(jobs):
        _, st = sg.count(dgs[gi], tmpls[j], 1, seed, return_stats=True)
        plain_ms += st["device_ms"]
    plain = len(jobs) / (plain_ms / 1000.0)
    # end to end: graphs already resident, templates planned on the host each step
    t0 = time.perf_counter()
    for _ in range(args.steps):
        for gi, idx in enumerate(by_graph):
            ts = [sg.Graph(jobs[j][1], jobs[j][2]) for j in idx]
            sg.count_jobs(dgs[gi], ts, [jobs[j][3] for j in idx], persistent=args.persistent, streams=args.batch)
    e2e_s = time.perf_counter() - t0
    line = {"metric": METRIC, "value": value, "unit": "colorings/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": tot / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "fp32", "data": "synthetic", "config": cfg,
            "latency_ms": {"p50": float(np.percentile(lat, 50)), "p99": float(np.percentile(lat, 99))},
            "forms": {"plain": plain, "batched": value, "batched_over_plain": value / plain, "unit": "colorings/s"},
            "roofline": None, "gpu_launches": launches[0], "clocks": clocks,
            "e2e": {"value": world * len(jobs) * args.steps / e2e_s, "unit": "colorings/s",
                    "h2d_bytes_per_step": 124 * len(jobs),   # one 31-word coloring window per job
                    "d2h_bytes_per_step": 16 * len(jobs)}}
    if rank == 0:
        print(json.dumps(line), flush=True)


def config_of(args, w):
    return {"workload": args.workload, "graph": f"rmat scale {w['scale']} edge factor {w['ef']} seed 1",
            "template": w["template"], "colorings_per_step": w["per_step"], "tables": "fp32",
            "sums": "fp64",
            "form": "plain" if args.batch == 0 else (f"persistent({args.batch})" if args.persistent
                                                     else f"interleaved groups({args.batch})"),
            "hub_threshold": args.hub, "l2": "inputs larger than L2 (count tables of several GB per coloring)"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=DEFAULT_WORKLOAD, choices=sorted(WORKLOADS))
    ap.add_argument("--batch", type=int, default=0, help="colorings per batch (0 = plain form)")
    ap.add_argument("--persistent", action="store_true", help="batched form: persistent work-queue launch per batch")
    ap.add_argument("--hub", type=int, default=1024)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-forms", action="store_true", help="skip timing the other form (plain vs batched)")
    args = ap.parse_args()
    w = WORKLOADS[args.workload]
    if w.get("mixed"):
        run_mixed(args)
        return
    if args.impl == "reference":
        run_reference_arm(args, w)
        return

    import numpy as np
    import torch

    import subgraph_b200 as sg

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))

    def barrier():
        torch.cuda.synchronize()
        if dist:
            dist.barrier()

    def max_over_ranks(x: float) -> float:
        if not dist:
            return x
        t = torch.tensor([x], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    t_build = time.perf_counter()
    gpath, csc = build_graph(w)
    g = csc.device_graph(local)
    n, edges = TEMPLATES[w["template"]]
    tmpl = sg.Graph(n, edges)
    B = w["per_step"]
    log(f"[rank {rank}] graph V={csc.getNumVertices()} nnz={csc.getNNZ()} built in {time.perf_counter() - t_build:.1f}s")

    def seeds(step):  # rank-disjoint colorings
        return w["seed"] + (step * world + rank) * B

    # warm-up; the first call on a new graph also allocates its tables and, in
    # the forms that tune (the persistent queue), times the tile shapes: its
    # wall time against the second call's is that cost
    warm_ms = []
    for s in range(args.warmup):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        sg.count(g, tmpl, B, seeds(s), batch=args.batch, hub_threshold=args.hub, persistent=args.persistent)
        warm_ms.append((time.perf_counter() - t0) * 1000.0)
    first_ms = warm_ms[0] if warm_ms else None
    steady_ms = warm_ms[1] if len(warm_ms) > 1 else None
    barrier()
    dev_ms, launches, fused_ms, fused_launches, fused_bytes, gather_bytes, hub_ms = 0.0, 0, 0.0, 0, 0.0, 0.0, 0.0
    top = {"ms": 0.0, "bytes": 0.0, "launches": 0, "sub": -1}
    raws = []
    with Clocks(local) as clk:
        barrier()
        torch.cuda.nvtx.range_push("timed")
        for s in range(args.steps):
            raw, st = sg.count(g, tmpl, B, seeds(args.warmup + s), batch=args.batch, hub_threshold=args.hub,
                               persistent=args.persistent, return_stats=True, profile=True)
            raws.append(raw)
            dev_ms += st["device_ms"]
            launches += st["kernel_launches"]
            fused_ms += st["fused_ms"]
            fused_launches += st["fused_launches"]
            fused_bytes += st["fused_alg_bytes"]
            gather_bytes += st["fused_gather_bytes"]
            hub_ms += st["hub_ms"]
            top["ms"] += st["top_ms"]
            top["bytes"] += st["top_alg_bytes"]
            top["launches"] += st["top_launches"]
            top["sub"] = st["top_sub"]
        barrier()
        torch.cuda.nvtx.range_pop()
    clocks = clk.summary()
    total_ms = max_over_ranks(dev_ms)
    ms_per_step = total_ms / args.steps
    value = world * B * args.steps / (total_ms / 1000.0)

    # the other form on the same colorings (plain <-> batched), for the batched-vs-plain ratio
    forms = None
    if not args.no_forms:
        other = B if args.batch == 0 else 0
        for s in range(min(args.warmup, 2)):
            sg.count(g, tmpl, B, seeds(s), batch=other, hub_threshold=args.hub)
        barrier()
        other_ms = 0.0
        for s in range(args.steps):
            _, st = sg.count(g, tmpl, B, seeds(args.warmup + s), batch=other, hub_threshold=args.hub,
                             return_stats=True)
            other_ms += st["device_ms"]
        barrier()
        other_value = world * B * args.steps / (max_over_ranks(other_ms) / 1000.0)
        plain_v, batched_v = (value, other_value) if args.batch == 0 else (other_value, value)
        forms = {"plain": plain_v, "batched": batched_v, "batch": args.batch or B,
                 "batched_over_plain": batched_v / plain_v, "unit": "colorings/s"}

    # end to end through the public API: pinned host CSC -> device graph -> count -> raw counts
    e2e = None
    if not args.no_e2e:
        col = torch.from_numpy(csc.getIndexCol()).pin_memory()
        row = torch.from_numpy(csc.getIndexRow()).pin_memory()
        col_np, row_np = col.numpy(), row.numpy()
        h2d = 4 * (len(col_np) + len(row_np))
        # untimed warm-up steps of this leg too: the first graph of the leg
        # grows the device memory pool by its tables (the timed steps reuse it)
        for s in range(args.warmup):
            dg = sg.DeviceGraph(col_np, row_np, local)
            sg.count(dg, tmpl, B, seeds(s), batch=args.batch, hub_threshold=args.hub, persistent=args.persistent)
            del dg
        barrier()
        t0 = time.perf_counter()
        for s in range(args.steps):
            dg = sg.DeviceGraph(col_np, row_np, local)
            sg.count(dg, tmpl, B, seeds(args.warmup + s), batch=args.batch, hub_threshold=args.hub,
                     persistent=args.persistent)
            del dg
        barrier()
        e2e_s = max_over_ranks(time.perf_counter() - t0)
        e2e = {"value": world * B * args.steps / e2e_s, "unit": "colorings/s", "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": 8 * B}

    # precision: FP32 tables against FP64 tables on the first two colorings of the run
    n_chk = min(2, B)
    r64 = sg.count(g, tmpl, n_chk, seeds(args.warmup), mode=sg.MODE_FP64, hub_threshold=args.hub)
    err = max(abs(a - b) / abs(b) for a, b in zip(raws[0][:n_chk], r64) if b != 0) if np.any(r64) else 0.0
    err = max_over_ranks(err)

    peak, peak_kind = peaks()
    # the dominant kernel: the sub-template stage whose fused launches take the most time
    achieved = top["bytes"] / (top["ms"] / 1000.0) / 1e9 if top["ms"] > 0 else 0.0
    all_achieved = fused_bytes / (fused_ms / 1000.0) / 1e9 if fused_ms > 0 else 0.0
    line = {
        "metric": METRIC, "value": value, "unit": "colorings/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "fp32", "data": "synthetic", "config": config_of(args, w),
        "rel_err_vs_fp64": err,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak if peak else 0.0, "peak_kind": peak_kind, "traffic": None,
                     "kernel": f"gather and product step of sub {top['sub']} (the dominant step)",
                     "launch_ms": top["ms"] / max(top["launches"], 1),
                     "alg_bytes_per_launch": top["bytes"] / max(top["launches"], 1),
                     "all_fused": {"achieved": all_achieved, "frac": all_achieved / peak if peak else 0.0,
                                   "ms_per_step": fused_ms / args.steps,
                                   "launches_per_step": fused_launches / args.steps,
                                   "alg_bytes_per_step": fused_bytes / args.steps,
                                   "gather_bytes_per_step": gather_bytes / args.steps},
                     "hub_ms_per_step": hub_ms / args.steps},
        "gpu_launches": launches,
        "clocks": clocks,
        "autotune": {"first_call_ms": first_ms, "second_call_ms": steady_ms,
                     "note": "wall clock of the first two warm-up steps: the first call on a new graph allocates its "
                             "tables; only the persistent queue times tile shapes"},
    }
    if forms:
        line["forms"] = forms
    if e2e:
        line["e2e"] = e2e
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        # the reference's CountMat on the first two colorings this run timed, same
        # graph file: its time is the CPU baseline, its raw counts the parity check
        cores = os.cpu_count() or 1
        s0 = seeds(args.warmup)
        n_ref = min(2, B)
        with tempfile.TemporaryDirectory() as tmp:
            got = reference_counts(gpath, n, edges, s0, n_ref, cores, tmp)
        if got is not None:
            ref_raw, ref_t = got
            per = [abs(a - b) / abs(b) if b else abs(a - b) for a, b in zip(raws[0][:n_ref], ref_raw)]
            est_gpu = sg.estimate(raws[0][:n_ref], n)
            est_ref = sg.estimate(ref_raw, n)
            line["rel_err_vs_reference"] = {
                "per_coloring": per, "max": max(per), "estimate": abs(est_gpu - est_ref) / abs(est_ref) if est_ref else 0.0,
                "seeds": [s0 + i for i in range(n_ref)],
                "reference": "CountMat::colorCounting of the compiled reference (oracle/_ref/ref_oracle), same text "
                             "edge list and seeds"}
            line["cpu_baseline"] = {"value": 1.0 / float(ref_t.mean()), "unit": "colorings/s", "cores": cores,
                                    "kind": "reference",
                                    "sample": f"{n_ref} colorings (seeds {s0}..{s0 + n_ref - 1}) of the workload, "
                                              f"counting loops on {cores} OpenMP threads"}
        else:
            # the oracle port on one coloring (single thread)
            from oracle import oracle as O
            P = O.Plan(n, edges)
            colors = O.colors(s0, csc.getNumVertices(), n)
            t0 = time.perf_counter()
            O.count_coloring(csc.getIndexCol(), csc.getIndexRow(), P, colors)
            line["cpu_baseline"] = {"value": 1.0 / (time.perf_counter() - t0), "unit": "colorings/s", "cores": 1,
                                    "kind": "port", "sample": "1 coloring of the workload"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
