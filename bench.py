#!/usr/bin/env python3
"""Fast-winding-number benchmark (one JSON line on rank 0).

Workload (default): displaced geodesic icosphere, frequency 316 (1,997,120 triangles, seed 1),
10M queries (5M uniform in bbox*1.2, 5M on the surface offset by +-U(1e-6, 1e-3)), beta = 2.
A step = one winding-number query pass over the 10M points against the built tree.

  value      queries/s of the mixed-precision engine with inputs resident in HBM (device time,
             CUDA events on the launching stream, L2 flushed before every step)
  e2e        the same metric through the C ABI's host-buffer call fwn_query_host (pinned host
             buffers; H2D of the points and D2H of Omega + inside inside the timed region)
  e2e_stream the same through fwn_query_host_batches: one call over K batches (a serving loop),
             each batch's copies overlapping the walk of its neighbour; every copy is inside the
             timed region
  plain_fp64 the plain FP64 form (FP64 everywhere, same tree), its queries/s and the max / RMS
             |dw| between the two forms over all queries (gate: <= 1e-4)
  roofline   FP32 roofline of the traversal kernel: algorithmic flops from device work
             counters over its CUDA-event time, against the FP32 FMA peak measured in the same
             process (fwn_probe_fp32_peak)
  cpu_baseline  the CPU implementation of the reference path on the host cores (the reference
             itself when a built one is present under baseline/_ref, else the oracle's
             restatement O2)
  batched    the 512-mesh forest (one persistent CUDA-graph launch; build ms, meshes/s, the
             per-mesh FP64 launches with max |dw| over every query, is_inside against the
             reference restatement on sampled meshes)
  soup       the defective 1M-triangle soup (|dw| split near / far against the FP64 form on
             every point and against the FP64 brute force on a sample; is_inside against the
             reference restatement on every point)
  uvsphere   the 64x32 UV sphere with 100k queries, checked on every point against the FP64
             brute force
  voxel      4 x 5M-triangle meshes on 256^3 voxel-centre grids (67M queries; explicit points in
             one persistent launch and the device-generated grid path; is_inside against the
             reference restatement on mesh 0's 16.7M voxels)

``--impl reference`` times the reference path's CPU implementation on the same workload (the
reference itself when a built one is present under baseline/_ref, else the oracle restatement)
and prints the same line with ``"impl": "reference"``.

Multi-GPU (torchrun): every rank builds its own replica of the tree. By default every rank
answers its own 10M queries (rank r > 0: a seeded shuffle of the set), with no collective on the
data path; value = all ranks' queries / the slowest rank's time (weak scaling). With
``--split-queries`` the ranks share one set: each answers its contiguous range of the query order
and the results are all-gathered (strong scaling).
"""
from __future__ import annotations

import argparse
import ctypes as C
import json
import math
import os
import statistics
import tempfile
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "winding queries/s @2M tris (mixed precision, |dw|<=1e-4 vs plain FP64 GPU form)"
FOUR_PI = 4.0 * math.pi

# Algorithmic work per unit (constants of the traversal kernel, counted from its source). An ncu
# instruction-mix capture of one traversal launch (2M queries, LBVH tree at leaf 12) counts 21.3
# kflop of executed FP32 work per query against 13.8 kflop from these constants and the launch's
# own counters: the rest is work the warp schedule does on lanes that discard it.
FLOPS_FAR = 82      # order-0/1/2 Taylor term incl. far test and Kahan add (FMA = 2)
FLOPS_TRI = 95      # Van Oosterom triangle incl. FP64-band test and Kahan add (atan2/sqrt on SFU)
FLOPS_TEST = 12     # far test of a near node (d = P - q, |d|^2, beta r, compare)
BYTES_NODE_TEST = 32   # sector 0 of a NodeF32 record
BYTES_NODE_FAR = 96    # sectors 1-3 (far-field coefficients)
BYTES_TRI = 48
BYTES_QUERY_IO = 12 + 4 + 1 + 4  # point in, Omega + inside out, sort index
CPU_LEAF = 8  # leaf size of the CPU restatement of the reference tree, in every CPU timing
# DRAM bytes (read + write) of one traversal launch, keyed by (workload, leaf size, warp-schedule
# variant, builder), from one-pass ncu captures (gpu__time_duration, dram__bytes_read/write) of
# the same bench command lines; other configurations: not captured (traffic null)
NCU_TRAFFIC = {("displaced_icosphere_nu316_q10000000", 12, 4, 0): 952.36e6 + 57.72e6,
               ("displaced_icosphere_nu316_q10000000", 8, 4, 1): 973.63e6 + 52.19e6,
               ("displaced_icosphere_nu316_q10000000", 8, 6, 1): 976.28e6 + 53.64e6,
               ("displaced_icosphere_nu316_q10000000", 8, 4, 2): 972.76e6 + 52.60e6,
               ("displaced_icosphere_nu316_q10000000", 8, 6, 2): 973.71e6 + 52.88e6}


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--workload", default="icosphere",
                   choices=["icosphere", "soup", "uvsphere", "forest", "voxel"])
    p.add_argument("--nu", type=int, default=None)
    p.add_argument("--meshes", type=int, default=512)  # forest workload: number of meshes
    p.add_argument("--queries", type=int, default=None)
    p.add_argument("--leaf", type=int, default=0)  # 0: the autotuner picks (untimed)
    p.add_argument("--tuning", type=int, default=0)  # with --leaf: warp-schedule variant (0 auto)
    p.add_argument("--builder", type=int, default=0)  # with --leaf: 0 LBVH, 1 top-down splits, 2 binned
    p.add_argument("--traversal", default="warp", choices=["thread", "warp"])
    p.add_argument("--block", type=int, default=128)
    p.add_argument("--fp64-steps", type=int, default=2)
    p.add_argument("--cpu-sample", type=int, default=100_000)
    p.add_argument("--brute", type=int, default=1024)      # CPU O1 sample
    p.add_argument("--brute-gpu", type=int, default=8192)  # GPU FP64 all-triangle sample
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--no-fp64", action="store_true")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-clocks", action="store_true")
    p.add_argument("--no-graph", action="store_true")  # time plain launches instead of a graph
    p.add_argument("--no-batched", action="store_true")  # default line without forest/soup parts
    # strong scaling: one query set split over the ranks (contiguous ranges of the query order,
    # results all-gathered) instead of a full set per rank
    p.add_argument("--split-queries", action="store_true")
    return p.parse_args()


# ---------------------------------------------------------------------------------------------
def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def init_dist(world, backend):
    if world > 1:
        import torch.distributed as dist
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group(backend=backend)
        return dist
    return None


def barrier(dist):
    if dist is not None:
        dist.barrier()


def max_over_ranks(dist, x: float, device=None) -> float:
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def rank0_choice(dist, values, device=None):
    """Every rank runs rank 0's tuning choice (ints), so all ranks time the same configuration."""
    if dist is None:
        return list(values)
    import torch
    t = torch.tensor([int(v) for v in values], dtype=torch.int64, device=device)
    dist.broadcast(t, src=0)
    return [int(v) for v in t.tolist()]


def rank_queries(Q, near_mask, rank: int):
    """The query set a rank answers (weak scaling: every rank has a full-size set). Rank 0 uses
    the workload as generated; rank r > 0 a seeded shuffle of it (different points per warp,
    same distribution)."""
    if rank == 0:
        return Q, near_mask
    perm = np.random.default_rng(1000 + rank).permutation(len(Q))
    return Q[perm], near_mask[perm]


def job_value(per_rank_units: int, world: int, max_seconds: float) -> float:
    """Whole-job throughput: the units all ranks processed over the slowest rank's time."""
    return world * per_rank_units / max_seconds


# ---------------------------------------------------------------------------------------------
def smi_gpu_id(local: int) -> str:
    """nvidia-smi's --id for CUDA device `local` of this process. nvidia-smi numbers GPUs by
    physical index, which differs from the CUDA ordinal under CUDA_VISIBLE_DEVICES or a leased
    subset, so the device is named by its UUID (falling back to the visible-devices mapping)."""
    try:
        import torch
        u = str(torch.cuda.get_device_properties(local).uuid)
        if u and u != "None":
            return u if u.startswith(("GPU-", "MIG-")) else "GPU-" + u
    except Exception:
        pass
    vis = [x.strip() for x in os.environ.get("CUDA_VISIBLE_DEVICES", "").split(",") if x.strip()]
    if local < len(vis):
        return vis[local]
    return str(local)


class Clocks:
    """nvidia-smi sampling (200 ms) during the timed region, of the GPU this process runs on."""

    def __init__(self, enabled: bool, index: int):
        self.enabled = enabled
        self.index = smi_gpu_id(index) if enabled else str(index)
        self.proc = None
        self.path = Path(tempfile.gettempdir()) / f"fwn_clocks_{os.getpid()}.csv"

    def __enter__(self):
        if not self.enabled:
            return self
        self.path.parent.mkdir(exist_ok=True)
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            time.sleep(0.25)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
            self.f.close()

    def summary(self):
        if self.proc is None or not self.path.exists():
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["not sampled"]}
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.path.read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax),
                "samples": len(sm), "reasons": sorted(reasons)}


def query_launches(n, max_queries, nodes, mesh_bits=0, key_bits=30, auto=False):
    """Kernels of one sorted query of n points (the library's choices): keys, the sort's passes, the
    walk, the walk of left-over groups, the results' scatter and, from a million points, the
    second output from the first. auto: the small batch of an engine whose schedule is AUTO, one
    kernel."""
    if auto and n <= 35_000:
        return 1
    need = max(1, mesh_bits + math.ceil(math.log2(max_queries)) + (-1 if nodes <= 32768 else 2))
    passes = min(math.ceil(need / 8), math.ceil(key_bits / 8))
    sort = 1 + passes if n <= 128 * 2048 else 3 * passes
    return 1 + sort + 2 + 1 + (1 if n >= 1_000_000 else 0)


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except Exception:
            pass
    return {}


# ---------------------------------------------------------------------------------------------
def make_workload(args):
    """Single-mesh workloads: icosphere (default: 1,997,120 triangles, 10M queries), soup (the
    defective 1M-triangle soup, 5M queries), uvsphere (3,968 triangles, 100k queries)."""
    from lagrange_gb300 import workloads as W
    if args.workload == "soup":
        return W.defective_soup_workload(nu=args.nu or 224, n_queries=args.queries or 5_000_000)
    if args.workload == "uvsphere":
        return W.uv_sphere_workload(n_queries=args.queries or 100_000)
    return W.displaced_icosphere_workload(nu=args.nu or 316, n_queries=args.queries or 10_000_000)


BUILDER_NAMES = {0: "lbvh", 1: "split", 2: "binned"}


def autotune_choice(fwn, Vd, Fd, Qd, sample: int = 16_000_000, seed: int = 5):
    """fwn_autotune on the workload's own queries (a seeded subsample above `sample` points):
    returns (leaf, traversal, block, tuning, builder, summary). Untimed; the bench then measures the
    chosen configuration. A subsample is sparser than the workload, so its warps are less
    coherent and it can favour larger leaves than the full query set does."""
    import torch
    n = Qd.shape[0]
    if n > sample:
        g = torch.Generator(device="cpu").manual_seed(seed)
        idx = torch.randperm(n, generator=g)[:sample].to(Qd.device)
        Qs = Qd[idx].contiguous()
    else:
        Qs = Qd
    r = fwn.autotune(Vd, Fd, Qs)
    summary = {"leaf_size": r["leaf_size"], "traversal": r["traversal"],
               "block_size": r["block_size"], "tuning": r["tuning"], "builder": r["builder"],
               "sample_ms": r["ms"], "candidates": r["candidates"], "sample": int(Qs.shape[0])}
    return r["leaf_size"], r["traversal"], r["block_size"], r["tuning"], r["builder"], summary


def percentiles(x):
    """p50/p90/p99/p99.9/max of a device tensor (quantiles of a 4M-element sample above that)."""
    import torch
    if x.numel() == 0:
        return None
    mx = float(x.max())
    if x.numel() > 4_000_000:
        g = torch.Generator(device=x.device).manual_seed(3)
        x = x[torch.randperm(x.numel(), device=x.device, generator=g)[:4_000_000]]
    qs = torch.tensor([0.5, 0.9, 0.99, 0.999], dtype=x.dtype, device=x.device)
    v = torch.quantile(x, qs).tolist()
    return {"p50": v[0], "p90": v[1], "p99": v[2], "p99.9": v[3], "max": mx}


def cpu_reference(V, F):
    """The CPU implementation of the reference path for the timed CPU legs: the reference's own
    FastWindingNumber when a built reference is present under baseline/_ref (kind "reference"),
    else the speed build of the oracle's restatement O2 (kind "port"). Returns (tree, kind,
    description)."""
    import oracle
    ok, why = oracle.reference_available()
    if ok:
        return (oracle.ReferenceEngine(V, F), "reference",
                "adobe/lagrange lagrange::winding::FastWindingNumber (baseline/_ref), per-point "
                "solid_angle calls over all host threads")
    return (oracle.RefTree(V, F, leaf_size=CPU_LEAF, fast=True), "port",
            "CPU restatement of the reference path (float order-2 Barill tree, beta 2, leaf "
            f"{CPU_LEAF}, -O3), per-point queries over all host threads; the reference itself: "
            + why)


def cpu_sample(wl, size: int, seed: int = 7):
    """A bounded sample of the workload's queries: half far/box, half near-surface when the
    workload has both kinds, else uniform."""
    rng = np.random.default_rng(seed)
    size = min(size, len(wl.Q))
    if wl.near_mask is None or not wl.near_mask.any() or wl.near_mask.all():
        return wl.Q[rng.choice(len(wl.Q), size, replace=False)]
    far_idx = np.nonzero(~wl.near_mask)[0]
    near_idx = np.nonzero(wl.near_mask)[0]
    half = size // 2
    return np.concatenate([wl.Q[rng.choice(far_idx, half, replace=False)],
                           wl.Q[rng.choice(near_idx, size - half, replace=False)]])


def run_reference(args, rank, world):
    """CPU implementation of the reference path (oracle restatement O2), all host threads."""
    dist = init_dist(world, "gloo")
    if rank != 0:
        barrier(dist)
        return
    import oracle
    if args.workload in ("forest", "voxel"):
        print(json.dumps({"impl": "reference", "unavailable": "the reference arm times the "
                          "single-mesh workloads; forest/voxel are GPU-side comparisons"}))
        barrier(dist)
        return
    wl = make_workload(args)
    nthr = oracle.nthreads_default()
    t0 = time.perf_counter()
    tree, kind, what = cpu_reference(wl.V, wl.F)
    build_s = time.perf_counter() - t0
    sample = cpu_sample(wl, args.cpu_sample)
    for _ in range(args.warmup):
        tree.query(sample[:2000], beta=wl.beta, nthreads=nthr)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        tree.query(sample, beta=wl.beta, nthreads=nthr)
    dt = (time.perf_counter() - t0) / args.steps
    qps = len(sample) / dt
    line = {
        "impl": "reference", "metric": METRIC, "value": qps, "unit": "queries/s", "n_gpus": 0,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": wl.name, "triangles": int(len(wl.F)), "queries": int(len(wl.Q)),
                   "beta": wl.beta, "leaf_size": CPU_LEAF},
        "cpu_baseline": {"value": qps, "unit": "queries/s", "cores": nthr, "kind": kind,
                         "sample": f"{len(sample)} queries per step (half far, half near-surface "
                                   f"where the workload has both) of the {len(wl.Q)}-query "
                                   f"workload; tree build "
                                   f"{build_s:.2f} s single-thread",
                         "build_s": build_s},
        "e2e": {"value": qps, "unit": "queries/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": what,
    }
    print(json.dumps(line), flush=True)
    barrier(dist)


# ---------------------------------------------------------------------------------------------
def measure_soup(dev, *, steps=5, warmup=3, cpu=True):
    """The defective soup (the displaced icosphere at frequency 224 with 10% of faces deleted, 1%
    flipped, 0.5% duplicated with 1e-7 jitter; 5M queries, half in the box, half within 1e-4 of
    the surface). Reports the mixed engine's queries/s, its |dw| distribution split near/far
    against the plain FP64 form on every point and against the FP64 brute force on a stratified
    sample, and is_inside against the CPU restatement of the reference on every point."""
    import torch
    import lagrange_gb300 as fwn
    from lagrange_gb300 import workloads as W
    t0 = time.perf_counter()
    wl = W.defective_soup_workload()
    gen_s = time.perf_counter() - t0
    n = len(wl.Q)
    Vd, Fd, Qd = (torch.from_numpy(a).to(dev) for a in (wl.V, wl.F, wl.Q))
    leaf, trav, block, tuning, builder, tuned = autotune_choice(fwn, Vd, Fd, Qd)
    eng = fwn.FastWindingNumber(Vd, Fd, leaf_size=leaf, traversal=trav, block_size=block,
                                tuning=tuning, builder=builder,
                                records=fwn.RECORDS_F32 | fwn.RECORDS_F64)
    L = fwn.library()
    stream = torch.cuda.current_stream(dev)
    sptr = C.c_void_p(stream.cuda_stream)
    w = torch.empty(n, dtype=torch.float32, device=dev)
    ins = torch.empty(n, dtype=torch.uint8, device=dev)
    w64 = torch.empty(n, dtype=torch.float64, device=dev)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    om = fwn._opts(precision=fwn.PRECISION_MIXED, traversal=trav, block_size=block, tuning=tuning)
    o64 = fwn._opts(precision=fwn.PRECISION_FP64, traversal=fwn.TRAVERSAL_THREAD)

    def q_mixed():
        fwn._check(L.fwn_query_ex(eng.handle, C.byref(om), C.c_void_p(Qd.data_ptr()), n,
                                  C.c_void_p(w.data_ptr()), C.c_void_p(ins.data_ptr()), None, None,
                                  sptr))

    def q_fp64():
        fwn._check(L.fwn_query_ex(eng.handle, C.byref(o64), C.c_void_p(Qd.data_ptr()), n, None,
                                  None, C.c_void_p(w64.data_ptr()), None, sptr))

    def timed(fn, k):
        ts = []
        for _ in range(k):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            fn()
            b.record(stream)
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return sum(ts) / len(ts)

    for _ in range(warmup):
        q_mixed()
    torch.cuda.synchronize()
    ms = timed(q_mixed, steps)
    q_fp64()
    ms64 = timed(q_fp64, 1)
    q_mixed()
    torch.cuda.synchronize()
    near = torch.from_numpy(wl.near_mask).to(dev)
    dw = (w.double() - w64).abs() / FOUR_PI
    band64 = (w64 / FOUR_PI - 0.5).abs() > 1e-3
    out = {
        "workload": wl.name, "triangles": int(len(wl.F)), "queries": n, "generation_s": gen_s,
        "leaf_size": leaf, "tuning": tuning, "builder": builder, "autotuned": tuned,
        "value": n / (ms / 1e3), "unit": "queries/s", "ms_per_step": ms, "steps": steps,
        "build_ms": eng.info()["build_ms"],
        "plain_fp64": {"value": n / (ms64 / 1e3), "ms": ms64, "speedup_mixed_over_fp64": ms64 / ms,
                       "max_dw": float(dw.max()), "rms_dw": float(dw.pow(2).mean().sqrt()),
                       "dw_percentiles": {"near": percentiles(dw[near]), "far": percentiles(dw[~near])},
                       "gate_1e-4": bool(float(dw.max()) <= 1e-4),
                       "inside_disagree_band": int(((ins.bool() != (w64 > 2 * math.pi)) & band64).sum())},
    }
    if cpu:
        import oracle
        nthr = oracle.nthreads_default()
        wg, ig = w.cpu().numpy(), ins.cpu().numpy()
        # FP64 brute force over all triangles on a stratified sample (1,024 far + 1,024 near)
        bs = cpu_sample(wl, 2048, seed=11)
        exact = oracle.brute_f64(wl.V, wl.F, bs, nthreads=nthr)
        wb, _ = eng.query(torch.from_numpy(bs).to(dev), traversal=trav)
        torch.cuda.synchronize()
        dwb = np.abs(wb.cpu().numpy().astype(np.float64) - exact) / FOUR_PI
        h = len(bs) // 2

        def npct(x):
            q = np.quantile(x, [0.5, 0.9, 0.99])
            return {"p50": float(q[0]), "p90": float(q[1]), "p99": float(q[2]), "max": float(x.max())}
        out["vs_brute_force_fp64"] = {"sample": len(bs), "far": npct(dwb[:h]), "near": npct(dwb[h:]),
                                      "note": "includes the beta=2 far-field truncation error"}
        # is_inside against the CPU restatement of the reference tree on every point
        t0 = time.perf_counter()
        ref, kind, _ = cpu_reference(wl.V, wl.F)
        om_ref, in_ref = ref.query(wl.Q, beta=wl.beta, nthreads=nthr)
        cpu_s = time.perf_counter() - t0
        band = np.abs(om_ref / FOUR_PI - 0.5) > 1e-3
        dref = np.abs(wg.astype(np.float64) - om_ref) / FOUR_PI
        out["inside_vs_reference"] = {
            "points": n, "outside_band": int(band.sum()),
            "disagree_outside_band": int(np.sum(ig[band] != in_ref[band])),
            "max_dw_vs_reference_restatement": float(dref.max()),
            "rms_dw_vs_reference_restatement": float(np.sqrt(np.mean(dref ** 2))),
            "reference_kind": kind, "cpu_s": cpu_s}
    eng.close()
    del Vd, Fd, Qd, w, ins, w64, flush
    return out


def measure_uvsphere(dev, *, steps=10, warmup=3, cpu=True):
    """The CPU-runnable configuration: the 64x32 UV sphere (3,968 triangles) with 100k queries
    uniform in [-1.5, 1.5]^3. Its oracle is the FP64 brute force over all triangles, evaluated on
    every point: |dw| of the mixed and FP64 forms against it (beta = 2 truncation included) and
    is_inside against it outside +-1e-3; plus the reference path's CPU rate on all points."""
    import torch
    import lagrange_gb300 as fwn
    from lagrange_gb300 import workloads as W
    wl = W.uv_sphere_workload()
    n = len(wl.Q)
    Vd, Fd, Qd = (torch.from_numpy(a).to(dev) for a in (wl.V, wl.F, wl.Q))
    leaf, trav, block, tuning, builder, tuned = autotune_choice(fwn, Vd, Fd, Qd)
    eng = fwn.FastWindingNumber(Vd, Fd, leaf_size=leaf, traversal=trav, block_size=block,
                                tuning=tuning, builder=builder,
                                records=fwn.RECORDS_F32 | fwn.RECORDS_F64)
    L = fwn.library()
    stream = torch.cuda.current_stream(dev)
    sptr = C.c_void_p(stream.cuda_stream)
    w = torch.empty(n, dtype=torch.float32, device=dev)
    ins = torch.empty(n, dtype=torch.uint8, device=dev)
    om = fwn._opts(precision=fwn.PRECISION_MIXED, traversal=trav, block_size=block, tuning=tuning)

    def q_mixed():
        fwn._check(L.fwn_query_ex(eng.handle, C.byref(om), C.c_void_p(Qd.data_ptr()), n,
                                  C.c_void_p(w.data_ptr()), C.c_void_p(ins.data_ptr()), None, None,
                                  sptr))
    for _ in range(warmup):
        q_mixed()
    torch.cuda.synchronize()
    ts = []
    for _ in range(steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        q_mixed()
        b.record(stream)
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b))
    ms = statistics.median(ts)
    _, _, w64 = eng.query(Qd, precision=fwn.PRECISION_FP64, traversal=fwn.TRAVERSAL_THREAD,
                          omega_f64=True)
    torch.cuda.synchronize()
    out = {"workload": wl.name, "triangles": int(len(wl.F)), "queries": n, "leaf_size": leaf,
           "tuning": tuning, "builder": builder, "value": n / (ms / 1e3), "unit": "queries/s",
           "ms_per_step": ms, "steps": steps, "build_ms": eng.info()["build_ms"],
           "step": "one query call (keys, sort, walk, scatter), CUDA events, median"}
    if cpu:
        import oracle
        nthr = oracle.nthreads_default()
        exact = oracle.brute_f64(wl.V, wl.F, wl.Q, nthreads=nthr)
        wm = w.cpu().numpy().astype(np.float64)
        w6 = w64.cpu().numpy()
        im = ins.cpu().numpy()
        dm, d6 = np.abs(wm - exact) / FOUR_PI, np.abs(w6 - exact) / FOUR_PI
        band = np.abs(exact / FOUR_PI - 0.5) > 1e-3
        out["vs_brute_force_fp64"] = {
            "points": n, "max_dw": float(dm.max()), "rms_dw": float(np.sqrt(np.mean(dm ** 2))),
            "fp64_form_max_dw": float(d6.max()), "mixed_vs_fp64_form_max_dw":
                float(np.max(np.abs(wm - w6)) / FOUR_PI),
            "inside_disagree_outside_band": int(np.sum(im[band] != (exact[band] / FOUR_PI > 0.5))),
            "note": "every point; includes the beta=2 far-field truncation error"}
        tree, kind, what = cpu_reference(wl.V, wl.F)
        tree.query(wl.Q[:1000], beta=wl.beta, nthreads=nthr)
        t0 = time.perf_counter()
        om_ref, in_ref = tree.query(wl.Q, beta=wl.beta, nthreads=nthr)
        dt = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": n / dt, "unit": "queries/s", "cores": nthr, "kind": kind,
                               "sample": f"all {n} queries; {what}"}
        out["inside_vs_reference"] = {
            "disagree_outside_band": int(np.sum(im[band] != in_ref[band])),
            "max_dw_vs_reference_restatement": float(np.max(np.abs(wm - om_ref)) / FOUR_PI)}
    eng.close()
    return out


def batched_summary(dev, *, steps=5, warmup=3, cpu=True, voxel=False):
    """A batched workload inside the default line. The 512-mesh forest (seed 3): its persistent
    CUDA-graph query, build, meshes/s, per-mesh FP64 launches with max |dw| over every query, and
    is_inside against the CPU restatement of the reference on sampled meshes. voxel=True: the 4
    displaced 5M-triangle meshes on 256^3 voxel-centre grids (the volume sign pass), the same
    figures plus the grid path that generates the centres on the device."""
    from lagrange_gb300 import workloads as W
    t0 = time.perf_counter()
    fo = W.voxel_workload() if voxel else W.batched_forest_workload()
    gen_s = time.perf_counter() - t0
    r = measure_forest(fo, dev, None, 0, 1, leaf=0, steps=steps, warmup=warmup, e2e=True, cpu=cpu,
                       fp64=True, clocks=False, grid=voxel)
    keep = ("value", "unit", "ms_per_step", "build_ms", "meshes_per_s_build_plus_query",
            "gpu_launches", "sort_key_bits", "plain_fp64_per_mesh_launches", "cpu_baseline",
            "inside_vs_reference", "grid_path")
    out = {"metric": r["metric"], **{k: r[k] for k in keep if k in r}}
    out["config"] = {**r["config"], "generation_s": gen_s}
    if "e2e" in r:
        out["e2e"] = {k: r["e2e"][k] for k in ("value", "unit", "ms_per_step", "h2d_bytes_per_step",
                                                "d2h_bytes_per_step", "api")}
        ph = r["e2e"].get("phases_ms_each") or {}
        out["e2e"]["phases_ms_mean"] = {k: sum(v) / len(v) for k, v in ph.items() if v}
    return out


def run_ours(args, rank, world, local):
    import torch
    torch.cuda.set_device(local)
    dist = init_dist(world, "nccl")
    dev = torch.device("cuda", local)
    import lagrange_gb300 as fwn
    from lagrange_gb300 import workloads as W

    wl = make_workload(args)
    if wl.near_mask is None:
        wl.near_mask = np.zeros(len(wl.Q), bool)
    if not args.split_queries:  # weak scaling: every rank answers its own full-size set
        wl.Q, wl.near_mask = rank_queries(wl.Q, wl.near_mask, rank)
    n = len(wl.Q)
    trav = fwn.TRAVERSAL_WARP if args.traversal == "warp" else fwn.TRAVERSAL_THREAD
    Vd = torch.from_numpy(wl.V).to(dev)
    Fd = torch.from_numpy(wl.F).to(dev)
    Qd = torch.from_numpy(wl.Q).to(dev)
    stream = torch.cuda.current_stream(dev)
    leaf, block, tuning, builder, tuned = args.leaf, args.block, args.tuning, args.builder, None
    if leaf == 0:  # the autotuner's choice for this mesh and query distribution (untimed)
        leaf, trav, block, tuning, builder, tuned = autotune_choice(fwn, Vd, Fd, Qd)
        leaf, trav, block, tuning, builder = rank0_choice(dist, (leaf, trav, block, tuning, builder),
                                                          dev)
    args.leaf, args.block = leaf, block
    # the handle's defaults are the chosen schedule too, so the host-buffer path (e2e) runs it
    eng = fwn.FastWindingNumber(Vd, Fd, leaf_size=args.leaf, traversal=trav, block_size=block,
                                tuning=tuning, builder=builder,
                                records=fwn.RECORDS_F32 | (0 if args.no_fp64 else fwn.RECORDS_F64))
    torch.cuda.synchronize()
    # build timing (device, CUDA events inside the library): best of 3 extra builds
    build_ms = []
    for _ in range(3):
        e2 = fwn.FastWindingNumber(Vd, Fd, leaf_size=args.leaf, builder=builder,
                                   records=fwn.RECORDS_F32)
        build_ms.append(e2.info()["build_ms"])
        e2.close()
    info = eng.info()
    w_out = torch.empty(n, dtype=torch.float32, device=dev)
    i_out = torch.empty(n, dtype=torch.uint8, device=dev)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)  # > L2 (129 MB)
    L = fwn.library()
    opts = fwn._opts(precision=fwn.PRECISION_MIXED, traversal=trav, block_size=args.block,
                     tuning=tuning)
    sptr = C.c_void_p(stream.cuda_stream)

    def query_mixed(s=None):
        fwn._check(L.fwn_query_ex(eng.handle, C.byref(opts), C.c_void_p(Qd.data_ptr()), n,
                                  C.c_void_p(w_out.data_ptr()), C.c_void_p(i_out.data_ptr()),
                                  None, None, sptr if s is None else C.c_void_p(s.cuda_stream)))

    for _ in range(args.warmup):
        query_mixed()
    torch.cuda.synchronize()
    step = query_mixed
    if not args.no_graph:
        # the timed step replays a CUDA graph of one query call (the same keys, sort and
        # traversal launches, without the host's launch overhead)
        side = torch.cuda.Stream(dev)
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            query_mixed(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            query_mixed(torch.cuda.current_stream(dev))
        graph.replay()
        torch.cuda.synchronize()
        step = graph.replay
    split_check = None
    if args.split_queries:
        # strong scaling: every rank computes the query order of the whole set, answers its
        # contiguous range of it and all-gathers the results (lagrange_gb300.shard)
        from lagrange_gb300 import shard
        gather = shard.torch_all_gather(dist) if dist is not None else (lambda x: [x])
        r_, w_ = (dist.get_rank(), dist.get_world_size()) if dist is not None else (0, 1)

        def step():
            order = eng.query_order(Qd)
            return shard.query_sharded(
                Qd, order, r_, w_,
                lambda sub: eng.query(sub.contiguous(), traversal=trav, sort_queries=False),
                gather)
        for _ in range(max(1, args.warmup)):
            step()
        query_mixed()
        ws, is_ = step()
        torch.cuda.synchronize()
        # each query's result depends on its own walk only, so the split set is bit-identical
        split_check = bool(torch.equal(ws, w_out) and torch.equal(is_, i_out))
    # work counters (untimed)
    _, _, stats = eng.query(Qd, traversal=trav, block_size=args.block, stats=True)
    torch.cuda.synchronize()

    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps)]
    barrier(dist)
    torch.cuda.synchronize()
    with Clocks(not args.no_clocks and rank == 0, local) as clk:
        t_wall = time.perf_counter()
        for k in range(args.steps):
            flush.zero_()  # L2 flush between timed steps (not inside the events)
            ev[k][0].record(stream)
            step()
            ev[k][1].record(stream)
        torch.cuda.synchronize()
        t_wall = time.perf_counter() - t_wall
    barrier(dist)
    step_ms = [a.elapsed_time(b) for a, b in ev]
    ms = sum(step_ms) / args.steps
    ms = max_over_ranks(dist, ms, dev)
    # strong scaling: the ranks share one set of n queries; weak: each rank answers n
    value = n / (ms / 1e3) if args.split_queries else job_value(n, world, ms / 1e3)
    clocks = clk.summary()

    result = {
        "metric": METRIC, "value": value, "unit": "queries/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
        "scaling": "strong" if args.split_queries else "weak", "vs_baseline": None,
        "dtype": "f32 (double-float/FP64 near field, FP64 refit)",
        "data": "synthetic",
        "config": {"workload": wl.name, "triangles": int(len(wl.F)),
                   "queries_per_gpu": n // world if args.split_queries else n,
                   "beta": wl.beta, "leaf_size": args.leaf,
                   "builder": BUILDER_NAMES.get(builder, str(builder)),
                   "traversal": ("auto", "thread", "warp")[trav],
                   "block": args.block, "tuning": tuning, "autotuned": tuned,
                   "step": "plain launches" if args.no_graph else "CUDA graph of one query call",
                   "l2": "flushed before every step (256 MB write)",
                   "parallelism": (f"tree replicas x{world}, one query set split in contiguous "
                                   f"ranges of the query order, results all-gathered"
                                   if args.split_queries else
                                   f"replicas x{world} (query shards, no collective)")},
        "build_ms": min(build_ms), "tree": {"nodes": info["num_nodes"], "leaves": info["num_leaves"],
                                            "device_bytes": info["device_bytes"]},
        "step_ms_min": min(step_ms), "step_ms_median": statistics.median(step_ms),
        "wall_s_timed": t_wall,
        "split_queries_bit_identical": split_check,
        "gpu_launches": query_launches(n, n, info["num_nodes"],
                                       auto=trav == fwn.TRAVERSAL_AUTO and tuning == 0) * args.steps,
        "clocks": clocks,
    }

    # ---- the traversal launch alone (roofline denominator) --------------------------------------
    # the points gathered once in the query's own Morton order and queried with sort_queries=0:
    # each call is then the status-word memset + one traversal launch, same warps, same results
    order = eng.query_order(Qd)
    Qs = Qd[order].contiguous()
    opts_k = fwn._opts(precision=fwn.PRECISION_MIXED, traversal=trav, block_size=args.block,
                       sort_queries=0, tuning=tuning)

    def query_kernel():
        fwn._check(L.fwn_query_ex(eng.handle, C.byref(opts_k), C.c_void_p(Qs.data_ptr()), n,
                                  C.c_void_p(w_out.data_ptr()), C.c_void_p(i_out.data_ptr()),
                                  None, None, sptr))

    for _ in range(max(3, args.warmup)):
        query_kernel()
    kev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
           for _ in range(args.steps)]
    torch.cuda.synchronize()
    for k in range(args.steps):
        flush.zero_()
        kev[k][0].record(stream)
        query_kernel()
        kev[k][1].record(stream)
    torch.cuda.synchronize()
    kernel_ms = sum(a.elapsed_time(b) for a, b in kev) / args.steps
    del Qs, order

    # ---- roofline from the counters --------------------------------------------------------
    far, tri, nodes = stats["far_evals"], stats["tri_evals"], stats["nodes_tested"]
    flops = far * FLOPS_FAR + tri * FLOPS_TRI + (nodes - far) * FLOPS_TEST
    l2_bytes = nodes * BYTES_NODE_TEST + far * BYTES_NODE_FAR + tri * BYTES_TRI + n * BYTES_QUERY_IO
    props = torch.cuda.get_device_properties(dev)
    sm_max = clocks.get("sm_max_mhz") or measured_peaks().get("sm_max_mhz") or 2070.0
    peak_nominal = props.multi_processor_count * 128 * 2 * sm_max * 1e6 / 1e12
    # the denominator, measured in this process on this GPU: FMA-throughput kernels in both FP32
    # instruction forms (scalar and paired f32x2); the faster one is the FP32 peak
    probes = {name: fwn.probe_fp32_peak(form, stream) for name, form in (("f32", 0), ("f32x2", 1))}
    peak_fp32 = max(p["tflops"] for p in probes.values())
    achieved = flops / (kernel_ms / 1e3) / 1e12
    # the warp-schedule variant the traversal ran (tuning 0 resolves by batch size, as in the
    # library: two queries per lane once the batch fills every SM's warp slots four times)
    variant = tuning or (4 if n >= 4 * props.multi_processor_count * 32 * 64 else 3)
    qpl = 2 if variant >= 4 else 1  # queries per lane of the variant
    traffic = NCU_TRAFFIC.get((wl.name, args.leaf, variant, builder)) if world == 1 else None
    hbm_peak = measured_peaks().get("hbm_gbs")
    result["roofline"] = {
        "bound": "fp32", "achieved": achieved, "peak": peak_fp32, "unit": "TFLOP/s",
        "frac": achieved / peak_fp32, "traffic": traffic,
        "kernel": "k_query_warp (traversal)", "variant": variant, "kernel_ms": kernel_ms,
        "kernel_share_of_step": kernel_ms / ms,
        "peak_source": "measured in this run: fwn_probe_fp32_peak (full-occupancy grid of "
                       "independent FMA chains, CUDA events, median of 5), the faster of the "
                       "scalar and paired-f32x2 forms (MEASURED_PEAKS.json has no FP32 figure)",
        "peak_measured": {k: v["tflops"] for k, v in probes.items()},
        "peak_nominal": peak_nominal,
        "traffic_source": (f"one-pass ncu capture (dram__bytes_read.sum + dram__bytes_write.sum) "
                           f"of the traversal launch of this workload at leaf {args.leaf}, "
                           f"variant {variant}, builder {builder}" if traffic else
                           "null: no capture for this workload / leaf / variant"),
        "hbm": ({"achieved_gbs": traffic / (kernel_ms / 1e3) / 1e9, "peak_gbs": hbm_peak,
                 "frac": traffic / (kernel_ms / 1e3) / 1e9 / hbm_peak,
                 "peak_source": "of measured (MEASURED_PEAKS.json hbm_gbs)"}
                if traffic and hbm_peak else None),
        "per_query": {"far_evals": far / n, "tri_evals": tri / n, "nodes_tested": nodes / n,
                      "tri_fp64": stats["tri_evals_fp64"] / n,
                      "warp_steps_per_warp": stats["warp_steps"] / math.ceil(n / (32 * qpl)),
                      "slot_utilisation": nodes / (stats["warp_steps"] * 32 * qpl),
                      "flops": flops / n, "l2_bytes": l2_bytes / n},
        "l2_gbs_algorithmic": l2_bytes / (kernel_ms / 1e3) / 1e9,
    }

    # ---- plain FP64 form + accuracy gate ----------------------------------------------------
    if not args.no_fp64:
        w64 = torch.empty(n, dtype=torch.float64, device=dev)
        o64 = fwn._opts(precision=fwn.PRECISION_FP64, traversal=fwn.TRAVERSAL_THREAD)

        def query_fp64():
            fwn._check(L.fwn_query_ex(eng.handle, C.byref(o64), C.c_void_p(Qd.data_ptr()), n,
                                      None, None, C.c_void_p(w64.data_ptr()), None, sptr))
        query_fp64()
        torch.cuda.synchronize()
        t64 = []
        for _ in range(max(1, args.fp64_steps)):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            query_fp64()
            b.record(stream)
            torch.cuda.synchronize()
            t64.append(a.elapsed_time(b))
        ms64 = sum(t64) / len(t64)
        query_mixed()
        torch.cuda.synchronize()
        dw = (w_out.double() - w64).abs() / FOUR_PI
        near = torch.from_numpy(wl.near_mask).to(dev)
        pct = percentiles
        result["plain_fp64"] = {
            "value": n / (ms64 / 1e3), "unit": "queries/s", "ms_per_step": ms64,
            "speedup_mixed_over_fp64": ms64 / ms,
            "max_dw": float(dw.max()), "rms_dw": float(dw.pow(2).mean().sqrt()),
            "max_dw_near": float(dw[near].max()) if bool(near.any()) else None,
            "max_dw_far": float(dw[~near].max()) if bool((~near).any()) else None,
            "dw_percentiles": {"near": pct(dw[near]), "far": pct(dw[~near])},
            "gate_1e-4": bool(float(dw.max()) <= 1e-4),
            "inside_disagree_band": int(((i_out.bool() != (w64 > 2 * math.pi)) &
                                         ((w64 / FOUR_PI - 0.5).abs() > 1e-3)).sum()),
        }
        # like-for-like: the FP64 form on the mixed form's warp schedule (same cursor and leaf
        # pairs), so that the speed-up from precision alone is separated from the schedule
        w64w = torch.empty(n, dtype=torch.float64, device=dev)
        o64w = fwn._opts(precision=fwn.PRECISION_FP64, traversal=fwn.TRAVERSAL_WARP)

        def query_fp64_warp():
            fwn._check(L.fwn_query_ex(eng.handle, C.byref(o64w), C.c_void_p(Qd.data_ptr()), n,
                                      None, None, C.c_void_p(w64w.data_ptr()), None, sptr))
        query_fp64_warp()
        torch.cuda.synchronize()
        t64w = []
        for _ in range(max(1, args.fp64_steps)):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            query_fp64_warp()
            b.record(stream)
            torch.cuda.synchronize()
            t64w.append(a.elapsed_time(b))
        ms64w = sum(t64w) / len(t64w)
        result["plain_fp64"]["warp_schedule"] = {
            "value": n / (ms64w / 1e3), "unit": "queries/s", "ms_per_step": ms64w,
            "speedup_mixed_over_fp64_warp": ms64w / ms,
            "speedup_warp_over_thread_fp64": ms64 / ms64w,
            "max_abs_domega_vs_thread_fp64": float((w64w - w64).abs().max()),
            "note": "FP64 records, Taylor terms and triangles on the mixed form's warp cursor "
                    "(one query per lane); same per-query sums as the thread FP64 form"}
        del w64, w64w

    # ---- e2e through the C ABI with host buffers ---------------------------------------------
    if not args.no_e2e:
        # strong scaling: each rank's host call takes its contiguous slice of the caller's array
        if args.split_queries:
            from lagrange_gb300 import shard
            q0, q1 = shard.shard_ranges(n, world)[rank]
        else:
            q0, q1 = 0, n
        ne = q1 - q0
        Qh = torch.from_numpy(wl.Q[q0:q1]).pin_memory()
        wh = torch.empty(ne, dtype=torch.float32).pin_memory()
        ih = torch.empty(ne, dtype=torch.uint8).pin_memory()

        def e2e_call():
            fwn._check(L.fwn_query_host(eng.handle, C.c_void_p(Qh.data_ptr()), ne,
                                        C.c_void_p(wh.data_ptr()), C.c_void_p(ih.data_ptr())))
        e2e_call()
        ts = []
        barrier(dist)
        for _ in range(max(3, args.steps // 2)):
            flush.zero_()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            e2e_call()
            ts.append(time.perf_counter() - t0)
        e2e_s = max_over_ranks(dist, sum(ts) / len(ts), dev)
        result["e2e"] = {"value": (n / e2e_s) if args.split_queries else job_value(n, world, e2e_s),
                         "unit": "queries/s",
                         "h2d_bytes_per_step": ne * 12, "d2h_bytes_per_step": ne * 5,
                         "ms_per_step": e2e_s * 1e3, "api": "fwn_query_host (pinned host buffers)"}

        # a serving loop: K batches in one fwn_query_host_batches call, batch b's copy in and
        # batch b - 1's copy out overlapping the walk between them (host wall clock, all copies
        # inside; the same pinned points each batch, results into the same pinned buffers)
        kb = max(3, args.steps)
        pts = (C.c_void_p * kb)(*([Qh.data_ptr()] * kb))
        cnt = (C.c_int64 * kb)(*([ne] * kb))
        pw = (C.c_void_p * kb)(*([wh.data_ptr()] * kb))
        pi = (C.c_void_p * kb)(*([ih.data_ptr()] * kb))

        def stream_call(k):
            fwn._check(L.fwn_query_host_batches(eng.handle, k, pts, cnt, pw, pi))
        stream_call(2)
        barrier(dist)
        flush.zero_()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        stream_call(kb)
        st_s = max_over_ranks(dist, (time.perf_counter() - t0) / kb, dev)
        result["e2e_stream"] = {
            "value": (n / st_s) if args.split_queries else job_value(n, world, st_s),
            "unit": "queries/s", "batches": kb, "ms_per_step": st_s * 1e3,
            "h2d_bytes_per_step": ne * 12, "d2h_bytes_per_step": ne * 5,
            "api": "fwn_query_host_batches (pinned host buffers, one batch per step; host "
                   "wall clock over the whole call)"}

    # ---- CPU baseline (rank 0, N=1 only) -----------------------------------------------------
    if rank == 0 and world == 1 and not args.no_cpu:
        import oracle
        nthr = oracle.nthreads_default()
        t0 = time.perf_counter()
        tree, kind, what = cpu_reference(wl.V, wl.F)
        build_s = time.perf_counter() - t0
        sample = cpu_sample(wl, args.cpu_sample)
        tree.query(sample[:1000], nthreads=nthr)
        t0 = time.perf_counter()
        om_cpu, in_cpu = tree.query(sample, beta=wl.beta, nthreads=nthr)
        dt = time.perf_counter() - t0
        s1 = sample[: max(1, len(sample) // 10)]
        t0 = time.perf_counter()
        tree.query(s1, beta=wl.beta, nthreads=1)
        dt1 = time.perf_counter() - t0
        result["cpu_baseline"] = {
            "value": len(sample) / dt, "unit": "queries/s", "cores": nthr, "kind": kind,
            "sample": f"{len(sample)} queries (half far, half near-surface) of the workload; "
                      f"{what}; build {build_s:.2f} s single-thread",
            "single_thread": {"value": len(s1) / dt1, "unit": "queries/s", "sample": len(s1)},
        }
        # is_inside agreement with the restated reference outside the +-1e-3 band, on every point
        # of the workload (the device results of the timed query; untimed CPU pass)
        t0 = time.perf_counter()
        om_all, in_all = tree.query(wl.Q, beta=wl.beta, nthreads=nthr)
        cpu_all_s = time.perf_counter() - t0
        query_mixed()  # the buffers may hold another pass's (permuted) results
        torch.cuda.synchronize()
        wg, ig = w_out.cpu().numpy(), i_out.cpu().numpy()
        band = np.abs(om_all / FOUR_PI - 0.5) > 1e-3
        dw_ref = np.abs(wg.astype(np.float64) - om_all) / FOUR_PI
        result["inside_vs_reference"] = {
            "points": int(len(wl.Q)), "outside_band": int(band.sum()),
            "disagree_outside_band": int(np.sum(ig[band] != in_all[band])),
            "max_dw_vs_reference_restatement": float(dw_ref.max()),
            "rms_dw_vs_reference_restatement": float(np.sqrt(np.mean(dw_ref ** 2))),
            "cpu_pass_s": cpu_all_s}
        # against the FP64 brute force over all triangles, on a stratified sample
        nb_pts = len(wl.Q) if len(wl.F) * len(wl.Q) <= 5e8 else args.brute
        bs = cpu_sample(wl, nb_pts, seed=11)
        exact = oracle.brute_f64(wl.V, wl.F, bs, nthreads=nthr)
        bq = torch.from_numpy(bs).to(dev)
        wm, _ = eng.query(bq, traversal=trav)
        torch.cuda.synchronize()
        dwb = np.abs(wm.cpu().numpy().astype(np.float64) - exact) / FOUR_PI
        half = len(bs) // 2 if wl.near_mask.any() else len(bs)
        result["vs_brute_force_fp64"] = {
            "sample": len(bs), "max_dw": float(dwb.max()), "rms_dw": float(np.sqrt(np.mean(dwb ** 2))),
            "max_dw_far": float(dwb[:half].max()),
            "max_dw_near": float(dwb[half:].max()) if half < len(bs) else None,
            "note": "includes the beta=2 far-field truncation error (same for the FP64 form)"}
        # FP64 brute force on the GPU: the FP64 form with beta = 1e30 evaluates every triangle
        # of every leaf exactly in FP64. Checked against O1 on the CPU sample, then run on a
        # larger stratified sample.
        if not args.no_fp64 and args.brute_gpu > 0:
            _, _, xb = eng.query(bq, precision=fwn.PRECISION_FP64,
                                  traversal=fwn.TRAVERSAL_THREAD, beta=1e30, omega_f64=True)
            torch.cuda.synchronize()
            check = float(np.max(np.abs(xb.cpu().numpy() - exact)) / FOUR_PI)
            gs = cpu_sample(wl, min(args.brute_gpu, len(wl.Q)), seed=12)
            gq = torch.from_numpy(gs).to(dev)
            t0 = time.perf_counter()
            _, _, xg = eng.query(gq, precision=fwn.PRECISION_FP64,
                                  traversal=fwn.TRAVERSAL_THREAD, beta=1e30, omega_f64=True)
            torch.cuda.synchronize()
            bt = time.perf_counter() - t0
            wmg, _ = eng.query(gq, traversal=trav)
            _, _, w64g = eng.query(gq, precision=fwn.PRECISION_FP64,
                                  traversal=fwn.TRAVERSAL_THREAD, omega_f64=True)
            torch.cuda.synchronize()
            xg = xg.cpu().numpy()
            dg = np.abs(wmg.cpu().numpy().astype(np.float64) - xg) / FOUR_PI
            d64 = np.abs(w64g.cpu().numpy() - xg) / FOUR_PI
            hg = len(gs) // 2 if wl.near_mask.any() else len(gs)
            result["vs_brute_force_fp64_gpu"] = {
                "sample": len(gs), "max_dw": float(dg.max()),
                "rms_dw": float(np.sqrt(np.mean(dg ** 2))),
                "max_dw_far": float(dg[:hg].max()),
                "max_dw_near": float(dg[hg:].max()) if hg < len(gs) else None,
                "fp64_form_max_dw": float(d64.max()),
                "fp64_form_rms_dw": float(np.sqrt(np.mean(d64 ** 2))),
                "brute_force_s": bt,
                "gpu_brute_vs_cpu_O1_max_dw": check,
                "note": "GPU FP64 all-triangle sums (FP64 form, beta=1e30); the mixed and FP64 "
                        "forms carry the same beta=2 truncation error"}

    # ---- the batched and defective-soup workloads (rank 0, N=1), after the headline ------------
    if rank == 0 and world == 1 and not args.no_batched and args.workload == "icosphere":
        eng.close()  # the headline's engine is done; the sub-workloads build their own
        torch.cuda.empty_cache()
        result["batched"] = batched_summary(dev, steps=min(args.steps, 5),
                                            warmup=max(3, min(args.warmup, 5)), cpu=not args.no_cpu)
        torch.cuda.empty_cache()
        result["soup"] = measure_soup(dev, steps=min(args.steps, 5),
                                      warmup=max(3, min(args.warmup, 5)), cpu=not args.no_cpu)
        torch.cuda.empty_cache()
        result["uvsphere"] = measure_uvsphere(dev, steps=max(args.steps, 10),
                                              warmup=max(3, min(args.warmup, 5)),
                                              cpu=not args.no_cpu)
        torch.cuda.empty_cache()
        result["voxel"] = batched_summary(dev, steps=min(args.steps, 5),
                                          warmup=max(3, min(args.warmup, 5)),
                                          cpu=not args.no_cpu, voxel=True)
    if rank == 0:
        print(json.dumps(result), flush=True)
    barrier(dist)
    if dist is not None:
        dist.destroy_process_group()


def run_forest(args, rank, world, local):
    """Batched workloads: `forest` (512 uneven spheres/tori, seed 3; `--meshes` for fewer) and
    `voxel` (4 x 5M-triangle meshes, each on a 256^3 voxel-centre grid). Build: one launch per stage over all meshes.
    Mixed query: one persistent launch over all meshes, captured in a CUDA graph and replayed.
    Plain form: FP64 everywhere, one launch per mesh."""
    import torch
    torch.cuda.set_device(local)
    dist = init_dist(world, "nccl")
    dev = torch.device("cuda", local)
    from lagrange_gb300 import workloads as W

    t0 = time.perf_counter()
    fo = W.batched_forest_workload(n_meshes=args.meshes) if args.workload == "forest" else W.voxel_workload(
        nu=args.nu or 500)
    gen_s = time.perf_counter() - t0
    result = measure_forest(fo, dev, dist, rank, world, leaf=args.leaf, builder=args.builder,
                            tuning=args.tuning, steps=args.steps,
                            warmup=args.warmup, e2e=not args.no_e2e, cpu=not args.no_cpu,
                            fp64=not args.no_fp64, clocks=not args.no_clocks,
                            grid=args.workload == "voxel", local=local)
    result["config"]["generation_s"] = gen_s
    if dist is not None:
        dist.destroy_process_group()
    return result


def measure_forest(fo, dev, dist, rank, world, *, leaf=0, builder=0, tuning=0, steps=10,
                   warmup=3, e2e=True, cpu=True, fp64=True, clocks=True, grid=False, local=0):
    """Measures one forest workload (see run_forest) and returns its result dict."""
    import torch
    import lagrange_gb300 as fwn
    M = len(fo.voff) - 1
    n = len(fo.Q)
    Vd = torch.from_numpy(fo.V).to(dev)
    Fd = torch.from_numpy(fo.F).to(dev)
    Qd = torch.from_numpy(fo.Q).to(dev)
    L = fwn.library()
    tuned = None
    if leaf == 0:  # builder and leaf size picked by the forest autotuner on this forest (untimed)
        r = fwn.autotune_forest(Vd, fo.voff, Fd, fo.foff, Qd, fo.qoff)
        leaf, tuning, builder = rank0_choice(dist, (r["leaf_size"], r["tuning"], r["builder"]), dev)
        tuned = {"leaf_size": r["leaf_size"], "tuning": r["tuning"], "builder": r["builder"],
                 "forest_query_ms": r["ms"], "candidates": r["candidates"]}
    builds = []
    for _ in range(3):
        f2 = fwn.Forest(Vd, fo.voff, Fd, fo.foff, leaf_size=leaf, builder=builder,
                        records=fwn.RECORDS_F32)
        builds.append(f2.info()["build_ms"])
        f2.close()
    forest = fwn.Forest(Vd, fo.voff, Fd, fo.foff, leaf_size=leaf, tuning=tuning, builder=builder,
                        records=fwn.RECORDS_F32 | (fwn.RECORDS_F64 if fp64 else 0))
    qoff = torch.from_numpy(fo.qoff.astype(np.int64)).pin_memory()  # pinned: capturable copy
    w = torch.empty(n, dtype=torch.float32, device=dev)
    ins = torch.empty(n, dtype=torch.uint8, device=dev)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    opts = fwn._opts(precision=fwn.PRECISION_MIXED, tuning=tuning)

    def q_mixed(stream_ptr):
        fwn._check(L.fwn_forest_query(forest.handle, C.c_void_p(Qd.data_ptr()),
                                      C.c_void_p(qoff.data_ptr()), C.c_void_p(w.data_ptr()),
                                      C.c_void_p(ins.data_ptr()), C.byref(opts), stream_ptr))
    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        for _ in range(warmup):
            q_mixed(C.c_void_p(side.cuda_stream))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        q_mixed(C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream(dev)
    ts = []
    with Clocks(clocks and rank == 0, local) as clk:
        for _ in range(steps):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            graph.replay()
            b.record(stream)
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
    ms = max_over_ranks(dist, sum(ts) / len(ts), dev)
    build_ms = min(builds)
    key_bits = fwn.forest_sort_key_bits(fo.qoff)  # the library's own choice for these offsets
    launches_per_query = query_launches(n, int(np.max(np.diff(fo.qoff))), forest.info()["num_nodes"] // M,
                                        math.ceil(math.log2(M)), key_bits, auto=tuning == 0)
    result = {
        "metric": f"winding queries/s, {M} meshes in one persistent CUDA-graph launch",
        "value": job_value(n, world, ms / 1e3), "unit": "queries/s", "n_gpus": world,
        "steps": steps, "warmup": warmup, "ms_per_step": ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32 (double-float/FP64 near field, FP64 refit)",
        "data": "synthetic",
        "config": {"workload": fo.name, "meshes": M, "triangles": int(fo.foff[-1]),
                   "queries": n, "beta": fo.beta, "leaf_size": leaf,
                   "builder": BUILDER_NAMES.get(builder, str(builder)), "autotuned": tuned,
                   "l2": "flushed before every step (256 MB write)"},
        "build_ms": build_ms, "tree_nodes": forest.info()["num_nodes"],
        "meshes_per_s_build_plus_query": M / ((build_ms + ms) / 1e3),
        "gpu_launches": launches_per_query * steps, "sort_key_bits": key_bits,
        "clocks": clk.summary(),
    }
    # ---- end to end: pinned host points in, Omega + inside out, through fwn_forest_query ------
    if e2e:
        Qh = torch.from_numpy(fo.Q).pin_memory()
        wh = torch.empty(n, dtype=torch.float32).pin_memory()
        ih = torch.empty(n, dtype=torch.uint8).pin_memory()
        Qe = torch.empty_like(Qd)
        sp = C.c_void_p(stream.cuda_stream)

        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]

        def e2e_call():
            ev[0].record(stream)
            Qe.copy_(Qh, non_blocking=True)
            ev[1].record(stream)
            fwn._check(L.fwn_forest_query(forest.handle, C.c_void_p(Qe.data_ptr()),
                                          C.c_void_p(qoff.data_ptr()), C.c_void_p(w.data_ptr()),
                                          C.c_void_p(ins.data_ptr()), C.byref(opts), sp))
            ev[2].record(stream)
            wh.copy_(w, non_blocking=True)
            ih.copy_(ins, non_blocking=True)
            ev[3].record(stream)
            stream.synchronize()
        e2e_call()
        te, phases = [], {"h2d": [], "query": [], "d2h": []}
        for _ in range(steps):
            flush.zero_()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            e2e_call()
            te.append(time.perf_counter() - t0)
            for k, (i, j) in zip(phases, ((0, 1), (1, 2), (2, 3))):
                phases[k].append(ev[i].elapsed_time(ev[j]))
        e2e_s = max_over_ranks(dist, sum(te) / len(te), dev)
        result["e2e"] = {"value": job_value(n, world, e2e_s), "unit": "queries/s",
                         "h2d_bytes_per_step": n * 12, "d2h_bytes_per_step": n * 5,
                         "ms_per_step": e2e_s * 1e3, "ms_each": [t * 1e3 for t in te],
                         "phases_ms_each": phases,
                         "api": "fwn_forest_query (pinned host points copied in, results out)"}
        del Qe
    # ---- CPU restatement of the reference path on a few meshes (rank 0, N=1) ---------------
    if rank == 0 and world == 1 and cpu:
        import oracle
        nthr = oracle.nthreads_default()
        rng = np.random.default_rng(21)
        picks = [0] if grid else sorted(rng.choice(M, 4, replace=False).tolist())
        wh_all, ih_all = w.cpu().numpy(), ins.cpu().numpy()
        nq_cpu, t_cpu, dis, maxdw, build_s = 0, 0.0, 0, 0.0, 0.0
        for m in picks:
            Vm = fo.V[fo.voff[m]:fo.voff[m + 1]]
            Fm = fo.F[fo.foff[m]:fo.foff[m + 1]]
            q0, q1 = int(fo.qoff[m]), int(fo.qoff[m + 1])
            idx = np.arange(q0, q1)  # every query of the mesh
            t0 = time.perf_counter()
            tree, kind, what = cpu_reference(Vm, Fm)
            build_s += time.perf_counter() - t0
            t0 = time.perf_counter()
            om, inn = tree.query(fo.Q[idx], beta=fo.beta, nthreads=nthr)
            t_cpu += time.perf_counter() - t0
            nq_cpu += len(idx)
            band = np.abs(om / FOUR_PI - 0.5) > 1e-3
            dis += int(np.sum(ih_all[idx][band] != inn[band]))
            maxdw = max(maxdw, float(np.max(np.abs(wh_all[idx] - om)) / FOUR_PI))
        result["cpu_baseline"] = {
            "value": nq_cpu / t_cpu, "unit": "queries/s", "cores": nthr, "kind": kind,
            "sample": f"all {nq_cpu} queries of meshes {picks}, one tree per mesh ({what}); "
                      f"builds {build_s:.2f} s single-thread, not in the rate"}
        result["inside_vs_reference"] = {"sample": nq_cpu, "disagree_outside_band": dis,
                                         "max_dw_vs_reference_restatement": maxdw}
    if grid:
        # the same classification through the grid sign pass: centres generated on the device,
        # no point array and no sort (one launch per mesh)
        res = round((fo.qoff[1] - fo.qoff[0]) ** (1 / 3))
        grids = []
        for m in range(M):
            Vm = fo.V[fo.voff[m]:fo.voff[m + 1]].astype(np.float64)
            lo, hi = Vm.min(0), Vm.max(0)
            c, h = (lo + hi) / 2, (hi - lo) / 2 * 1.05
            grids.append(((c - h).astype(np.float32), (2 * h / res).astype(np.float32)))
        wg = torch.empty(n, dtype=torch.float32, device=dev)
        ig = torch.empty(n, dtype=torch.uint8, device=dev)
        dims = (C.c_int64 * 3)(res, res, res)

        def q_grid():
            for m, (o, s) in enumerate(grids):
                q0 = int(fo.qoff[m])
                fwn._check(L.fwn_query_grid(forest.handle, m, (C.c_float * 3)(*o), (C.c_float * 3)(*s),
                                            dims, C.c_void_p(wg.data_ptr() + 4 * q0),
                                            C.c_void_p(ig.data_ptr() + q0),
                                            C.c_void_p(stream.cuda_stream)))
        q_grid()
        torch.cuda.synchronize()
        tg = []
        for _ in range(steps):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            q_grid()
            b.record(stream)
            torch.cuda.synchronize()
            tg.append(a.elapsed_time(b))
        msg = sum(tg) / len(tg)
        result["grid_path"] = {
            "value": n / (msg / 1e3), "unit": "queries/s", "ms_per_step": msg, "launches": M,
            "api": "fwn_query_grid (voxel centres generated on the device, no point array)",
            "inside_fraction": float(ig.float().mean()),
            "inside_fraction_explicit_points": float(ins.float().mean()),
            "h2d_bytes_per_step": 0}
    if fp64:
        w64 = torch.empty(n, dtype=torch.float32, device=dev)
        o64 = fwn._opts(precision=fwn.PRECISION_FP64, traversal=fwn.TRAVERSAL_THREAD)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        fwn._check(L.fwn_forest_query(forest.handle, C.c_void_p(Qd.data_ptr()),
                                      C.c_void_p(qoff.data_ptr()), C.c_void_p(w64.data_ptr()),
                                      None, C.byref(o64), C.c_void_p(stream.cuda_stream)))
        b.record(stream)
        torch.cuda.synchronize()
        ms64 = a.elapsed_time(b)
        dw = (w.double() - w64.double()).abs() / FOUR_PI
        band = (w64.double() / FOUR_PI - 0.5).abs() > 1e-3
        result["plain_fp64_per_mesh_launches"] = {
            "value": n / (ms64 / 1e3), "unit": "queries/s", "ms": ms64, "launches": M,
            "speedup_mixed_over_fp64": ms64 / ms,
            "max_dw": float(dw.max()), "rms_dw": float(dw.pow(2).mean().sqrt()),
            "note": "FP64 output rounded to float; |dw| includes that rounding (<= 4e-8)",
            "inside_disagree_band": int(((ins.bool() != (w64.double() > 2 * math.pi)) & band).sum()),
        }
    return result


def main():
    args = parse()
    rank, world, local = dist_env()
    if args.impl == "reference":
        run_reference(args, rank, world)
    elif args.workload in ("forest", "voxel"):
        result = run_forest(args, rank, world, local)
        if rank == 0:
            print(json.dumps(result), flush=True)
    else:
        run_ours(args, rank, world, local)


if __name__ == "__main__":
    main()
