"""The work that a user of this framework has it do, as cases that can be timed and compared.

Each case goes through the public entry points (FastWindingNumber, Forest and their methods) with
seeded synthetic inputs of this repository's own workload families: displaced geodesic spheres, a
UV sphere, the defective soup (holes, flipped and jittered duplicate facets), forests of spheres
and tori, voxel grids. Query points lie half in the mesh's bounding box grown by 20 %, half close
to the surface on both sides, as in those workloads, unless a case says otherwise.

A case is a dict of plain values. Meshes: "nu" is the frequency of a geodesic sphere (20 nu^2
triangles; 0: the 64 x 32 UV sphere, 3,968 triangles), "soup" 1 makes its facets defective.
"builder", "leaf", "precision" are the configuration's fields (their defaults: LBVH, 8, mixed).
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

MIXED, FP64 = fwn.PRECISION_MIXED, fwn.PRECISION_FP64
LBVH, SPLIT, BINNED = fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED


def listed():
    return [
        # The reference's own call: one point on the host, one answer (picking, a caller's loop).
        {"name": "point", "kind": "host_point", "nu": 0},
        # A small batch on the device: the probes of one step of an interactive tool.
        {"name": "query_4k", "kind": "query", "nu": 0, "queries": 4096},
        # The UV-sphere workload: 100k points against 3,968 triangles, uniform in the box.
        {"name": "query_100k", "kind": "query", "nu": 0, "queries": 100_000, "near": 0},
        # The 2M-triangle workload: one large mesh queried many times, built for that (binned).
        {"name": "query_10m", "kind": "query", "nu": 316, "queries": 10_000_000, "builder": BINNED},
        # The defective soup, default configuration: a scan that has to be signed as it is.
        {"name": "soup_5m", "kind": "query", "nu": 224, "queries": 5_000_000, "soup": 1},
        # The FP64 form, for callers who want every digit: 20k triangles, 100k points.
        {"name": "fp64_100k", "kind": "query", "nu": 32, "queries": 100_000, "precision": FP64},
        # A small mesh from host arrays, built and asked a few points: a part of a scene.
        {"name": "build_4k", "kind": "build_host", "nu": 0, "queries": 1000},
        # A large mesh on the device, built and asked once: the cost of the build itself.
        {"name": "build_2m", "kind": "build", "nu": 316, "queries": 100_000, "builder": SPLIT},
        # A batch of meshes built and queried together (1k to 500k triangles, 1k to 1M queries each).
        {"name": "forest_64", "kind": "forest", "meshes": 64, "f_lo": 1000, "f_hi": 500_000,
         "q_lo": 1000, "q_hi": 1_000_000, "builder": SPLIT, "sizes": 3},
        # The sign pass of a voxelizer, ragged dimensions, a 1M-triangle mesh.
        {"name": "grid_213x200x187", "kind": "grid", "nu": 224, "nx": 213, "ny": 200, "nz": 187},
        # Orientation repair: 10 % of the facets flipped, two queries per facet.
        {"name": "orient_500k", "kind": "orient", "nu": 158, "ref_nu": 100},
        # A server's loop over point sets in pinned host memory.
        {"name": "batches_6x1m", "kind": "batches", "nu": 224, "batches": 6, "queries": 1_000_000,
         "builder": SPLIT},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["host_point", "query", "query", "query", "fp64", "build_host", "build",
                       "forest", "grid", "orient", "batches"])
    nu = _log(rng, 7, 316)
    opt = {"builder": rng.choice([LBVH, SPLIT, BINNED]), "leaf": rng.choice([4, 8, 8, 12, 16])}
    if kind == "host_point":
        return {"kind": kind, "nu": nu, **opt}
    if kind == "query":
        return {"kind": kind, "nu": nu, "queries": _log(rng, 1000, 8_000_000),
                "soup": int(rng.random() < 0.25), "near": int(rng.random() < 0.75), **opt}
    if kind == "fp64":
        return {"kind": "query", "nu": min(nu, 60), "queries": _log(rng, 1000, 60_000),
                "precision": FP64, **opt}
    if kind == "build_host":
        return {"kind": kind, "nu": min(nu, 60), "queries": _log(rng, 1, 20_000), **opt}
    if kind == "build":
        return {"kind": kind, "nu": nu, "queries": _log(rng, 1000, 200_000), **opt}
    if kind == "forest":
        return {"kind": kind, "meshes": _log(rng, 2, 64), "f_lo": 1000, "f_hi": _log(rng, 2000, 300_000),
                "q_lo": 1000, "q_hi": _log(rng, 2000, 500_000), "sizes": rng.randrange(1000), **opt}
    if kind == "grid":
        return {"kind": kind, "nu": nu, "nx": _log(rng, 17, 220), "ny": _log(rng, 17, 200),
                "nz": _log(rng, 17, 190), **opt}
    if kind == "orient":
        return {"kind": kind, "nu": min(nu, 200), "ref_nu": _log(rng, 7, 200), **opt}
    return {"kind": kind, "nu": nu, "batches": rng.randrange(1, 8), "queries": _log(rng, 1000, 1_000_000),
            **opt}


# ---- inputs --------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _sphere(nu):
    """Unit directions and facets of a geodesic sphere (nu > 0) or of the UV sphere (nu = 0)."""
    V, F = W.icosphere(nu) if nu else W.uv_sphere(64, 32)
    return np.asarray(V, np.float64), F


@functools.lru_cache(maxsize=None)
def _torus(nu, nv, ratio):
    _, F, n, c = W.torus_grid(nu, nv, 1.0, 1.0 / ratio)
    return n, c, F


def _bumps(dirs, rng, k=8):
    """Sum of k sines over directions (float64 CUDA tensor), amplitudes up to 0.02."""
    a, f = rng.uniform(0.0, 0.02, k), rng.uniform(2.0, 12.0, k)
    d = rng.normal(size=(k, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    phi = rng.uniform(0.0, 2 * np.pi, k)
    s = torch.zeros(len(dirs), dtype=torch.float64, device="cuda")
    for ak, fk, dk, pk in zip(a, f, d, phi):
        s += ak * torch.sin(fk * (dirs * torch.from_numpy(dk).cuda()).sum(1) + pk)
    return s


def _mesh(nu, seed, soup=0):
    """Displaced sphere as CUDA tensors (float32 vertices, int32 facets)."""
    rng = np.random.default_rng([seed, nu])
    P, F = _sphere(nu)
    P = torch.from_numpy(P).cuda()
    V = (P * (1.0 + _bumps(P, rng))[:, None]).float()
    F = torch.from_numpy(F).cuda()
    if soup:  # 10 % of the facets deleted, 1 % flipped, 0.5 % duplicated with 1e-7 jitter
        g = torch.Generator(device="cuda").manual_seed(seed)
        F = F[torch.rand(len(F), generator=g, device="cuda") >= 0.1]
        flip = torch.rand(len(F), generator=g, device="cuda") < 0.01
        F = torch.where(flip[:, None], F[:, [0, 2, 1]], F)
        dup = F[torch.rand(len(F), generator=g, device="cuda") < 0.005].long().reshape(-1)
        jit = (torch.rand((len(dup), 3), generator=g, device="cuda", dtype=torch.float64) - 0.5) * 2e-7
        F = torch.cat([F, (len(V) + torch.arange(len(dup), device="cuda")).int().reshape(-1, 3)])
        V = torch.cat([V, (V[dup].double() + jit).float()])
    return V.contiguous(), F.contiguous()


def _points(V, F, n, seed, near=1, off_hi=1e-3):
    """n query points: the box grown by 20 %, the second half (near = 1) within off_hi of the
    surface along the facet normals, on both sides."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1000)
    rnd = lambda *s: torch.rand(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    lo, hi = V.min(0).values.double(), V.max(0).values.double()
    nb = n - n // 2 if near else n
    Q = (lo + hi) / 2 + (rnd(nb, 3) * 2 - 1) * (hi - lo) / 2 * 1.2
    if n - nb:
        m = n - nb
        a, b, c = (V[F[:, j].long()].double() for j in range(3))
        nrm = torch.cross(b - a, c - a, dim=1)
        area = nrm.norm(dim=1)
        cdf = area.cumsum(0)
        t = torch.searchsorted(cdf, rnd(m) * cdf[-1]).clamp(max=len(F) - 1)
        r1, r2 = rnd(m).sqrt()[:, None], rnd(m)[:, None]
        p = (1 - r1) * a[t] + r1 * (1 - r2) * b[t] + r1 * r2 * c[t]
        off = torch.where(rnd(m) < 0.5, -1.0, 1.0) * (1e-6 + rnd(m) * (off_hi - 1e-6))
        Q = torch.cat([Q, p + off[:, None] * nrm[t] / area[t].clamp(min=1e-300)[:, None]])
    return Q.float().contiguous()


def _forest(case, seed):
    """Meshes' concatenated vertices and facets, query points, and the three host offset arrays.
    Mesh sizes and query counts come from the case, shapes and points from the seed."""
    size = random.Random(case["sizes"])
    rng = np.random.default_rng([seed, case["meshes"]])
    Vs, Fs, Qs = [], [], []
    for m in range(case["meshes"]):
        nf, nq = _log(size, case["f_lo"], case["f_hi"]), _log(size, case["q_lo"], case["q_hi"])
        if size.random() < 0.5:
            P, F = _sphere(max(7, round(math.sqrt(nf / 20))))
            P = torch.from_numpy(P).cuda()
            V = P * (1.0 + _bumps(P, rng))[:, None]
        else:
            ratio = round(size.uniform(2.0, 5.0), 2)
            nv = max(6, round(math.sqrt(nf / (2 * ratio))))
            n, c, F = _torus(max(6, round(nf / (2 * nv))), nv, ratio)
            n = torch.from_numpy(n).cuda()
            V = torch.from_numpy(c).cuda() + (1.0 / ratio * (1.0 + _bumps(n, rng)))[:, None] * n
        Vs.append(V.float())
        Fs.append(torch.from_numpy(F).cuda())
        Qs.append(_points(Vs[-1], Fs[-1], nq, seed + 7 * m, near=0))
    off = [np.concatenate([[0], np.cumsum([len(x) for x in xs])]).astype(np.int64) for xs in (Vs, Fs, Qs)]
    return torch.cat(Vs), torch.cat(Fs), torch.cat(Qs), *off


def _config(case):
    precision = case.get("precision", MIXED)
    return {"builder": case.get("builder", LBVH), "leaf_size": case.get("leaf", 8),
            "precision": precision,
            "records": fwn.RECORDS_F64 if precision == FP64 else fwn.RECORDS_F32}


# ---- cases ---------------------------------------------------------------------------------------


def prepare(case, seed):
    kind, s = case["kind"], {"case": case, "config": _config(case)}
    if kind == "forest":
        s["V"], s["F"], s["Q"], s["voff"], s["foff"], s["qoff"] = _forest(case, seed)
        return s
    V, F = _mesh(case.get("ref_nu", case["nu"]), seed, case.get("soup", 0))
    if kind == "build":
        return {**s, "V": V, "F": F, "Q": _points(V, F, case["queries"], seed)}
    if kind == "build_host":
        return {**s, "V": V.cpu().numpy(), "F": F.cpu().numpy(),
                "Q": _points(V, F, case["queries"], seed).cpu().numpy()}
    s["engine"] = fwn.FastWindingNumber(V, F, **s["config"])
    if kind == "query":
        s["Q"] = _points(V, F, case["queries"], seed, case.get("near", 1),
                         1e-4 if case.get("soup") else 1e-3)
    elif kind == "host_point":
        s["Q"] = _points(V, F, 2, seed, near=0)[0].cpu().numpy()
    elif kind == "grid":
        lo, hi = (np.asarray(x, np.float64) for x in (V.min(0).values.tolist(), V.max(0).values.tolist()))
        c, h = (lo + hi) / 2, (hi - lo) / 2 * 1.05
        s["origin"] = (c - h).tolist()
        s["spacing"] = (2 * h / np.array([case["nx"], case["ny"], case["nz"]])).tolist()
    elif kind == "orient":
        s["V"], F = _mesh(case["nu"], seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        flip = torch.rand(len(F), generator=g, device="cuda") < 0.1
        s["F"] = torch.where(flip[:, None], F[:, [0, 2, 1]], F).contiguous()
    elif kind == "batches":
        s["Q"] = [_points(V, F, case["queries"], seed + 31 * b).cpu().pin_memory()
                  for b in range(case["batches"])]
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "host_point":
        return s["engine"].solid_angle(s["Q"])
    if kind == "query":
        if case.get("precision", MIXED) == FP64:
            omega, inside, omega64 = s["engine"].query(s["Q"], omega_f64=True)
            return {"omega": omega, "inside": inside, "omega64": omega64}
        omega, inside = s["engine"].query(s["Q"])
        return {"omega": omega, "inside": inside}
    if kind in ("build", "build_host"):
        engine = fwn.FastWindingNumber(s["V"], s["F"], **s["config"])
        omega, inside = engine.query(s["Q"])
        engine.close()
        return {"omega": omega, "inside": inside}
    if kind == "forest":
        forest = fwn.Forest(s["V"], s["voff"], s["F"], s["foff"], **s["config"])
        omega, inside = forest.query_forest(s["Q"], s["qoff"])
        forest.close()
        return {"omega": omega, "inside": inside}
    if kind == "grid":
        omega, inside = s["engine"].query_grid(s["origin"], s["spacing"], (case["nx"], case["ny"], case["nz"]))
        return {"omega": omega, "inside": inside}
    if kind == "orient":
        criterion, flip = s["engine"].orientation_criterion(s["V"], s["F"])
        return {"criterion": criterion, "flip": flip}
    return {"batch%d" % b: {"omega": w, "inside": i}
            for b, (w, i) in enumerate(s["engine"].query_host_batches(s["Q"]))}


def _sizes(case):
    """(triangles, queries, meshes' triangles per mesh) of one pass."""
    tris = lambda nu: 20 * nu * nu if nu else 3968  # noqa: E731
    kind = case["kind"]
    if kind == "forest":
        size, nf, nq = random.Random(case["sizes"]), 0, 0
        for _ in range(case["meshes"]):
            nf += _log(size, case["f_lo"], case["f_hi"])
            nq += _log(size, case["q_lo"], case["q_hi"])
            if size.random() >= 0.5:
                size.uniform(2.0, 5.0)
        return nf, nq, nf / case["meshes"]
    if kind == "orient":
        return tris(case["nu"]), 2 * tris(case["nu"]), tris(case["ref_nu"])
    n = {"host_point": 1, "grid": case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 0),
         "batches": case.get("batches", 0) * case.get("queries", 0)}.get(kind, case.get("queries", 0))
    return tris(case["nu"]), n, tris(case["nu"])


def work(case):
    """One pass: the mesh and the points read, the answers written; the operations of the walk
    (per query of a tree over f triangles about 4.3 log2 f expansion terms of 82, 4.7 log2 f far
    tests of 12, and 30 triangles of 95 operations) and of the moments (about 400 per triangle)."""
    nf, nq, f = _sizes(case)
    kind = case["kind"]
    out = 13 if case.get("precision", MIXED) == FP64 else 5
    nbytes = nq * (out if kind in ("grid", "orient") else 12 + out)
    flops = nq * (math.log2(f) * (4.3 * 82 + 4.7 * 12) + 30 * 95)
    if kind in ("build", "build_host", "forest", "orient"):
        nbytes += nf * (12 + 6)
    if kind in ("build", "build_host", "forest"):
        flops += 400 * nf
    return {"bytes": nbytes, "flops": flops}


def _solid_angle(V, F, Q):
    """Sum of the triangles' solid angles (Van Oosterom and Strackee 1983), float64, all pairs."""
    a, b, c = (V.double()[F[:, j].long()].T[:, None, :] for j in range(3))
    out = torch.zeros(len(Q), dtype=torch.float64, device=V.device)
    dot = lambda x, y: x[0] * y[0] + x[1] * y[1] + x[2] * y[2]  # noqa: E731
    step = max(1, (1 << 26) // max(1, len(F)))
    for i in range(0, len(Q), step):
        q = Q[i:i + step].double().T[:, :, None]
        A, B, C = a - q, b - q, c - q
        la, lb, lc = (dot(x, x).sqrt() for x in (A, B, C))
        det = (A[0] * (B[1] * C[2] - B[2] * C[1]) + A[1] * (B[2] * C[0] - B[0] * C[2]) +
               A[2] * (B[0] * C[1] - B[1] * C[0]))
        den = la * lb * lc + dot(A, B) * lc + dot(B, C) * la + dot(C, A) * lb
        t = torch.where((det == 0) | (la == 0) | (lb == 0) | (lc == 0), 0.0, 2 * torch.atan2(det, den))
        out[i:i + step] = t.sum(1)
    return out


def exact(case, seed):
    """Every triangle's solid angle in float64 (the engine's answers carry the expansion's error on
    top of rounding), where the pairs are few enough."""
    kind = case["kind"]
    nf, nq, f = _sizes(case)
    if kind in ("forest", "grid", "orient", "batches") or f * nq > 3e9:
        return None
    V, F = _mesh(case["nu"], seed, case.get("soup", 0))
    if kind == "host_point":
        return float(_solid_angle(V, F, _points(V, F, 2, seed, near=0)[:1])[0])
    Q = _points(V, F, case["queries"], seed, case.get("near", 1), 1e-4 if case.get("soup") else 1e-3)
    w = _solid_angle(V, F, Q)
    res = {"omega": w, "inside": None}
    if kind == "query" and case.get("precision", MIXED) == FP64:
        res["omega64"] = w
    return res
