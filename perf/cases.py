"""What users of this framework have it do, as timed cases.

A case is one pass through the framework's public entry points with the data a
program holds before the call: meshes and masks in host arrays, the GPU context
and the proposer's weights kept from one call to the next. `listed()` names the
cases, `draw(rng)` gives more of the same ranges, `prepare` makes a case's
inputs from a seed, `run` is one pass, `work` what the pass cannot do without
and `exact` its outputs in 64 bits, where they are computed numbers.

Kinds (the decomposition's stages in the order a decomposition meets them):

  matrix    visibility edges of one part against its cage, everything in one
            call: BVH builds, visibility, the edge list
  parts     the new sub-parts of a split: their BVHs and cages' BVHs, one
            batched visibility call over the pairs with a new endpoint
  split     the split-plane search: the drawn edges' candidate planes, scored
  learned   the same search with the learned proposer in front
  score     plane scoring on device arrays (the precision sweep's shape)
  clip      one part cut by a plane
  remesh    the signed-distance remesh that makes bodies and cages
  concavity the sampled Hausdorff distances of all parts to their hulls
  hulls     the union hulls of one pass of hull merging
  train     loss and gradients of one proposer training batch
  process   a whole decomposition
"""
from __future__ import annotations

import math

import numpy as np
import torch

from visacd_gb300 import _native, meshgen, proposer
from visacd_gb300 import visacd as V

_kept: dict = {}


def _context() -> _native.Context:
    """The GPU context a program keeps for all its calls."""
    if "ctx" not in _kept:
        _kept["ctx"] = _native.Context(0)
    return _kept["ctx"]


def _proposer() -> _native.PlaneProposer:
    """The proposer with the shipped weights, kept like the context."""
    if "lp" not in _kept:
        _kept["lp"] = _native.PlaneProposer(_context(), params=proposer.load_params())
    return _kept["lp"]


# ---- cases -------------------------------------------------------------------


def listed():
    return [
        # The smallest call: a fragment late in a decomposition (162 vertices,
        # 13 thousand pairs); launches and waits count.
        {"name": "matrix_fragment", "kind": "matrix", "shape": "blob", "f": 4, "offset": 0.03},
        # The benchmark's workload: 10,242 vertices, 52 million pairs.
        {"name": "matrix_blob_s5", "kind": "matrix", "shape": "blob", "f": 32, "offset": 0.03},
        # A split of a remeshed body: both halves against their own remeshed
        # cages, only pairs with a vertex on the cut.
        {"name": "parts_of_split", "kind": "parts", "shape": "blob", "f": 16, "stretch": 0.8},
        # The split search on a large part, with the reference's 2500 planes.
        {"name": "split_blob_s5", "kind": "split", "shape": "blob", "f": 32, "planes": 2500},
        # The learned search on an ordinary part (one proposal, 64 probe planes).
        {"name": "learned_blob_s4", "kind": "learned", "shape": "blob", "f": 16, "planes": 64},
        # The precision sweep's shape: a million edges against 4096 planes.
        {"name": "score_sweep", "kind": "score", "edges": 1 << 20, "planes": 4096},
        # A remeshed body cut near its centre.
        {"name": "clip_body", "kind": "clip", "shape": "blob", "f": 32, "stretch": 1.0},
        # The cage of the largest benchmark blob.
        {"name": "remesh_cage", "kind": "remesh", "shape": "blob", "f": 32, "stretch": 1.0, "scale": 40.0,
         "level": 0.03},
        # The concavity of a decomposition's parts midway (12 parts, 3000 samples per unit of area).
        {"name": "concavity_12_parts", "kind": "concavity", "shape": "blob", "f": 16, "stretch": 0.8, "parts": 12,
         "samples": 3000},
        # One pass of hull merging: the union hulls of the 96 closest pairs of 32 parts.
        {"name": "hulls_merge_pass", "kind": "hulls", "shape": "blob", "f": 16, "parts": 32, "pairs": 96},
        # One training batch of the proposer (64 parts of 2048 edges, 8 labels).
        {"name": "train_batch_64", "kind": "train", "batch": 64, "labels": 8},
        # A whole decomposition as the benchmark runs it on its held-out blobs.
        {"name": "process_blob_s4", "kind": "process", "shape": "blob", "f": 16, "stretch": 1.0, "concavity": 0.02,
         "parts": 64, "search": "exhaustive"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matrix", "matrix", "parts", "parts", "split", "learned", "score", "clip", "remesh",
                       "concavity", "hulls", "train", "process"])
    shape = rng.choice(["blob", "blob", "torus"])
    stretch = round(rng.uniform(0.35, 1.0), 3)
    if kind == "matrix":
        return {"kind": kind, "shape": shape, "f": _log_int(rng, 3, 32), "offset": round(rng.uniform(0.02, 0.05), 4)}
    if kind in ("parts", "clip"):
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 32), "stretch": stretch}
    if kind == "split":
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 32), "planes": _log_int(rng, 60, 2500)}
    if kind == "learned":
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 32), "planes": _log_int(rng, 16, 256)}
    if kind == "score":
        return {"kind": kind, "edges": _log_int(rng, 500, 1 << 20), "planes": _log_int(rng, 16, 4096)}
    if kind == "remesh":
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 32), "stretch": stretch,
                "scale": round(rng.uniform(15.0, 40.0), 2), "level": round(rng.uniform(0.02, 0.03), 4)}
    if kind == "concavity":
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 32), "stretch": stretch,
                "parts": _log_int(rng, 1, 12), "samples": rng.randint(1000, 3000)}
    if kind == "hulls":
        parts = rng.randint(4, 32)
        return {"kind": kind, "shape": shape, "f": rng.randint(8, 16), "parts": parts,
                "pairs": rng.randint(1, 3 * parts)}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "labels": rng.randint(1, 8)}
    return {"kind": kind, "shape": shape, "f": rng.randint(8, 20), "stretch": stretch,
            "concavity": round(rng.uniform(0.02, 0.1), 3), "parts": rng.randint(2, 24),
            "search": rng.choice(["exhaustive", "learned"])}


# ---- inputs ------------------------------------------------------------------


def _geodesic(f: int):
    """The icosahedron with every edge divided in f, on the unit sphere:
    10 f^2 + 2 vertices, 20 f^2 triangles."""
    v0, t0 = meshgen.icosphere(0)
    rows = np.array([(i, j) for i in range(f + 1) for j in range(f + 1 - i)], dtype=np.float64)
    at = -np.ones((f + 2, f + 2), dtype=np.int64)
    for k, (i, j) in enumerate(rows.astype(np.int64)):
        at[i, j] = k
    tri = []
    for i in range(f):
        for j in range(f - i):
            tri.append((at[i, j], at[i + 1, j], at[i, j + 1]))
            if j < f - i - 1:
                tri.append((at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]))
    tri = np.array(tri, dtype=np.int64)
    a, b, c = v0[t0[:, 0]], v0[t0[:, 1]], v0[t0[:, 2]]
    w = rows / f
    p = (a[:, None] * (1 - w.sum(1))[None, :, None] + b[:, None] * w[None, :, :1] + c[:, None] * w[None, :, 1:])
    p = p.reshape(-1, 3)
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    t = (tri[None] + len(rows) * np.arange(len(t0))[:, None, None]).reshape(-1, 3)
    _, first, inv = np.unique(np.round(p, 7), axis=0, return_index=True, return_inverse=True)
    return p[first], inv.reshape(-1)[t].astype(np.int32)


def _mesh(case, seed: int):
    """The case's raw mesh: a displaced sphere (the benchmark's blob at any
    edge division) or a perturbed torus."""
    f = case["f"]
    if case["shape"] == "torus":
        return meshgen.torus(1.0, 0.35, 2 * f, f, 0.02, seed=seed % (1 << 31))
    rng = np.random.default_rng([seed, 1])
    v, t = _geodesic(f)
    a = rng.uniform(-1.0, 1.0, size=8)
    c = rng.normal(size=(8, 3))
    c /= np.linalg.norm(c, axis=1, keepdims=True)
    d2 = ((v[:, None, :] - c[None, :, :]) ** 2).sum(-1)
    return v * (1.0 + 0.3 * (a * np.exp(-d2 / (2.0 * 0.15 * 0.15))).sum(-1))[:, None], t


def _normal(v: np.ndarray, stretch: float = 1.0) -> np.ndarray:
    """Stretched along y and z, then into [-1, 1] by the longest side, as a
    decomposition begins."""
    v = v * np.array([1.0, stretch, stretch])
    lo, hi = v.min(axis=0), v.max(axis=0)
    return 2.0 * (v - 0.5 * (lo + hi)) / float((hi - lo).max())


def _body(case, seed: int):
    """The remeshed body a decomposition works on (its grid sizes)."""
    v, t = _mesh(case, seed)
    v = _normal(v, case.get("stretch", 1.0))
    bv, bt = _context().sdf_remesh(v, t, 30.0, 0.55 / 30)
    if len(bv) > 15000:
        bv, bt = _context().sdf_remesh(v, t, 20.0, 0.55 / 20)
    return bv, bt


def _plane_through(v: np.ndarray, rng) -> list:
    n = rng.normal(size=3)
    n /= np.linalg.norm(n)
    return [*n, -float(n @ (0.5 * (v.min(axis=0) + v.max(axis=0)))) + float(rng.uniform(-0.05, 0.05))]


def _pieces(v, t, count: int, rng):
    """The mesh cut by `count` - 1 planes, always the piece with most vertices."""
    parts = [{"vertices": v, "triangles": t}]
    for _ in range(8 * count):
        if len(parts) >= count:
            break
        k = max(range(len(parts)), key=lambda i: len(parts[i]["vertices"]))
        p = parts[k]
        halves, _, _ = V._clip(p["vertices"], p["triangles"], _plane_through(p["vertices"], rng))
        if len(halves) == 2 and min(len(h["vertices"]) for h in halves) >= 10:
            parts[k:k + 1] = halves
    return parts


def _edges_of(v, t):
    cv, ct = meshgen.offset_cage(v, t, 0.03)
    return _context().compute_intersection_matrix(v, t, cv, ct)[0]


# Results whose size depends on the input go to arrays the program keeps, with
# room for the largest result of the case (rows, columns, type).
def _room(case):
    kind = case["kind"]
    if kind == "matrix":
        n, _ = _counts(case)
        return {"edges": (n * (n - 1) // 2 // (4 if case["shape"] == "torus" else 64) + 4096, 2, np.uint32)}
    if kind == "parts":
        return {"edges": (1 << 20, 2, np.uint32)}
    if kind == "clip":
        return {"pos_tris": (1 << 16, 3, np.int32), "neg_tris": (1 << 16, 3, np.int32), "pos_map": (1 << 14, 1, np.int32),
                "neg_map": (1 << 14, 1, np.int32), "border": (1 << 12, 3, np.float64),
                "border_edges": (1 << 12, 2, np.int32)}
    if kind == "remesh":
        return {"vertices": (1 << 16, 3, np.float64), "triangles": (1 << 17, 3, np.int32)}
    if kind == "hulls":
        return {"triangles": (4096 * case["pairs"], 3, np.int32)}
    if kind == "process":
        return {"vertices": (1 << 16, 3, np.float64), "triangles": (1 << 17, 3, np.int32),
                "counts": (256, 2, np.int64)}
    return {}


def _put(s, name: str, a):
    """`a` at the front of the program's array `name`."""
    room = s["room"][name]
    a = np.asarray(a).reshape(-1, room.shape[1])
    room[:len(a)] = a
    return room


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    rng = np.random.default_rng([seed, 2])
    s = {"kind": kind, "ctx": ctx, "room": {k: np.zeros((r, c), t) for k, (r, c, t) in _room(case).items()}}
    if kind == "matrix":
        v, t = _mesh(case, seed)
        v = _normal(v)
        cv, ct = meshgen.offset_cage(v, t, case["offset"])
        s["mesh"] = (v.astype(np.float32), t.astype(np.uint32), cv.astype(np.float32), ct.astype(np.uint32))
    elif kind == "parts":
        v, t = _body(case, seed)
        s["parts"] = []
        for h in _pieces(v, t, 2, rng):
            cv, ct = ctx.sdf_remesh(h["vertices"], h["triangles"], 40.0, 0.02)
            s["parts"].append((h["vertices"].astype(np.float32), h["triangles"].astype(np.uint32),
                               cv.astype(np.float32), ct.astype(np.uint32), h.get("is_new")))
    elif kind in ("split", "learned"):
        v, t = _mesh(case, seed)
        s["v"] = np.ascontiguousarray(_normal(v))
        s["edges"] = _edges_of(s["v"], t)
        s["planes"] = case["planes"]
        s["draws"] = rng.integers(0, max(len(s["edges"]), 1), size=5 * case["planes"]).astype(np.int32)
        if kind == "learned":
            s["lp"] = _proposer()
            s["center"], s["half"] = proposer.part_frame(s["v"])
    elif kind == "score":
        E, P = case["edges"], case["planes"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["points"] = torch.rand(2 * E, 3, device="cuda", generator=g) * 2 - 1
        s["edges"] = torch.randperm(2 * E, device="cuda", generator=g).to(torch.int32).reshape(E, 2)
        n = torch.randn(P, 3, device="cuda", generator=g)
        d = torch.rand(P, 1, device="cuda", generator=g) * 1.6 - 0.8
        s["planes"] = torch.cat([n / n.norm(dim=1, keepdim=True), d], dim=1).contiguous()
        s["scores"] = torch.empty(P, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    elif kind == "clip":
        s["v"], s["t"] = _body(case, seed)
        s["plane"] = _plane_through(s["v"], rng)
    elif kind == "remesh":
        v, s["t"] = _mesh(case, seed)
        s["v"] = np.ascontiguousarray(_normal(v, case["stretch"]))
        s["scale"], s["level"] = case["scale"], case["level"]
    elif kind == "concavity":
        v, t = _body(case, seed)
        V.set_seed(seed % (1 << 31))
        s["jobs"] = []
        for p in _pieces(v, t, case["parts"], rng):
            h = V._convex_hull(p["vertices"])
            xa, ia = V._sample_points(p["vertices"], p["triangles"], case["samples"])
            xb, ib = V._sample_points(h["vertices"], h["triangles"], case["samples"])
            s["jobs"].append((p["vertices"], p["triangles"], xa, ia, h["vertices"], h["triangles"], xb, ib))
    elif kind == "hulls":
        v, t = _mesh(case, seed)
        sets = [p["vertices"] for p in _pieces(_normal(v), t, case["parts"], rng)]
        c = np.array([p.mean(axis=0) for p in sets])
        pairs = [(float(((c[a] - c[b]) ** 2).sum()), a, b) for a in range(len(sets)) for b in range(a)]
        s["sets"] = [np.concatenate([sets[a], sets[b]]) for _, a, b in sorted(pairs)[:case["pairs"]]]
    elif kind == "train":
        B, L = case["batch"], case["labels"]
        mid = rng.uniform(-1, 1, size=(B, _native.LP_POINTS, 3)) * rng.uniform(0.4, 1.0, size=(B, 1, 3))
        u = rng.normal(size=(B, _native.LP_POINTS, 3))
        u /= np.linalg.norm(u, axis=2, keepdims=True)
        big = np.take_along_axis(u, np.abs(u).argmax(axis=2)[..., None], axis=2)
        u = np.where(big < 0, -u, u)
        ln = rng.uniform(0.05, 1.5, size=(B, _native.LP_POINTS, 1))
        s["feats"] = np.concatenate([mid, u, ln], axis=2).astype(np.float32)
        n = rng.normal(size=(B, L, 3))
        n /= np.linalg.norm(n, axis=2, keepdims=True)
        s["labels"] = np.concatenate([n, rng.uniform(-0.5, 0.5, size=(B, L, 1))], axis=2).astype(np.float32)
        w = np.sort(rng.uniform(0.8, 1.0, size=(B, L)), axis=1)[:, ::-1]
        s["weights"] = np.ascontiguousarray(w / w[:, :1]).astype(np.float32)
        s["lp"] = _proposer()
    elif kind == "process":
        v, t = _mesh(case, seed)
        v = v * np.array([1.0, case["stretch"], case["stretch"]])
        m = V.Mesh()
        m.vertices = V.VecArray3d(v.tolist())
        m.triangles = V.make_vecarray3i(t.astype(np.int32))
        s.update(mesh=m, seed=seed % (1 << 31), concavity=case["concavity"], parts=case["parts"],
                 search=case["search"])
        V.config.verbose = False
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


# ---- one pass ----------------------------------------------------------------


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "matrix":
        v, t, cv, ct = s["mesh"]
        edges, stats = ctx.compute_intersection_matrix(v, t, cv, ct, capacity=len(s["room"]["edges"]))
        return {"edges": _put(s, "edges", edges), "count": len(edges), "pairs": stats["pairs_tested"], "leaving": stats["cage_hits"]}
    if kind == "parts":
        bvhs = [(ctx.bvh(v, t), ctx.bvh(cv, ct)) for v, t, cv, ct, _ in s["parts"]]
        edges, stats = ctx.visibility_batch([(p[0], a, b, p[4]) for p, (a, b) in zip(s["parts"], bvhs)])
        for a, b in bvhs:
            a.close()
            b.close()
        return {"edges": _put(s, "edges", np.concatenate(edges)), "counts": np.array([len(e) for e in edges]),
                "pairs": stats["pairs_tested"], "leaving": stats["cage_hits"]}
    if kind == "split":
        best, info = ctx.split_search(s["v"], s["edges"], s["draws"], s["planes"])
        return {"plane": best, "info": info}
    if kind == "learned":
        best, info = s["lp"].split_search(s["v"], s["edges"], s["center"], s["half"], s["half"], 32, s["draws"],
                                          s["planes"])
        return {"plane": best, "info": info}
    if kind == "score":
        ctx.score_planes_device(s["planes"].data_ptr(), len(s["planes"]), s["points"].data_ptr(), len(s["points"]),
                                s["edges"].data_ptr(), len(s["edges"]), s["scores"].data_ptr())
        return s["scores"]
    if kind == "clip":
        out = ctx.clip(s["v"], s["t"], s["plane"])
        return {k: _put(s, k, x) if isinstance(x, np.ndarray) else x for k, x in out.items()}
    if kind == "remesh":
        v, t = ctx.sdf_remesh(s["v"], s["t"], s["scale"], s["level"])
        return {"vertices": _put(s, "vertices", v), "triangles": _put(s, "triangles", t), "counts": [len(v), len(t)]}
    if kind == "concavity":
        return ctx.face_hausdorff_batch(s["jobs"], independent=True)
    if kind == "hulls":
        tris = ctx.convex_hulls(s["sets"])
        return {"triangles": _put(s, "triangles", np.concatenate(tris)), "counts": np.array([len(t) for t in tris])}
    if kind == "train":
        loss, grads = s["lp"].grads(s["feats"], s["labels"], s["weights"])
        return {"loss": loss, "grads": grads}
    V.config.plane_proposer = s["search"]
    V.set_seed(s["seed"])
    r = V.process(s["mesh"], s["concavity"], s["parts"])
    return {"vertices": _put(s, "vertices", np.concatenate([m.vertex_array() for m in r.parts])),
            "triangles": _put(s, "triangles", np.concatenate([m.triangle_array() for m in r.parts])),
            "counts": _put(s, "counts", [[len(m.vertices), len(m.triangles)] for m in r.parts]),
            "concavity": r.concavity}


# ---- what a pass cannot do without -------------------------------------------

_PAIR_FLOPS = 30  # one bound on one segment: its direction, a point, a distance


def _counts(case):
    """Vertices and triangles of the case's raw mesh."""
    f = case["f"]
    return (2 * f * f, 4 * f * f) if case["shape"] == "torus" else (10 * f * f + 2, 20 * f * f)


def _remeshed(case, scale: float):
    """About the vertices of the case's remesh at a grid of `scale` cells per
    unit: 1.5 vertices per cell-sized square of a body of radius 0.9."""
    k = case.get("stretch", 1.0)
    return 1.5 * 4.0 * math.pi * 0.81 * (0.3 + 0.7 * k) * k * scale * scale


def work(case):
    kind = case["kind"]
    if kind == "matrix":
        n, t = _counts(case)
        pairs = n * (n - 1) // 2
        return {"bytes": 2 * (12 * n + 12 * t) + 8 * 0.002 * pairs, "flops": _PAIR_FLOPS * pairs}
    if kind == "parts":
        n = _remeshed(case, 20.0 if _remeshed(case, 30.0) > 15000 else 30.0)
        c = 1.3 * _remeshed(case, 40.0)  # both cages
        new = 2.0 * math.sqrt(n)  # cut vertices of a half
        return {"bytes": 36 * n + 36 * c, "flops": _PAIR_FLOPS * 2 * new * (0.5 * n + new)}
    if kind in ("split", "learned"):
        n, _ = _counts(case)
        edges = 0.001 * n * n / 2
        planes = case["planes"] + (16 + 300 if kind == "learned" else 0)
        net = 2.0 * _native.LP_POINTS * (16 * 64 + 64 * 128 + 128 * 256) if kind == "learned" else 0.0
        return {"bytes": 24 * n + 8 * edges + 20 * case["planes"], "flops": 12.0 * planes * edges + net}
    if kind == "score":
        return {"bytes": 32 * case["edges"] + 24 * case["planes"], "flops": 12.0 * case["planes"] * case["edges"]}
    if kind == "clip":
        n = _remeshed(case, 20.0 if _remeshed(case, 30.0) > 15000 else 30.0)
        return {"bytes": (24 + 2 * 12 + 2 * 12 + 8) * n, "flops": 6 * n}
    if kind == "remesh":
        n, t = _counts(case)
        m = _remeshed(case, case["scale"])
        return {"bytes": 24 * n + 12 * t + 48 * m, "flops": 60.0 * 4 * m}
    if kind == "concavity":
        n = _remeshed(case, 20.0 if _remeshed(case, 30.0) > 15000 else 30.0)
        x = 12000 * case["samples"] / 3000 * case["parts"]
        return {"bytes": 2 * 48 * n + 28 * x, "flops": x * (10 * 8 + 10 * 60)}
    if kind == "hulls":
        n = 2.0 * case["pairs"] * (_counts(case)[0] / case["parts"] + 60)
        return {"bytes": 24 * n + 24 * n, "flops": 8.0 * n * math.log2(max(n / case["pairs"], 2.0))}
    if kind == "train":
        rows = case["batch"] * _native.LP_POINTS
        per_edge = 16 * 64 + 64 * 128 + 128 * 256
        return {"bytes": 28 * rows + 8 * 87744, "flops": 3 * 2.0 * rows * per_edge}
    n, t = _counts(case)
    m = _remeshed(case, 20.0 if _remeshed(case, 30.0) > 15000 else 30.0)
    return {"bytes": 24 * n + 12 * t + 72 * m, "flops": _PAIR_FLOPS * m * m / 2 * math.log2(2 + case["parts"])}


# ---- the same in 64 bits -------------------------------------------------------


def _least(a, b):
    """The metric's minimum: a NaN second value never wins, a NaN first stays."""
    return torch.where(b < a, b, a)


def _tri_dist(p, a, b, c):
    """The metric's point-triangle distance, row by row: the plane distance
    where the projection falls in the triangle, else the least of the edge
    distances (by Pythagoras, none where the foot is off the edge) and the
    vertex distances. Triangles without area give what that formula gives."""
    e1, e2 = b - a, c - a
    n = torch.linalg.cross(e1, e2)
    n = n / n.norm(dim=1, keepdim=True)
    ev = (n * p).sum(1) - (n * a).sum(1)
    w = p - n * ev[:, None] - a
    d00, d01, d11 = (e2 * e2).sum(1), (e2 * e1).sum(1), (e1 * e1).sum(1)
    d02, d12 = (e2 * w).sum(1), (e1 * w).sum(1)
    inv = 1.0 / (d00 * d11 - d01 * d01)
    u, v = (d11 * d02 - d01 * d12) * inv, (d00 * d12 - d01 * d02) * inv
    side = []
    for s0, s1 in ((a, b), (b, c), (c, a)):
        edge, to = s0 - s1, p - s1
        ln = edge.norm(dim=1)
        q = (to * edge).sum(1) / ln
        h = (to.norm(dim=1) ** 2 - q ** 2).sqrt()
        side.append(torch.where((q < 0) | (q > ln), torch.full_like(h, float("inf")), h))
    corner = [(p - x).norm(dim=1) for x in (a, b, c)]
    best = _least(_least(_least(side[0], side[1]), side[2]), _least(_least(corner[0], corner[1]), corner[2]))
    return torch.where((u >= 0) & (v >= 0) & (u + v <= 1), ev.abs(), best)


def _half_hausdorff(x, y, ids, v, t) -> float:
    """The largest, over the samples x, of the least distance to the triangles
    that the 10 nearest of the samples y were drawn from."""
    a, b, c = (v[t[:, k]] for k in range(3))
    top = 0.0
    for q in x.split(512):
        d2 = sum((q[:, None, k] - y[None, :, k]) ** 2 for k in range(3))
        near = d2.topk(min(10, len(y)), dim=1, largest=False)
        tri = ids[near.indices]
        k = tri.shape[1]
        d = _tri_dist(q.repeat_interleave(k, 0), a[tri].reshape(-1, 3), b[tri].reshape(-1, 3), c[tri].reshape(-1, 3))
        d = torch.nan_to_num(d, nan=float("inf")).reshape(-1, k).amin(1)
        d = torch.where(d > 10.0, near.values[:, 0].sqrt(), d)
        top = max(top, float(d.max()))
    return top


def _exact_scores(planes, points, edges):
    """Edge length cut by each plane (endpoints strictly on opposite sides),
    FP32 inputs, everything else in 64 bits."""
    pl, pt, ed = planes.double(), points.double(), edges.long()
    p, q = pt[ed[:, 0]], pt[ed[:, 1]]
    length = (q - p).norm(dim=1)
    eps = float(np.float32(1e-6))
    out = torch.empty(len(pl), dtype=torch.float64, device=pl.device)
    step = max(1, (1 << 26) // max(len(ed), 1))
    for k in range(0, len(pl), step):
        n, d = pl[k:k + step, :3], pl[k:k + step, 3]
        a, b = n @ p.T + d[:, None], n @ q.T + d[:, None]
        cut = ((a > eps) & (b < -eps)) | ((a < -eps) & (b > eps))
        out[k:k + step] = cut.double() @ length
    return out


def _candidates(v, edges, draws, count: int) -> np.ndarray:
    """The bisector planes of the drawn edges, near-duplicates dropped."""
    p, q = v[edges[draws, 0].astype(np.int64)], v[edges[draws, 1].astype(np.int64)]
    n = q - p
    ln = np.linalg.norm(n, axis=1)
    n = n / np.where(ln > 0, ln, 1)[:, None]
    d = -(n * (0.5 * (p + q))).sum(axis=1)
    keep = np.zeros((count, 4))
    got, cos5 = 0, math.cos(5.0 * math.pi / 180.0)
    for k in range(len(draws)):
        if got == count:
            break
        if ln[k] < 1e-6:
            continue
        near = np.nonzero(np.abs(keep[:got, 3] - d[k]) < 1e-3)[0]
        if len(near) and (np.abs(keep[near, :3] @ n[k]) > cos5).any():
            continue
        keep[got] = [*n[k], d[k]]
        got += 1
    return keep[:got]


def _bf16(x):
    """x rounded to BF16, with x's own derivative."""
    return x + (x.bfloat16().double() - x).detach()


def _exact_grads(feats, labels, weights):
    """Loss and parameter gradients of the proposer's network in 64 bits. The
    operands of its layers (input, weights, activations) are BF16 by
    definition, so they are rounded to BF16; everything else is 64 bits."""
    K, N = [16, 64, 128, 256, 128, 64], [64, 128, 256, 128, 64, 64]
    p = torch.from_numpy(proposer.load_params()).cuda().double().requires_grad_(True)
    at, layers = 0, []
    for k, n in zip(K, N):
        layers.append((_bf16(p[at:at + k * n]).reshape(n, k), p[at + k * n:at + k * n + n]))
        at += k * n + n
    f = _bf16(torch.from_numpy(feats).cuda().double())
    B, S, F = f.shape
    lab = torch.from_numpy(labels.astype(np.float64)).cuda()
    w = torch.from_numpy(weights.astype(np.float64)).cuda()
    rank = torch.arange(S, device="cuda")[None, :, None]
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for b0 in range(0, B, 8):
        x = torch.nn.functional.pad(f[b0:b0 + 8], (0, 16 - F))
        for W, c in layers[:3]:
            x = _bf16(torch.relu(x @ W.T + c))
        top = x.detach().amax(dim=1, keepdim=True)
        first = torch.where(x.detach() == top, rank, S).amin(dim=1, keepdim=True)  # the first maximum
        x = x.gather(1, first)[:, 0]
        for W, c in layers[3:5]:
            x = _bf16(torch.relu(x @ W.T + c))
        z = (x @ layers[5][0].T + layers[5][1]).reshape(len(x), -1, 4)
        n, d = z[..., :3] / (z[..., :3].norm(dim=2, keepdim=True) + 1e-12), z[..., 3]
        l, lw = lab[b0:b0 + 8], w[b0:b0 + 8]
        c = n @ l[..., :3].transpose(1, 2)
        D = torch.minimum(2 - 2 * c + (d[:, :, None] - l[:, None, :, 3]) ** 2,
                          2 + 2 * c + (d[:, :, None] + l[:, None, :, 3]) ** 2)
        part = (lw * D.amin(dim=1)).sum(1) / lw.sum(1) + 0.1 / 16 * D.amin(dim=2).sum(1)
        loss = part.sum() / B
        loss.backward(retain_graph=b0 + 8 < B)
        total = total + loss.detach()
    return float(total), p.grad.cpu().numpy()


def exact(case, seed):
    """Edges, masks and triangles are decisions, not computed numbers; a
    remeshed or clipped mesh is defined step by step together with its
    connectivity, and a whole decomposition takes many minutes in 64 bits."""
    kind = case["kind"]
    if kind in ("matrix", "parts", "clip", "remesh", "hulls", "learned", "process"):
        return None
    s = prepare(case, seed)
    if kind == "score":
        return _exact_scores(s["planes"], s["points"], s["edges"])
    if kind == "split":
        if len(s["edges"]) == 0:
            return None
        cand = _candidates(s["v"], s["edges"], s["draws"], s["planes"])
        sc = _exact_scores(torch.from_numpy(cand.astype(np.float32)).cuda(),
                           torch.from_numpy(s["v"].astype(np.float32)).cuda(),
                           torch.from_numpy(s["edges"].astype(np.int64)).cuda()).cpu().numpy()
        k = int(sc.argmax())
        return {"plane": cand[k], "info": {"best_index": None, "n_candidates": None, "draws_used": None,
                                           "best_score": float(sc[k])}}
    if kind == "concavity":
        out = []
        g = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        for va, ta, xa, ia, vb, tb, xb, ib in s["jobs"]:
            va, xa, vb, xb = (g(np.asarray(a, dtype=np.float64)) for a in (va, xa, vb, xb))
            ta, ia, tb, ib = (g(np.asarray(a, dtype=np.int64)) for a in (ta, ia, tb, ib))
            out.append(max(_half_hausdorff(xa, xb, ib, vb, tb), _half_hausdorff(xb, xa, ia, va, ta)))
        return np.array(out)
    loss, grads = _exact_grads(s["feats"], s["labels"], s["weights"])
    return {"loss": loss, "grads": grads}
