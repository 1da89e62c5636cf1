"""Workloads of the symmetry detector, each through the entry point a program calls.

A case is a dict with an "op" and its sizes:

  detect     Gb300Backend.detect_fast on a resident mesh (curvature, prune, pairing, votes, vote
             sort, mean shift, modes, verification); with "raw", the mesh is also loaded from host
             memory (GPU prepare) and given back in every pass, and the sample drawn on the device
  fused      Gb300Backend.detect_fast_fused on a batch of uneven meshes, one mean shift for all
  modes      Gb300Backend.meanshift6 on 6-D votes from host memory
  verify     Gb300Backend.verification_resident on a resident mesh
  curvature, votes, cluster, verification
             the exact FP64 stages, from and to host memory as the reference's Backend has them

Meshes are this package's seeded generators: "sphere" (motif icosphere, size = subdivision
level), "torus" (motif torus, size x size/2 grid), "field" (mirrored height field, size x size).
"""
import math

import numpy as np
import torch

from mitra_algo_gb300 import Gb300Backend, Options, Rng
from mitra_algo_gb300.mesh import add_noise, mirrored_heightfield, motif_sphere, motif_torus
from mitra_algo_gb300.mesh import prepare as prepare_mesh
from mitra_algo_gb300.mesh import uneven_batch
from mitra_algo_gb300.types import ClusterOutput, Csr, Pairs

_shared = []


def _backend():
    """One backend for the whole program: its context keeps the workspace from call to call."""
    if not _shared:
        _shared.append(Gb300Backend(0))
    return _shared[0]


def _detect(name, mesh, size, samples, seeds, **more):
    case = {"name": name, "op": "detect", "mesh": mesh, "size": size, "samples": samples,
            "seeds": seeds, "precision": "bf16", "kernel": "epanechnikov", "mode": "rigid",
            "threshold": 0.25, "bandwidth": 0.1, "iterations": 300, "clusters": 20, "refine": 0,
            "vote_cap": 0, "raw": False}
    case.update(more)
    return case


def listed():
    return [
        # the smallest whole call: a scanned part of a few thousand vertices, straight from host
        # memory; launches and round trips count
        _detect("detect_small_raw", "sphere", 4, 2000, 128, raw=True, iterations=60, clusters=4),
        # a mirror plane of a height field of the size the reference runs on a CPU, with FP64
        # refinement of the planes; few votes, so the FP32 form is the one to take
        _detect("detect_mirror_fp32", "field", 128, 2000, 512, precision="fp32", mode="reflection",
                threshold=0.05, bandwidth=0.02, iterations=100, clusters=8, refine=5),
        # a mid-sized part with the smooth kernel and no tensor cores, ragged vertex count
        _detect("detect_gauss_fp32", "torus", 171, 5000, 256, precision="fp32", kernel="gaussian",
                clusters=8),
        # the headline detection: all votes of 20,000 samples, 2,048 seeds
        _detect("detect_motif", "sphere", 6, 20000, 2048),
        # the large single scan: a million triangles, votes subsampled for the mean shift
        _detect("detect_torus_large", "torus", 1000, 200000, 4096, threshold=0.05,
                vote_cap=1000000),
        # a shelf of small parts handed over as one batch
        {"name": "fused_batch", "op": "fused", "count": 12, "samples": 2000, "seeds": 256,
         "precision": "bf16"},
        # mode seeking alone, as a program with votes of its own calls it
        {"name": "modes_planted", "op": "modes", "votes": 200003, "modes": 48, "seeds": 512,
         "precision": "bf16", "kernel": "epanechnikov"},
        # checking given motions of a scan that stays on the device
        {"name": "verify_resident", "op": "verify", "mesh": "torus", "size": 400, "clusters": 20},
        # the reference's stages one by one, FP64 and in its order of operations
        {"name": "stage_curvature", "op": "curvature", "mesh": "torus", "size": 333,
         "smoothing": 3},
        {"name": "stage_votes", "op": "votes", "mesh": "field", "size": 96, "samples": 3000,
         "mirrored": 3000, "others": 12001},
        {"name": "stage_cluster", "op": "cluster", "mesh": "field", "size": 128, "samples": 2000,
         "mirrored": 1500, "others": 2200},
        {"name": "stage_verification", "op": "verification", "mesh": "field", "size": 128,
         "clusters": 8},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["detect", "detect", "detect", "detect", "fused", "modes", "verify",
                     "curvature", "votes", "cluster", "verification"])
    if op == "fused":
        return {"op": op, "count": rng.randint(2, 11), "samples": _spread(rng, 500, 2500),
                "seeds": _spread(rng, 64, 300), "precision": rng.choice(["bf16", "bf16", "fp32"])}
    if op == "modes":
        return {"op": op, "votes": _spread(rng, 5000, 400000), "modes": rng.randint(3, 60),
                "seeds": _spread(rng, 31, 1500), "precision": rng.choice(["bf16", "fp32"]),
                "kernel": rng.choice(["epanechnikov", "gaussian"])}
    mesh = rng.choice(["torus", "field", "sphere"] if op == "detect" else ["torus", "field"])
    size = {"torus": _spread(rng, 60, 600), "field": _spread(rng, 40, 220),
            "sphere": rng.randint(4, 6)}[mesh]
    if op == "verify":
        return {"op": op, "mesh": mesh, "size": size, "clusters": rng.randint(1, 20)}
    if op == "curvature":
        return {"op": op, "mesh": mesh, "size": size, "smoothing": rng.randint(0, 5)}
    if op == "votes":
        return {"op": op, "mesh": "field", "size": _spread(rng, 40, 140),
                "samples": _spread(rng, 500, 4000), "mirrored": _spread(rng, 50, 9000),
                "others": _spread(rng, 50, 40000)}
    if op == "cluster":
        return {"op": op, "mesh": "field", "size": _spread(rng, 40, 140),
                "samples": _spread(rng, 300, 2200), "mirrored": _spread(rng, 50, 2000),
                "others": _spread(rng, 50, 3000)}
    if op == "verification":
        return {"op": op, "mesh": "field", "size": _spread(rng, 40, 160),
                "clusters": rng.randint(1, 10)}
    mode = "reflection" if mesh == "field" else "rigid"
    # the thresholds go with the meshes: a torus has many vertices of nearly one curvature
    threshold = 0.25 if mesh == "sphere" else 0.05
    case = _detect("", mesh, size, _spread(rng, 800, 12000), _spread(rng, 64, 2000),
                   precision=rng.choice(["bf16", "bf16", "fp32"]),
                   kernel=rng.choice(["epanechnikov", "epanechnikov", "gaussian"]), mode=mode,
                   threshold=threshold, bandwidth=0.02 if mode == "reflection" else 0.1,
                   iterations=rng.choice([60, 100, 300]), clusters=rng.randint(2, 20),
                   refine=rng.choice([0, 0, 3]), vote_cap=rng.choice([0, 0, 500000]),
                   raw=rng.random() < 0.4)
    del case["name"]
    return case


# ------------------------------------------------------------------ inputs
def _mesh(kind, size, seed):
    if kind == "sphere":
        return motif_sphere(level=size, bumps=12, folds=5, partial_shift=0.4, noise=1e-3, seed=seed)
    if kind == "torus":
        return motif_torus(nu=size, nv=max(12, size // 2), copies=12, mirrored=2, bumps=2,
                           noise=5e-4, seed=seed)
    # scanner noise a tenth of the generators' usual: the mirror plane stays exact to 1e-4
    return add_noise(mirrored_heightfield(size=size, bumps=8, seed=seed), 1e-4, seed + 1)


def _counts(case):
    """(vertices, faces) of the case's mesh, a sphere's without its partial copy."""
    n = case["size"]
    if case["mesh"] == "sphere":
        return 10 * 4 ** n + 2, 20 * 4 ** n
    if case["mesh"] == "torus":
        nv = n * max(12, n // 2)
        return nv, 2 * nv
    return n * n, 2 * (n - 1) ** 2


def _motions(case, context, rng):
    """Motions such as a clustering hands to the verification: near the
    planted symmetries, with the scatter of modes, and some wrong ones."""
    n = case["clusters"]
    c = np.asarray(context.center)
    refl, rot, tr = np.zeros(n, np.uint8), np.zeros((n, 9)), np.zeros((n, 3))
    normal, offset = np.zeros((n, 3)), np.zeros(n)
    for i in range(n):
        if case["mesh"] == "field":
            spread = 1e-4 if i < (n + 1) // 2 else 0.05
            m = np.array([1.0, 0, 0]) + rng.normal(0, spread, 3)
            m /= np.linalg.norm(m)
            d = rng.normal(0, spread)
            r, t = np.eye(3) - 2 * np.outer(m, m), -2 * d * m
            refl[i], normal[i], offset[i] = 1, m, d
        else:
            folds = 5 if case["mesh"] == "sphere" else 12
            a = 2 * np.pi * rng.integers(1, folds) / folds + rng.normal(0, 1e-3)
            if i >= (n + 1) // 2:
                a = rng.uniform(0, 2 * np.pi)
            r = np.array([[np.cos(a), -np.sin(a), 0], [np.sin(a), np.cos(a), 0], [0, 0, 1.0]])
            t = c - r @ c if case["mesh"] == "sphere" else np.zeros(3)
            t = t + rng.normal(0, 1e-3, 3)
        rot[i], tr[i] = r.ravel(), t
    empty = Csr(np.zeros(n + 1, np.uint64), np.zeros(0, np.int32))
    return ClusterOutput(refl, rot, tr, normal, offset, empty)


def _planted_votes(case, seed):
    """Half of the votes in tight clusters (width a seventh of the bandwidth),
    half spread over the vote space; values are FP32 as vote records are."""
    rng = np.random.default_rng(seed)
    q, m, h = case["votes"], case["modes"], 0.06
    centres = np.concatenate([rng.uniform(-1.5, 1.5, (m, 3)), rng.uniform(-0.6, 0.6, (m, 3))], 1)
    which = rng.integers(0, m, q // 2)
    near = centres[which] + rng.normal(0, h / 7 / math.sqrt(6) * 1.6, (q // 2, 6))
    far = np.concatenate([rng.uniform(-1.57, 1.57, (q - q // 2, 3)),
                          rng.uniform(-1, 1, (q - q // 2, 3))], 1)
    votes = np.concatenate([near, far]).astype(np.float32).astype(np.float64)
    seeds = np.sort(rng.choice(q // 2, min(case["seeds"], q // 2), replace=False))
    return votes, seeds, h


def _features(gpu, case, seed):
    """Host inputs of the stages after the selection."""
    o = Options(sample_ratio=min(1.0, case["samples"] / _counts(case)[0]), pair_threshold=0.05,
                bandwidth=0.02, max_pairs=10 ** 7, max_votes=2 * 10 ** 7)
    p = prepare_mesh(_mesh(case["mesh"], case["size"], seed), o)
    f = gpu.curvature(p.mesh, p.topology, o)
    rng = Rng(o.seed)
    s = gpu.select(p.mesh, f, p.topology.weights, o, rng)
    pairs = gpu.pairing(p.mesh, f, s.pruned, p.context, o)
    # a given number of pairs whose mirrored frames agree (three votes each)
    # and of others (two), in pair order: the number of votes is the case's
    kinds = gpu.transformations(p.mesh, f, pairs, p.context, o)
    agree = np.zeros(len(pairs), bool)
    agree[kinds.pair[kinds.kind == 1]] = True
    keep = np.sort(np.concatenate([np.resize(np.flatnonzero(agree), case["mirrored"]),
                                   np.resize(np.flatnonzero(~agree), case["others"])]))
    return o, p, f, Pairs(pairs.a[keep], pairs.b[keep]), rng


def prepare(case, seed):
    gpu = _backend()
    s = {"gpu": gpu, "case": case}
    op = case["op"]
    if op == "detect":
        mesh = _mesh(case["mesh"], case["size"], seed)
        s["options"] = Options(sample_ratio=min(1.0, case["samples"] / mesh.vertex_count),
                               pair_threshold=case["threshold"], bandwidth=case["bandwidth"],
                               max_pairs=10 ** 9, max_votes=2 * 10 ** 9 - 1,
                               max_clusters=case["clusters"])
        s["keywords"] = {k: case[k] for k in ("precision", "kernel", "mode", "seeds", "refine",
                                              "vote_cap")}
        s["keywords"].update(max_iterations=case["iterations"], polish_iterations=30)
        if case["raw"]:
            s["mesh"] = mesh
        else:
            s["resident"] = gpu.load_mesh_raw(mesh, s["options"])
    elif op == "fused":
        s["jobs"], s["modes"] = [], []
        for mesh, mode, _ in uneven_batch(case["count"], seed):
            o = Options(sample_ratio=min(1.0, case["samples"] / mesh.vertex_count),
                        pair_threshold=0.25 if mode == "rigid" else 0.05, bandwidth=0.1,
                        max_pairs=10 ** 8, max_votes=2 * 10 ** 9 - 1, max_clusters=8)
            s["jobs"].append((gpu.load_mesh_raw(mesh, o), None, o))
            s["modes"].append(mode)
    elif op == "modes":
        s["votes"], s["seeds"], s["bandwidth"] = _planted_votes(case, seed)
    elif op == "verify":
        o = s["options"] = Options()
        p = prepare_mesh(_mesh(case["mesh"], case["size"], seed), o)
        s["resident"] = gpu.load_mesh(p)
        s["clusters"] = _motions(case, p.context, np.random.default_rng(seed + 2))
    elif op == "curvature":
        s["options"] = Options(smoothing=case["smoothing"])
        s["prepared"] = prepare_mesh(_mesh(case["mesh"], case["size"], seed), s["options"])
    elif op == "verification":
        s["options"] = Options()
        p = s["prepared"] = prepare_mesh(_mesh(case["mesh"], case["size"], seed), s["options"])
        s["clusters"] = _motions(case, p.context, np.random.default_rng(seed + 2))
    else:
        s["options"], s["prepared"], s["features"], s["pairs"], s["rng"] = _features(gpu, case, seed)
        if op == "cluster":
            s["votes"] = gpu.transformations(s["prepared"].mesh, s["features"], s["pairs"],
                                             s["prepared"].context, s["options"])
    return s


# ------------------------------------------------------------------- passes
_INTEGERS = ("sampled", "pruned", "pairs", "votes", "modes", "clusters")
_ARRAYS = (("support", np.int64, 1), ("patches", np.int64, 2), ("precise", np.uint8, 1),
           ("reflection", np.uint8, 1), ("rotation", np.float64, 9),
           ("translation", np.float64, 3), ("plane_normal", np.float64, 3),
           ("plane_offset", np.float64, 1), ("coverage", np.float64, 1), ("rms", np.float64, 1))


def _padded(a, size, dtype, empty=0):
    """`a` at the start of an array of `size`: what is found differs in number
    from input to input, the array does not."""
    out = np.full(size, empty, dtype)
    a = np.asarray(a, dtype).reshape(-1)
    out[:a.size] = a
    return out


def _result(r, most):
    """What a detection found, at most `most` motions; its timers and work
    counters are left out."""
    out = {"counts": np.array([r[k] for k in _INTEGERS], np.int64)}
    out.update({k: _padded(r[k], most * n, t) for k, t, n in _ARRAYS})
    return out


def _sides(v, clusters, vertices):
    n = clusters * vertices
    return {"side_a": _padded(v.side_a.indices, n, np.int32, -1),
            "side_b": _padded(v.side_b.indices, n, np.int32, -1),
            "patches_a": _padded(v.patches_a.indices, n, np.int32, -1),
            "patches_b": _padded(v.patches_b.indices, n, np.int32, -1),
            "patches_a_offsets": _padded(v.patches_a.offsets, n + 1, np.int64, -1),
            "patches_b_offsets": _padded(v.patches_b.offsets, n + 1, np.int64, -1),
            "side_a_offsets": v.side_a.offsets.astype(np.int64),
            "side_b_offsets": v.side_b.offsets.astype(np.int64),
            "patches_a_groups": v.patches_a_groups.astype(np.int64),
            "patches_b_groups": v.patches_b_groups.astype(np.int64),
            "coverage": v.coverage, "rms": v.rms}


def run(s):
    gpu, case = s["gpu"], s["case"]
    op = case["op"]
    if op == "detect":
        if not case["raw"]:
            return _result(gpu.detect_fast(s["resident"], None, s["options"], **s["keywords"]),
                           case["clusters"])
        resident = gpu.load_mesh_raw(s["mesh"], s["options"])
        r = gpu.detect_fast(resident, None, s["options"], **s["keywords"])
        resident.close()
        return _result(r, case["clusters"])
    if op == "fused":
        found, _ = gpu.detect_fast_fused(s["jobs"], precision=case["precision"],
                                         seeds=case["seeds"], max_iterations=300,
                                         polish_iterations=30, mode=s["modes"])
        every = [_result(r, 8) for r in found]
        return {k: np.concatenate([r[k] for r in every]) for k in every[0]}
    if op == "modes":
        means, state, _ = gpu.meanshift6(s["votes"], s["seeds"], s["bandwidth"], case["precision"],
                                         200, 30, case["kernel"])
        return {"means": means, "state": state}
    if op == "verify":
        found, _ = gpu.verification_resident(s["resident"], s["clusters"], s["options"])
        return _sides(found, case["clusters"], s["resident"].vertex_count)
    p, o = s["prepared"], s["options"]
    if op == "curvature":
        f = gpu.curvature(p.mesh, p.topology, o)
        return {"normal": f.normal, "dmin": f.dmin, "dmax": f.dmax, "kmin": f.kmin,
                "kmax": f.kmax, "valid": f.valid}
    if op == "verification":
        return _sides(gpu.verification(p.mesh, p.topology, s["clusters"], p.context, o),
                      case["clusters"], p.mesh.vertex_count)
    if op == "votes":
        v = gpu.transformations(p.mesh, s["features"], s["pairs"], p.context, o)
        return {"pair": v.pair, "kind": v.kind, "rotation": v.rotation,
                "translation": v.translation, "plane_normal": v.plane_normal,
                "plane_offset": v.plane_offset, "descriptor": v.descriptor}
    c = gpu.clustering(s["votes"], p.context, o, s["rng"].copy())
    n = o.max_clusters
    owner = np.full(len(s["votes"]), -1, np.int32)  # each vote's cluster
    owner[c.votes.indices] = np.repeat(np.arange(len(c), dtype=np.int32),
                                       np.diff(c.votes.offsets.astype(np.int64)))
    return {"reflection": _padded(c.reflection, n, np.uint8),
            "rotation": _padded(c.rotation, 9 * n, np.float64),
            "translation": _padded(c.translation, 3 * n, np.float64),
            "plane_normal": _padded(c.plane_normal, 3 * n, np.float64),
            "plane_offset": _padded(c.plane_offset, n, np.float64), "owner": owner}


# --------------------------------------------------------------------- work
def _detect_work(v, f, samples, seeds, threshold, mode, vote_cap, clusters):
    """Bytes: the mesh and its topology once, the pairs and vote records
    written and read once, the surface once per motion and direction.  Flops:
    each seed's trajectory over the votes in its window (about 1/3,000 of the
    vote space, 40 steps, 30 flops), closest points of each query (2 x 150)."""
    pairs = samples * samples / 2 * (0.05 if threshold > 0.1 else 0.0017)
    votes = pairs * (2 if mode == "rigid" else 0.3)
    kept = min(votes, vote_cap) if vote_cap else votes
    surface = 57 * v + 36 * f + 24 * 1.5 * f
    queries = 2 * v * clusters
    return {"bytes": surface + 8 * pairs + 64 * kept + 25 * queries,
            "flops": seeds * kept / 3000 * 40 * 30 + 300 * queries}


def work(case):
    op = case["op"]
    if op == "fused":  # log-uniform 2,000 to 60,000 vertices: 17,000 on average
        w = _detect_work(17000, 34000, case["samples"], case["seeds"], 0.15, "rigid", 0, 8)
        return {k: x * case["count"] for k, x in w.items()}
    if op == "modes":  # a cluster's members are the window of its seeds, some 6 steps
        return {"bytes": 48 * case["votes"] + 49 * case["seeds"],
                "flops": case["seeds"] * case["votes"] / 2 / case["modes"] * 6 * 30}
    v, f = _counts(case)
    if op == "detect":
        return _detect_work(v, f, min(case["samples"], v), case["seeds"], case["threshold"],
                            case["mode"], case["vote_cap"], case["clusters"])
    if op in ("verify", "verification"):  # the surface in, flags and members out
        return {"bytes": 48 * v + 36 * f + 25 * 2 * v * case["clusters"],
                "flops": 300 * 2 * v * case["clusters"]}
    if op == "curvature":  # positions, normals, rings and edges in, 11 lanes out
        return {"bytes": (48 + 8 + 24 + 89) * v + (24 + 36) * f,
                "flops": 80 * 3 * f + 63 * case["smoothing"] * v + 100 * v}
    pairs, q = case["mirrored"] + case["others"], 3 * case["mirrored"] + 2 * case["others"]
    if op == "votes":  # frames and pairs in, 28 FP64 lanes per vote out
        return {"bytes": 96 * v + 8 * pairs + 229 * q, "flops": 250 * pairs}
    # cluster: descriptors in, memberships out; every vote's trajectory over its window
    return {"bytes": 101 * q + 4 * q, "flops": q * q / 300 * 20 * 40}


# -------------------------------------------------------------------- exact
def _cross(a, b):
    return np.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _unit(a):
    n = np.sqrt((a * a).sum(0))
    return np.where(n > 1e-14, a / np.where(n > 1e-14, n, 1), 0)


def _exact_curvature(s):
    p, o = s["prepared"], s["options"]
    x, fn, vn = p.mesh.vertices, p.topology.face_normals, p.topology.normals
    edges = np.asarray(p.topology.edges).reshape(-1, 6)
    lo, hi, a, b, f0, f1 = edges.T.astype(np.int64)
    n = x.shape[1]
    mean = np.sqrt(((x[:, hi] - x[:, lo]) ** 2).sum(0)).mean()
    inner = f1 >= 0
    a, b, f0, f1 = a[inner], b[inner], f0[inner], f1[inner]
    d = x[:, b] - x[:, a]
    length = np.sqrt((d * d).sum(0))
    d = _unit(d)
    n0, n1 = fn[:, f0], fn[:, f1]
    beta = np.arctan2((_cross(n0, n1) * d).sum(0), np.clip((n0 * n1).sum(0), -1, 1))
    t = np.zeros((n, 9))
    each = (d[:, None] * d[None] * (beta * length / mean)).reshape(9, -1).T
    count = np.zeros(n)
    for ends in (a, b):
        np.add.at(t, ends, each)
        np.add.at(count, ends, 1)
    t /= np.maximum(count, 1)[:, None]
    off = p.topology.neighbors.offsets.astype(np.int64)
    ring, degree = p.topology.neighbors.indices.astype(np.int64), np.diff(off)
    row = np.repeat(np.arange(n), degree)
    for _ in range(o.smoothing):
        around = t.copy()
        np.add.at(around, row, t[ring])
        t = around / (degree + 1)[:, None]
    ok = ~((np.sqrt((vn * vn).sum(0)) < 0.5) | (degree < 3))
    axis = np.where(np.abs(vn[0]) < 0.8, np.array([[1.0], [0], [0]]), np.array([[0.0], [1], [0]]))
    u = _unit(_cross(vn, axis))
    w = _cross(vn, u)
    m = t.reshape(n, 3, 3)
    qa, qb, qc = (np.einsum("in,nij,jn->n", l, m, r) for l, r in ((u, u), (u, w), (w, w)))
    angle = 0.5 * np.arctan2(2 * qb, qa - qc)
    low = _unit(_cross(u * np.cos(angle) + w * np.sin(angle), vn))
    delta = np.hypot(qa - qc, 2 * qb)
    keep = lambda v: np.where(ok, v, 0.0)  # noqa: E731
    return {"normal": keep(vn), "dmin": keep(low), "dmax": keep(_unit(_cross(vn, low))),
            "kmin": keep((qa + qc - delta) / 2), "kmax": keep((qa + qc + delta) / 2), "valid": None}


def _exact_votes(s):
    p, f = s["prepared"], s["features"]
    x, c, box = p.mesh.vertices, np.asarray(p.context.center)[:, None], p.context.box_size
    a, b = s["pairs"].a, s["pairs"].b
    np_, P, Q = a.size, x[:, a], x[:, b]
    n = _unit(Q - P)
    dom = np.argmax(np.abs(n), 0)
    n = n * np.where(n[dom, np.arange(np_)] < 0, -1.0, 1.0)
    d = -(n * (P + Q)).sum(0) / 2
    refl = np.eye(3)[:, :, None] - 2 * n[:, None] * n[None]
    turn = lambda m, v: np.einsum("ijn,jn->in", m, v)  # noqa: E731
    mirrored = ((turn(refl, f.normal[:, a]) * f.normal[:, b]).sum(0) > 0.75) & \
        (np.abs((turn(refl, f.dmin[:, a]) * f.dmin[:, b]).sum(0)) > 0.75)
    first = np.concatenate([[0], np.cumsum(2 + mirrored)])
    q = int(first[-1])
    out = {"rotation": np.zeros((9, q)), "translation": np.zeros((3, q)),
           "plane_normal": np.zeros((3, q)), "plane_offset": np.zeros(q),
           "descriptor": np.zeros((12, q)), "pair": None, "kind": None}
    at = first[:-1][mirrored]
    out["rotation"][:, at] = refl.reshape(9, -1)[:, mirrored]
    out["translation"][:, at] = (-2 * d * n)[:, mirrored]
    out["plane_normal"][:, at] = n[:, mirrored]
    out["plane_offset"][at] = d[mirrored]
    out["descriptor"][:3, at] = n[:, mirrored]
    out["descriptor"][3, at] = ((d + (n * c).sum(0)) / box)[mirrored]
    for k, sign in enumerate((1.0, -1.0)):
        r = sum(w * v[:, None] * z[None] for w, v, z in
                ((sign, f.dmin[:, b], f.dmin[:, a]), (sign, f.dmax[:, b], f.dmax[:, a]),
                 (1.0, f.normal[:, b], f.normal[:, a])))
        t = Q - turn(r, P)
        at = first[:-1] + mirrored + k
        out["rotation"][:, at] = r.reshape(9, -1)
        out["translation"][:, at] = t
        out["descriptor"][:9, at] = r.reshape(9, -1) / 2
        out["descriptor"][9:, at] = (np.einsum("ijn,j->in", r, c[:, 0]) + t - c) / box
    return out


def _exact_modes(s):
    """Plain mean-shift steps in FP64 until nothing moves."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    votes, h2 = torch.from_numpy(s["votes"]).to(dev), s["bandwidth"] ** 2
    gauss = s["case"]["kernel"] == "gaussian"
    means = []
    for part in torch.from_numpy(s["votes"][s["seeds"]]).to(dev).split(64):
        m = part.clone()
        for _ in range(200):
            d2 = sum((m[:, k:k + 1] - votes[None, :, k]) ** 2 for k in range(6)) / h2
            w = torch.exp2(-8 * d2) - 2.0 ** -8 if gauss else 1 - d2
            w = torch.where(d2 < 1, w, 0.0)
            step = w @ votes / w.sum(1, keepdim=True) - m
            m = m + step
            if float(step.abs().max()) < 1e-13:
                break
        means.append(m)
    return {"means": torch.cat(means).cpu().numpy(), "state": None}


def exact(case, seed):
    """FP64 values where plain numpy gives them: curvature, vote transforms and
    well-separated modes.  A detection's floats follow from its choice of
    modes and supporting vertices (whole numbers), and the exact stages are
    FP64 sums in a prescribed order, so those have no other value here."""
    if case["op"] == "curvature":
        return _exact_curvature(prepare(case, seed))
    if case["op"] == "votes":
        return _exact_votes(prepare(case, seed))
    if case["op"] == "modes":
        return _exact_modes(prepare(case, seed))
    return None
