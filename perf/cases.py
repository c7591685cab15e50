"""Timing cases of the product path, through its public entry points.

Each case is one call, or one short sequence of calls, that a program using this library
makes with points it has just received: nothing that is computed from the points is kept
from one pass to the next (every pass starts from the points again), while the context,
the server and the caller's output buffers are kept, as such a program keeps them.

`op` names the call:

    chain         Context: host points -> LBVH, EMST, k = 1 forest, and the hierarchy of orders
                  1..K (node supports, child arena, batches, roots, vertical maps), copied into
                  buffers the caller owns
    fit           ehgp.fit on a CUDA tensor: the one-call front end, its own context each time
    lbvh          canonical cloud + exact Morton LBVH, reference-layout snapshot on the host
    lbvh_noalloc  the allocation-free LBVH entry point
    knn           exact k nearest neighbours of every point with the exact cutoffs
    emst          exact Boruvka EMST and the compact k = 1 forest
    pairs         relevant pair supports (records and exact levels)
    higher        relevant triple/quad supports (records)
    serve         a batch of clouds through the serving engine, all submitted at once

`shape` names the generator of workloads.py: `uniform` (binary64), `lattice` (jittered unit
lattice, binary32), `mixture` (Gaussian mixture with noise, binary32) and `clustered`
(anisotropic Gaussians + background with 5 % of the points on a 2^-10 grid: exact ties,
binary64; the hierarchy refuses such clouds, so only the stages before it take them).

Every output is whole numbers (ids, counts, record words, exact integers).  The result arrays
go to buffers of a fixed capacity that the caller allocates once, as the C interface is meant
to be used; a pass returns them with the record counts, zeros behind the last record.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path[:0] = [os.path.join(_ROOT, "e-hgp_b200")]

import ehgp  # noqa: E402
import workloads  # noqa: E402


def listed() -> list[dict]:
    return [
        # the smallest call: the plain one-cloud workload, where launches and host steps count
        {"name": "chain_uniform_256", "op": "chain", "shape": "uniform", "n": 256, "K": 10},
        # an ordinary interactive cloud with few orders
        {"name": "chain_mixture_5003_K4", "op": "chain", "shape": "mixture", "n": 5003, "K": 4},
        # a medium scan-like cloud, binary64, all orders
        {"name": "chain_uniform_12289", "op": "chain", "shape": "uniform", "n": 12289, "K": 10},
        # the regular volumetric cloud of the benchmark (37^3 points), the largest call
        {"name": "chain_lattice_50653", "op": "chain", "shape": "lattice", "n": 50653, "K": 10},
        # a notebook's one-off call on a tensor already on the GPU
        {"name": "fit_mixture_2999_K4", "op": "fit", "shape": "mixture", "n": 2999, "K": 4},
        # index builds: a latency-critical small one inside a host framework, and a large one
        {"name": "lbvh_noalloc_1021", "op": "lbvh_noalloc", "shape": "uniform", "n": 1021, "K": 0},
        {"name": "lbvh_clustered_200000", "op": "lbvh", "shape": "clustered", "n": 200000, "K": 0},
        # the exact geometry queries on their own
        {"name": "knn_lattice_50653", "op": "knn", "shape": "lattice", "n": 50653, "K": 11},
        {"name": "emst_clustered_100003", "op": "emst", "shape": "clustered", "n": 100003, "K": 0},
        # the support catalogues on their own: regular and clustered with exact ties
        {"name": "pairs_lattice_29791", "op": "pairs", "shape": "lattice", "n": 29791, "K": 10},
        {"name": "higher_clustered_8009", "op": "higher", "shape": "clustered", "n": 8009, "K": 10},
        # a batch of uneven clouds at a server (sizes log-uniform in [1,000, n])
        {"name": "serve_mixtures_8", "op": "serve", "shape": "mixture", "n": 12000, "K": 10, "clouds": 8},
    ]


# (op, shape, smallest n, largest n, smallest K, largest K)
_RANGES = [
    ("chain", "uniform", 64, 30000, 1, 10),
    ("chain", "lattice", 64, 46656, 1, 10),
    ("chain", "mixture", 500, 15000, 1, 10),
    ("fit", "mixture", 500, 5000, 1, 6),
    ("fit", "uniform", 64, 8000, 1, 6),
    ("lbvh_noalloc", "uniform", 16, 16384, 0, 0),
    ("lbvh", "clustered", 500, 200000, 0, 0),
    ("lbvh", "lattice", 64, 195112, 0, 0),
    ("knn", "lattice", 64, 50653, 1, 11),
    ("knn", "clustered", 500, 50000, 1, 11),
    ("emst", "clustered", 500, 100003, 0, 0),
    ("emst", "uniform", 64, 100003, 0, 0),
    ("pairs", "lattice", 64, 50653, 1, 10),
    ("pairs", "clustered", 500, 20000, 1, 10),
    ("higher", "uniform", 64, 50000, 2, 10),
    ("higher", "clustered", 500, 8009, 2, 10),
    ("serve", "mixture", 2000, 12000, 4, 10),
]


def draw(rng: random.Random) -> dict:
    op, shape, lo, hi, klo, khi = rng.choice(_RANGES)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if shape == "lattice":  # whole lattices only
        n = round(n ** (1.0 / 3.0)) ** 3
    case = {"op": op, "shape": shape, "n": n, "K": rng.randint(klo, khi)}
    if op == "serve":
        case["clouds"] = rng.randint(3, 8)
    return case


# ---- inputs -------------------------------------------------------------------------------
def _cloud(shape: str, n: int, seed: int) -> np.ndarray:
    if shape == "uniform":
        return workloads.uniform_cube(n, seed)
    if shape == "lattice":
        return workloads.jittered_lattice(round(n ** (1.0 / 3.0)), seed)
    if shape == "clustered":
        return workloads.clustered(n, seed)
    return workloads.mixture_cloud(n, np.random.Generator(np.random.PCG64(seed)))


def _serve_clouds(case: dict, seed: int) -> list[np.ndarray]:
    rng = np.random.Generator(np.random.PCG64(seed))
    # one size from each equal part of the logarithm of the range: every batch is uneven
    # and two batches of one case cost about the same
    m = case["clouds"]
    at = (np.arange(m) + 0.5) / m
    sizes = np.exp(np.log(1000.0) + at * (math.log(case["n"]) - math.log(1000.0))).astype(int)
    return [workloads.mixture_cloud(int(s), rng) for s in rng.permutation(sizes)]


def _records_per_point(K: int) -> float:
    """Support events per point at K: about 490 at K = 10, 57 at K = 4, 7 at K = 1 inside a
    homogeneous cloud."""
    return 7.0 + 483.0 * (K / 10.0) ** 2.3


def _buffers(case: dict, n: int) -> dict:
    """The output buffers a program keeps for clouds of n points in all, with room to spare."""
    op, K = case["op"], case["K"]
    r = int(1.3 * n * _records_per_point(K)) + 4096
    if op == "pairs":
        return {"records": np.zeros(64 * n + 4096, ehgp.PAIR_RECORD), "levels": np.zeros((64 * n + 4096, 4), np.uint64)}
    if op == "higher":
        return {"records": np.zeros(r, ehgp.HIGHER_RECORD)}
    if op == "knn":
        return {"ids": np.zeros((n, K), np.uint32), "meta": np.zeros((n, 2), np.uint32),
                "cutoff": np.zeros((n, 4), np.uint64)}
    nodes = (4 + 5 * K) * n + 64
    buf = {"nodes": np.zeros(nodes, ehgp.FOREST_NODE), "children": np.zeros(nodes, np.uint32),
           "batches": np.zeros(2 * r, ehgp.FOREST_BATCH), "roots": np.zeros(max(256, n // 4), ehgp.FOREST_ROOT),
           "vertical": np.zeros(nodes, ehgp.VERTICAL_ASSIGNMENT), "node_supports": np.zeros((nodes, 5), np.uint32),
           "emst_u": np.zeros(n, np.uint32), "emst_v": np.zeros(n, np.uint32)}
    if op == "chain":
        buf["emst_D"] = np.zeros((n, 4), np.uint64)
    return buf


def prepare(case: dict, seed: int) -> dict:
    op, n = case["op"], case["n"]
    st = {"op": op, "K": case["K"]}
    if op == "serve":
        st["clouds"] = _serve_clouds(case, seed)
        st["server"] = ehgp.Server(workers=4, max_points=max(n, 1000))
        st["buf"] = _buffers(case, sum(len(c) for c in st["clouds"]))
        return st
    pts = _cloud(case["shape"], n, seed)
    st["points"] = torch.from_numpy(pts).cuda() if op in ("fit", "lbvh") else pts
    if op not in ("fit", "lbvh_noalloc"):
        st["ctx"] = ehgp.Context(max_points=len(pts))
    if op in ("chain", "fit", "knn", "pairs", "higher"):
        st["buf"] = _buffers(case, len(pts))
    return st


# ---- one pass -----------------------------------------------------------------------------
_RESULT = ("nodes", "children", "batches", "roots", "vertical", "node_supports", "emst_u", "emst_v")
_COUNT = dict(zip(_RESULT, ("nodes", "children", "journal_batches", "final_roots", "vertical_assignments", "nodes")))


def _words(buf: dict) -> dict:
    """The buffers as plain words (views)."""
    return {k: b.view(np.int64 if b.dtype == np.uint64 else np.uint32).reshape(-1) for k, b in buf.items()}


def _fits(buf: dict, at: dict) -> None:
    for k, m in at.items():
        if m > len(buf[k]):
            raise RuntimeError(f"{m} {k} do not fit a buffer of {len(buf[k])}")


def _chain(st: dict) -> dict:
    ctx, K, buf = st["ctx"], st["K"], st["buf"]
    ctx.lbvh_build(st["points"], outputs=False)
    ctx._check(ctx.lib.ehgp_emst(ctx._h, C.byref(ehgp.EmstOut(buf["emst_u"].ctypes.data, buf["emst_v"].ctypes.data,
                                                              buf["emst_D"].ctypes.data, None, None, 0, None))))
    k1 = ctx.k1_forest()
    hc = ehgp.HierCounts()
    ctx._check(ctx.lib.ehgp_hierarchy(ctx._h, K, C.byref(hc)))
    _fits(buf, {k: getattr(hc, c) for k, c in _COUNT.items()})
    out = ehgp.HierOut(**{k: buf[k].ctypes.data for k in ("nodes", "children", "batches", "roots", "vertical")})
    ctx._check(ctx.lib.ehgp_hier_copy(ctx._h, C.byref(out)))
    levels = np.ascontiguousarray(buf["nodes"]["level_event"][:hc.nodes])
    ctx._check(ctx.lib.ehgp_event_supports(ctx._h, levels.ctypes.data, hc.nodes, buf["node_supports"].ctypes.data))
    res = _words(buf)
    # the k = 1 forest of a tie-free cloud has one binary node per EMST edge
    res.update({"k1_nodes": k1["nodes"].view(np.int64), "k1_children": k1["children"].view(np.int64),
                "k1_levels": k1["level_num"].view(np.int64), "k1_batches": k1["batches"].view(np.int64),
                "counts": np.array([getattr(hc, f) for f, _ in ehgp.HierCounts._fields_], np.int64)})
    return res


def _serve(st: dict) -> dict:
    srv, buf = st["server"], st["buf"]
    ids = [srv.submit(p, st["K"]) for p in st["clouds"]]
    counts, at = [], {k: 0 for k in _RESULT}  # the results one after another in the order of submission
    for rid, pts in zip(ids, st["clouds"]):
        if srv.wait(rid):
            raise RuntimeError(f"request failed: {srv.info(rid)['error']}")
        c = srv.info(rid)["counts"]
        size = {k: c[_COUNT[k]] if k in _COUNT else len(pts) - 1 for k in _RESULT}
        end = {k: at[k] + size[k] for k in _RESULT}
        _fits(buf, end)
        out = ehgp.ServedOut(*[buf[k].ctypes.data + at[k] * buf[k].strides[0] for k, _ in ehgp.ServedOut._fields_])
        if srv.lib.ehgp_result_copy(srv._h, rid, C.byref(out)):
            raise RuntimeError("ehgp_result_copy failed")
        srv.release(rid)
        counts.append(list(size.values()))
        at = end
    return {**_words(buf), "counts": np.array(counts, np.int64)}


def run(st: dict):
    op, K = st["op"], st["K"]
    if op == "chain":
        return _chain(st)
    if op == "serve":
        return _serve(st)
    if op == "fit":
        r, buf = ehgp.fit(st["points"], K), st["buf"]
        _fits(buf, {k: len(r[k]) for k in _RESULT})
        for k in _RESULT:
            buf[k][:len(r[k])] = r[k]
        return {**_words(buf), "counts": np.array([len(r[k]) for k in _RESULT], np.int64)}
    if op in ("lbvh", "lbvh_noalloc"):
        s = ehgp.lbvh_build_noalloc(st["points"]) if op == "lbvh_noalloc" else \
            st["ctx"].lbvh_build_dlpack(st["points"], outputs=True)
        return {k: getattr(s, k).view(np.int64) for k in ("source_index", "leaves", "nodes", "counters", "root_aabb")}
    ctx = st["ctx"]
    ctx.lbvh_build(st["points"], outputs=False)
    if op == "emst":
        e = ctx.emst(with_minima=False)
        f = ctx.k1_forest()
        # equal lengths make the forest's node count a property of the cloud: whole arenas, zeros behind
        out = {"u": e["u"], "v": e["v"], "D": e["D"].view(np.int64)}
        for k in ("nodes", "children", "level_num", "batches"):
            full = np.zeros((2 if k == "children" else 1) * len(e["u"]) * (f[k].shape[1] if f[k].ndim > 1 else 1), np.uint64)
            full[:f[k].size] = f[k].reshape(-1)
            out[k] = full.view(np.int64)
        return out
    buf = st["buf"]
    if op == "knn":
        ctx._check(ctx.lib.ehgp_knn(ctx._h, K, C.byref(ehgp.KnnOut(*[buf[k].ctypes.data
                                                                    for k in ("ids", "meta", "cutoff")]))))
        return _words(buf)
    count = np.zeros(1, np.uint64)
    if op == "pairs":
        out = ehgp.PairsOut(buf["records"].ctypes.data, buf["levels"].ctypes.data, len(buf["records"]),
                            count.ctypes.data)
        ctx._check(ctx.lib.ehgp_pairs(ctx._h, K, C.byref(out)))
    else:
        out = ehgp.HigherOut(buf["records"].ctypes.data, len(buf["records"]), count.ctypes.data)
        ctx._check(ctx.lib.ehgp_higher(ctx._h, K, C.byref(out)))
    return {**_words(buf), "count": count.view(np.int64)}


# ---- what a pass cannot do without --------------------------------------------------------
def _chain_bytes(n: float, K: int) -> float:
    """Input points and the arrays handed back: 48-byte batches (about 1.8 per support event),
    nodes with their supports, children and vertical maps (up to 4 per point and order), the EMST."""
    return 12.0 * n + 48.0 * 1.8 * n * _records_per_point(K) + (28.0 + 20 + 4 + 16) * 4 * K * n + 40.0 * n


def work(case: dict) -> dict:
    op, n, K = case["op"], case["n"], case["K"]
    points = (12.0 if case["shape"] in ("lattice", "mixture") else 24.0) * n
    if op in ("chain", "fit"):
        return {"bytes": _chain_bytes(n, K), "flops": 0}
    if op == "serve":
        return {"bytes": sum(_chain_bytes(len(c), K) for c in _serve_clouds(case, 0)), "flops": 0}
    if op in ("lbvh", "lbvh_noalloc"):
        return {"bytes": points + 24.0 * n + 80.0 * (2 * n - 1), "flops": 0}
    if op == "knn":
        return {"bytes": points + n * (4.0 * K + 8 + 32), "flops": 0}
    if op == "emst":
        return {"bytes": points + n * (40.0 + 32 + 48 + 16 + 56), "flops": 0}
    if op == "pairs":
        return {"bytes": points + n * 3.8 * K * 96, "flops": 0}
    return {"bytes": points + n * 0.9 * _records_per_point(K) * 64, "flops": 0}


def exact(case: dict, seed: int):
    return None  # every output is a whole number: compared for equality
