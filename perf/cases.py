"""Work that a user of the framework has it do, as cases that can be timed.

A case is a dict of plain values.  listed() names the standing ones, draw()
gives more of the same ranges, prepare() makes what a user's program holds
before the call (inputs from a seed, and the generator handles that it keeps),
run() is one pass through the public entry points, exact() the same result by
plain numpy in 64 bits where that exists, work() the bytes and operations that
a pass cannot do without.

Kinds of pass:

* "ratio", "mincost": a handle in hand, as in a loop over modes or features:
  edge costs generated, one minimum ratio or minimum cost cycle solved, the
  matching read;
* "request": what a matching service does per pair, from host arrays to the
  matching, through a handle of its own;
* "batch": many uneven pairs with their costs regenerated, solved together;
* "fwdbwd": a training step's part: the ratios of many pairs as a function of
  their feature distances, forward and backward;
* "costs": the edge costs as a matrix, for a caller's own solver;
* "normals": the vertex normals of a mesh and of a curve.

Shapes are spheres pushed out by smooth noise with a silhouette curve on
them, and features that are smooth over the mesh, drawn from the seed.  The
connectivity of a sphere depends on its vertex count alone and is kept
between preparations.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "product-graph-cycles_b200"))

import cyclic_product_graphs as cpg  # noqa: E402
from cyclic_product_graphs import synthetic  # noqa: E402
from cyclic_product_graphs.autograd import ratio_cycle_objectives  # noqa: E402

# (cost, time) names with the regulariser, as users set them
PLAIN_MODES = {"mean": ("vanilla", "nomode"), "length": ("feature", "lengthnormalisation")}
CONJ_MODES = {"length": ("vanilla", "lengthnormalisation"), "robust": ("robustso3", "feature")}


def _solve(name, kind, nvx, nvy, k, conj=False, reg=False, prune=False, mode="mean", dim=32):
    return {"name": name, "kind": kind, "nvx": nvx, "nvy": nvy, "k": k, "conj": conj, "reg": reg, "prune": prune,
            "mode": mode, "dim": dim}


def listed():
    return [
        # a coarse shape in an interactive program: nothing but latency
        _solve("ratio_plain_162_20_k2", "ratio", 162, 20, 2),
        # the plain method on the resolution that the reference's CPU users run
        _solve("ratio_plain_642_60_k2", "ratio", 642, 60, 2),
        _solve("mincost_plain_642_60_k2", "mincost", 642, 60, 2),
        # odd, ragged sizes, the regulariser and a time column of its own
        _solve("ratio_plain_reg_1777_97_k3", "ratio", 1777, 97, 3, reg=True, mode="length"),
        # one request of a service: fresh handle, conjugate graph
        _solve("request_conj_2k_100_k3", "request", 2000, 100, 3, conj=True, mode="length", dim=64),
        # the ordinary higher-order pair, both solvers
        _solve("ratio_conj_5k_200_k3", "ratio", 5000, 200, 3, conj=True, mode="length", dim=64),
        _solve("mincost_conj_5k_200_k3", "mincost", 5000, 200, 3, conj=True, mode="length", dim=64),
        # the largest pair: pruned conjugate graph, SO(3) cost against feature time
        _solve("ratio_conj_prune_20k_500_k4", "ratio", 20000, 500, 4, conj=True, reg=True, prune=True, mode="robust",
               dim=64),
        # batched serving of uneven plain pairs
        {"name": "batch_plain_64_1k8k", "kind": "batch", "pairs": 64, "nvx_lo": 1000, "nvx_hi": 8000, "nvy_lo": 50,
         "nvy_hi": 250, "dim": 32},
        # differentiation: ratios of many equal pairs and their gradients
        {"name": "fwdbwd_plain_32_2k_100_k2", "kind": "fwdbwd", "pairs": 32, "nvx": 2000, "nvy": 100, "k": 2,
         "dim": 64},
        # edge costs for a solver outside the framework
        {"name": "costs_plain_reg_2k_100", "kind": "costs", "nvx": 2000, "nvy": 100, "dim": 32},
        # normals of a fine mesh and its curve, before a conjugate solve
        {"name": "normals_20k_500", "kind": "normals", "nvx": 20000, "nvy": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ratio", "ratio", "ratio", "mincost", "request", "request", "batch", "fwdbwd", "costs",
                       "normals"])
    if kind == "normals":
        return {"kind": kind, "nvx": _log_int(rng, 150, 20000), "nvy": _log_int(rng, 10, 500)}
    if kind == "costs":
        return {"kind": kind, "nvx": _log_int(rng, 150, 2000), "nvy": _log_int(rng, 10, 100), "dim": 32}
    if kind == "fwdbwd":
        return {"kind": kind, "pairs": rng.randint(2, 32), "nvx": _log_int(rng, 300, 2000),
                "nvy": _log_int(rng, 40, 100), "k": rng.randint(1, 2), "dim": rng.choice([16, 64])}
    if kind == "batch":
        lo, hi = _log_int(rng, 300, 1000), _log_int(rng, 1000, 8000)
        return {"kind": kind, "pairs": rng.randint(3, 64), "nvx_lo": lo, "nvx_hi": hi, "nvy_lo": rng.randint(40, 60),
                "nvy_hi": rng.randint(61, 250), "dim": 32}
    graph = rng.choice(["plain", "conj", "prune"]) if kind != "mincost" else rng.choice(["plain", "conj"])
    if graph == "plain":
        reg = rng.random() < 0.5
        c = _solve("", kind, _log_int(rng, 150, 8000), _log_int(rng, 10, 250), rng.randint(1, 4), reg=reg,
                   mode="length" if reg and rng.random() < 0.5 else "mean")
    elif graph == "conj":
        # K = 1 is left out: the reference's initial bound is then often that of an empty cycle
        c = _solve("", kind, _log_int(rng, 150, 5000), _log_int(rng, 10, 200), rng.randint(2, 3), conj=True,
                   mode="length", dim=64)
    else:
        c = _solve("", kind, _log_int(rng, 1000, 20000), _log_int(rng, 20, 300), rng.randint(2, 4), conj=True,
                   reg=True, prune=True, mode="robust", dim=64)
    del c["name"]
    return c


# ---------------------------------------------------------------- shapes ----
@functools.lru_cache(maxsize=256)
def _sphere(nvx):
    """Unit sphere of nvx vertices: positions, faces, both orientations of
    every edge, and each vertex's neighbours padded with itself."""
    levels = {12: 0, 42: 1, 162: 2, 642: 3}
    V, F = synthetic.icosphere(levels[nvx]) if nvx in levels else synthetic.fibonacci_sphere(nvx)
    EX = synthetic.directed_edges(F)
    start = np.searchsorted(EX[:, 0], np.arange(nvx + 1))
    nbr = np.repeat(np.arange(nvx)[:, None], int(np.diff(start).max()), axis=1)
    nbr[EX[:, 0], np.arange(len(EX)) - start[EX[:, 0]]] = EX[:, 1]
    return V, F, EX, nbr


def _smooth(x, nbr, rounds=4):
    for _ in range(rounds):
        x = 0.5 * x + 0.5 * x[nbr].mean(dim=1)
    return x


def _pair(nvx, nvy, dim, seed):
    """One shape pair: mesh and curve on the host, feature distances on the
    GPU (float32, |VX| x |VY|)."""
    V, F, EX, nbr = _sphere(nvx)
    g = torch.Generator(device="cuda").manual_seed(seed)
    at = torch.from_numpy(nbr).cuda()
    noise = _smooth(torch.randn(nvx, generator=g, device="cuda", dtype=torch.float64), at)
    noise = (noise / noise.abs().max()).cpu().numpy()
    VX = np.ascontiguousarray(V * (1.0 + 0.1 * noise)[:, None])
    VY, EY = synthetic.silhouette_curve(VX, nvy)
    out = {"VX": VX, "EX": EX, "VY": VY, "EY": EY, "F": F}
    if dim:
        fX = _smooth(torch.randn(nvx, dim, generator=g, device="cuda", dtype=torch.float32), at)
        near = torch.cdist(torch.from_numpy(VY[:, :2]).cuda(), torch.from_numpy(VX[:, :2]).cuda()).argmin(dim=1)
        fY = fX[near] + 0.05 * torch.randn(nvy, dim, generator=g, device="cuda", dtype=torch.float32)
        out["fd"] = torch.cdist(fX, fY, compute_mode="donot_use_mm_for_euclid_dist")
    return out


def _normals(p):
    # the curve is moved off the origin, so that its plane is recognised
    return (synthetic.vertex_normals(p["VX"], p["F"]),
            synthetic.normals_2d(p["VY"] + np.array([10.0, 10.0, 0.0]), p["EY"]))


def _modes(c):
    return (CONJ_MODES if c["conj"] else PLAIN_MODES)[c["mode"]]


def _handle(p, fd, conj=False, reg=False, prune=False, modes=PLAIN_MODES["mean"], normals=None):
    g = cpg.product_graph_generator(p["VX"], p["EX"], p["VY"], p["EY"], fd, conj, reg, prune)
    if conj:
        g.set_normals(*normals)
    g.set_cost_time_ratio_mode(*modes)
    return g


def _batch_sizes(c):
    """(|VX|, |VY|, K) of every pair: spread over the ranges, uneven, K 2 or 3."""
    out = []
    for i in range(c["pairs"]):
        a, b = (i * 0.6180339887498949) % 1.0, (i * 0.7548776662466927) % 1.0
        out.append((c["nvx_lo"] + int(a * (c["nvx_hi"] - c["nvx_lo"])),
                    c["nvy_lo"] + int(b * (c["nvy_hi"] - c["nvy_lo"])), 2 + i % 2))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        gens = []
        for i, (nvx, nvy, k) in enumerate(_batch_sizes(c)):
            p = _pair(nvx, nvy, c["dim"], seed * 1000 + i)
            g = _handle(p, p["fd"].double().cpu().numpy())
            g.set_max_depth_cost_time_ratio(k)
            gens.append(g)
        return {"kind": kind, "gens": gens, "rows": [_rows(y, k) for _, y, k in _batch_sizes(c)]}
    if kind == "fwdbwd":
        gens, fds = [], []
        for i in range(c["pairs"]):
            p = _pair(c["nvx"], c["nvy"], c["dim"], seed * 1000 + i)
            gens.append(_handle(p, p["fd"].double().cpu().numpy()))
            fds.append(p["fd"].requires_grad_(True))
        return {"kind": kind, "gens": gens, "fds": fds, "k": c["k"]}
    if kind == "normals":
        p = _pair(c["nvx"], c["nvy"], 0, seed)
        return {"kind": kind, "VX": p["VX"], "F": np.ascontiguousarray(p["F"].astype(np.int32)),
                "VY": p["VY"] + np.array([10.0, 10.0, 0.0]), "EY": p["EY"]}
    p = _pair(c["nvx"], c["nvy"], c["dim"], seed)
    fd = p["fd"].double().cpu().numpy()
    if kind == "costs":
        return {"kind": kind, "gen": _handle(p, fd, reg=True)}
    how = {"conj": c["conj"], "reg": c["reg"], "prune": c["prune"], "modes": _modes(c),
           "normals": _normals(p) if c["conj"] else None}
    if kind == "request":
        return {"kind": kind, "pair": p, "fd": fd, "how": how, "k": c["k"], "rows": _rows(c["nvy"], c["k"])}
    return {"kind": kind, "gen": _handle(p, fd, **how), "k": c["k"], "rows": _rows(c["nvy"], c["k"])}


def _rows(nvy, k):
    """Rows that hold any matching met here: a lap takes at most K edges per
    curve point, and a cycle a few laps."""
    return 8 * k * nvy


def _padded(matching, rows):
    """The matching in an array of fixed size, -1 past its end, as a program
    that collects many answers stores them."""
    out = np.full((rows, matching.shape[1]), -1, dtype=np.int32)
    out[:len(matching)] = matching
    return out


def _answer(r, rows):
    return {"passes": r[0], "objective": r[1], "matching": _padded(r[2], rows)}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        rs = cpg.solve_batch(state["gens"], "lawlergpu", regenerate=True)
        return {"objectives": np.array([r[1] for r in rs]), "passes": np.array([r[0] for r in rs], dtype=np.int32),
                "matchings": np.concatenate([_padded(r[2], n) for r, n in zip(rs, state["rows"])])}
    if kind == "fwdbwd":
        objectives = ratio_cycle_objectives(state["gens"], state["fds"], state["k"])
        grads = torch.autograd.grad(objectives.sum(), state["fds"])
        return {"objectives": objectives.detach(), "grads": list(grads)}
    if kind == "normals":
        return {"x": cpg.compute_normals_3d(state["VX"], state["F"]),
                "y": cpg.compute_normals_2d(state["VY"], state["EY"])}
    if kind == "request":
        g = _handle(state["pair"], state["fd"], **state["how"])
        return _answer(g.solve_with_cost_time_ratio("lawlergpu", state["k"]), state["rows"])
    g = state["gen"]
    g.generate()
    if kind == "costs":
        return g.get_cost_vector()
    if kind == "mincost":
        return _answer(g.solve_with_minimum_cost("dijkstragpu", state["k"]), state["rows"])
    return _answer(g.solve_with_cost_time_ratio("lawlergpu", state["k"]), state["rows"])


def exact(case, seed):
    """Costs and normals by numpy in 64 bits.  A solve returns a cycle, whole
    numbers, and its objective in 32 bits, which the solver's own stopping
    rules decide: no plain formula gives them, and a solve of the general
    search on the host takes minutes at most of these sizes."""
    c = case
    if c["kind"] == "normals":
        p = _pair(c["nvx"], c["nvy"], 0, seed)
        x, y = _normals(p)
        return {"x": x, "y": y}
    if c["kind"] != "costs":
        return None
    p = _pair(c["nvx"], c["nvy"], c["dim"], seed)
    fd, n = p["fd"].double().cpu().numpy(), c["nvx"]
    # rows of one curve edge (y0, y1): per mesh edge (a, b) one inside the
    # layer and one to the next, then one per vertex to the next
    a = np.concatenate([np.repeat(p["EX"][:, 0], 2), np.arange(n)])
    b = np.concatenate([np.repeat(p["EX"][:, 1], 2), np.arange(n)])
    ahead = np.concatenate([np.tile([0, 1], len(p["EX"])), np.ones(n, dtype=np.int64)])
    dx = ((p["VX"][a] - p["VX"][b]) ** 2).sum(axis=1)
    out = []
    for y0, y1 in p["EY"]:
        y = np.where(ahead == 1, y1, y0)
        dy = ((p["VY"][y0] - p["VY"][y]) ** 2).sum(axis=1)
        out.append(0.5 * (fd[a, y0] + fd[b, y]) * np.sqrt(dx + dy))
    return np.concatenate(out)[:, None]


def work(case):
    """Inputs read once and results written once, and the arithmetic of the
    least that answers the question: every product edge's cost once; for a
    ratio solve one relaxation of the whole graph for the first bound and one
    for the final verdict, for a minimum cost solve one (an add, a product with
    lambda, a sum and a comparison per source depth)."""
    c, kind = case, case["kind"]
    if kind == "normals":
        return {"bytes": 24 * 2 * (c["nvx"] + c["nvy"]) + 24 * c["nvx"] + 8 * c["nvy"], "flops": 60 * c["nvx"]}
    if kind == "batch":
        sizes = [(x, y, k, False, False, 2) for x, y, k in _batch_sizes(c)]
    elif kind == "fwdbwd":
        sizes = [(c["nvx"], c["nvy"], c["k"], False, False, 2)] * c["pairs"]
    elif kind == "costs":
        sizes = [(c["nvx"], c["nvy"], 1, False, False, 0)]
    else:
        sizes = [(c["nvx"], c["nvy"], c["k"], c["conj"], c["prune"], 1 if kind == "mincost" else 2)]
    total, flops = 0, 0
    for nvx, nvy, k, conj, prune, sweeps in sizes:
        ex = 6 * nvx - 12  # directed edges of a closed triangle mesh
        if conj:
            inter, intra = (12 * ex, 0) if prune else (17 * ex, 10 * ex)
        else:
            inter, intra = ex + nvx, 0 if prune else ex
        edges = (inter + intra) * nvy
        total += 8 * nvx * nvy + 24 * (nvx + nvy) + 8 * (ex + nvy) + (24 if conj else 16) * nvy
        flops += 6 * edges + sweeps * 4 * nvy * (inter * k + intra * (k - 1))
        if kind == "costs":
            total += 8 * edges
        if kind == "fwdbwd":
            total += 4 * nvx * nvy  # the gradients
    return {"bytes": total, "flops": flops}
