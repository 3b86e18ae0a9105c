"""The workloads that performance work on this solver is measured with.

Each case is one call a user's program makes: a multicut solve of one graph
(through the drop-in `rama_torch` / `rama_cuda` functions or `Solver.solve_device`),
one batch of graphs, or the parse of a MULTICUT text.  The graphs are made on the
GPU from the seed, with the shapes and cost distributions of
`rama_b200/instances.py`:

* grid2d: 4-neighbour image grid, boundary probabilities p ~ Beta(0.5, 0.5);
* voxels: 3-D grid, 6 neighbours and long-range offsets, smoothed boundaries;
* cube:   3-D grid, 6 neighbours, N(0.2, 1) costs with 5 % strongly repulsive edges;
* rag:    region adjacency graph: a planar triangulation (about 3 edges per node) with
          random node numbers, the same costs;
* knn:    k nearest neighbours of uniform points in the unit square, N(0.3, 1) costs;
* batch:  many rag graphs, node counts log-uniform;
* text:   the MULTICUT text of a rag graph.
"""
import math

import numpy as np
import torch

from rama_b200 import rama_py
from rama_b200.solver import Solver


def listed():
    return [
        # a superpixel-sized image patch: latency of the smallest calls
        {"name": "grid2d_15x17_pd", "kind": "grid2d", "h": 15, "w": 17, "mode": "PD", "call": "torch"},
        # the 64x64 image grid of the repository's first benchmark configuration
        {"name": "grid2d_64x64_pd", "kind": "grid2d", "h": 64, "w": 64, "mode": "PD", "call": "torch"},
        # a small region graph held in host arrays, primal only
        {"name": "rag_3001_p_host", "kind": "rag", "nodes": 3001, "mode": "P", "call": "host"},
        # the largest region graph of the batch configuration, solved alone
        {"name": "rag_20000_pd", "kind": "rag", "nodes": 20000, "mode": "PD", "call": "torch"},
        # a served cube request in the mode with the longest duals
        {"name": "cube_41_pd_plus", "kind": "cube", "side": 41, "mode": "PD+", "call": "device"},
        # a served k-NN request
        {"name": "knn_30000_pd", "kind": "knn", "nodes": 30000, "k": 10, "mode": "PD", "call": "torch"},
        # lower bound only on the 1M-point k-NN graph of the clustering configuration
        {"name": "knn_1000000_d", "kind": "knn", "nodes": 1000000, "k": 20, "mode": "D", "call": "device"},
        # a block of a segmentation volume
        {"name": "voxels_64x64x32_pd", "kind": "voxels", "nx": 64, "ny": 64, "nz": 32, "mode": "PD", "call": "device"},
        # the whole volume of the headline benchmark, primal only and primal-dual
        {"name": "voxels_256x256x64_p", "kind": "voxels", "nx": 256, "ny": 256, "nz": 64, "mode": "P", "call": "device"},
        {"name": "voxels_256x256x64_pd", "kind": "voxels", "nx": 256, "ny": 256, "nz": 64, "mode": "PD", "call": "device"},
        # half the batch configuration: region graphs of 500 to 20,000 nodes
        {"name": "batch_256_pd", "kind": "batch", "count": 256, "nmin": 500, "nmax": 20000, "mode": "PD"},
        # reading an instance file that is already in memory
        {"name": "text_60000", "kind": "text", "nodes": 60000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid2d", "rag", "cube", "knn", "voxels", "batch", "text"])
    call = rng.choice(["torch", "device", "host"])
    if kind == "grid2d":
        return {"kind": kind, "h": _log_int(rng, 12, 300), "w": _log_int(rng, 12, 300),
                "mode": rng.choice(["P", "PD", "PD+"]), "call": call}
    if kind == "rag":
        return {"kind": kind, "nodes": _log_int(rng, 400, 200000), "mode": rng.choice(["P", "PD", "D"]), "call": call}
    if kind == "cube":
        return {"kind": kind, "side": _log_int(rng, 16, 96), "mode": rng.choice(["P", "PD"]), "call": call}
    if kind == "knn":
        mode = rng.choice(["P", "PD", "D"])
        return {"kind": kind, "nodes": _log_int(rng, 2000, 200000 if mode == "PD" else 900000), "k": rng.choice([10, 20]),
                "mode": mode, "call": rng.choice(["torch", "device"])}
    if kind == "voxels":
        return {"kind": kind, "nx": _log_int(rng, 24, 250), "ny": _log_int(rng, 24, 250), "nz": _log_int(rng, 12, 63),
                "mode": rng.choice(["P", "PD"]), "call": rng.choice(["torch", "device"])}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 4, 250), "nmin": _log_int(rng, 200, 1000), "nmax": _log_int(rng, 2000, 20000),
                "mode": rng.choice(["P", "PD"])}
    return {"kind": kind, "nodes": _log_int(rng, 500, 60000)}


# ----------------------------------------------------------------- the graphs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _cost_of(p, scale=1.0):
    p = p.clamp(1e-12, 1 - 1e-12)
    return (torch.log((1.0 - p) / p).clamp(-10.0, 10.0) * scale).to(torch.float32)


def _arcsine(shape, g):
    """Beta(0.5, 0.5) values."""
    return torch.sin(torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (math.pi / 2)) ** 2


def _normal_costs(n, g, mean=0.2, frac_neg=0.05):
    c = torch.randn(n, generator=g, device="cuda") + mean
    if frac_neg:
        c[torch.rand(n, generator=g, device="cuda") < frac_neg] = -5.0
    return c


def _grid2d(h, w, g):
    ids = torch.arange(h * w, device="cuda", dtype=torch.int32).view(h, w)
    i = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    j = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    return i, j, _cost_of(_arcsine(i.numel(), g))


def _voxels(nx, ny, nz, g):
    b = _arcsine((1, 1, nx, ny, nz), g)
    b = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(b, (1,) * 6, mode="replicate"), 3, stride=1)[0, 0]
    ids = torch.arange(nx * ny * nz, device="cuda", dtype=torch.int32).view(nx, ny, nz)
    i, j, c = [], [], []
    for (x, y, z), scale in (((1, 0, 0), 1.0), ((0, 1, 0), 1.0), ((0, 0, 1), 1.0), ((4, 0, 0), 0.5), ((0, 4, 0), 0.5),
                             ((0, 0, 2), 0.5)):
        i.append(ids[: nx - x, : ny - y, : nz - z].reshape(-1))
        j.append(ids[x:, y:, z:].reshape(-1))
        c.append(_cost_of(torch.maximum(b[: nx - x, : ny - y, : nz - z], b[x:, y:, z:]).reshape(-1), scale))
    return torch.cat(i), torch.cat(j), torch.cat(c)


def _cube(side, g):
    ids = torch.arange(side ** 3, device="cuda", dtype=torch.int32).view(side, side, side)
    i = torch.cat([ids[:-1].reshape(-1), ids[:, :-1].reshape(-1), ids[:, :, :-1].reshape(-1)])
    j = torch.cat([ids[1:].reshape(-1), ids[:, 1:].reshape(-1), ids[:, :, 1:].reshape(-1)])
    return i, j, _normal_costs(i.numel(), g)


def _undirected(a, b, n):
    """Each edge once, endpoints and list in ascending order."""
    key = torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b))
    return (key // n).to(torch.int32), (key % n).to(torch.int32)


def _rag(n, g):
    w = int(math.ceil(math.sqrt(n)))
    h = -(-n // w)
    ids = torch.arange(h * w, device="cuda").view(h, w)
    a, b, c, d = (ids[y: h - 1 + y, x: w - 1 + x].reshape(-1) for y, x in ((0, 0), (0, 1), (1, 0), (1, 1)))
    flip = (torch.rand(a.numel(), generator=g, device="cuda") < 0.5) & (d < n)
    i = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1), torch.where(flip, a, b)])
    j = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1), torch.where(flip, d, c)])
    keep = (i < n) & (j < n)
    number = torch.randperm(n, generator=g, device="cuda")
    i, j = _undirected(number[i[keep]], number[j[keep]], n)
    return i, j, _normal_costs(i.numel(), g)


def _knn(n, k, g):
    pts = torch.rand((n, 2), generator=g, device="cuda")
    side = max(1, int(math.sqrt(n / (0.4 * k))))
    cell = (pts * side).long().clamp_(max=side - 1)
    cid = cell[:, 1] * side + cell[:, 0]
    order = torch.argsort(cid, stable=True)
    count = torch.bincount(cid, minlength=side * side)
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    slots = torch.arange(cap, device="cuda")
    src, dst = [], []
    for rows in torch.split(order, 1 << 17):  # a point's candidates: the 3x3 cells around its own
        cand, dist = [], []
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                x, y = cell[rows, 0] + dx, cell[rows, 1] + dy
                inside = (x >= 0) & (x < side) & (y >= 0) & (y < side)
                q = torch.where(inside, y * side + x, 0)
                have = inside[:, None] & (slots < count[q][:, None])
                p = order[(start[q][:, None] + slots).clamp_(max=n - 1)]
                have &= p != rows[:, None]
                cand.append(p)
                dist.append(torch.where(have, (pts[p] - pts[rows][:, None]).square().sum(2), math.inf))
        cand, dist = torch.cat(cand, 1), torch.cat(dist, 1)
        best, at = torch.topk(dist, min(k, dist.size(1)), dim=1, largest=False)
        ok = torch.isfinite(best)
        src.append(rows[:, None].expand_as(at)[ok])
        dst.append(cand.gather(1, at)[ok])
    i, j = _undirected(torch.cat(src), torch.cat(dst), n)
    return i, j, _normal_costs(i.numel(), g, 0.3, 0.0)


def _batch_sizes(case):
    """Node counts of a batch: evenly spread over the logarithm of their range."""
    n, lo, hi = case["count"], math.log(case["nmin"]), math.log(case["nmax"])
    return [int(math.exp(lo + (hi - lo) * (k + 0.5) / n)) for k in range(n)]


def _graph(case, seed):
    g = _generator(seed)
    if case["kind"] == "grid2d":
        return _grid2d(case["h"], case["w"], g)
    if case["kind"] == "voxels":
        return _voxels(case["nx"], case["ny"], case["nz"], g)
    if case["kind"] == "cube":
        return _cube(case["side"], g)
    if case["kind"] == "knn":
        return _knn(case["nodes"], case["k"], g)
    return _rag(case["nodes"], g)


def _text(case, seed):
    i, j, c = (x.cpu().numpy() for x in _graph(case, seed))
    lines = ["%d %d %.7g" % e for e in zip(i.tolist(), j.tolist(), c.tolist())]
    return ("MULTICUT\n" + "\n".join(lines) + "\n").encode()


# ------------------------------------------------------------------- the calls
_solver = None  # a program keeps one solver


def prepare(case, seed):
    global _solver
    if _solver is None:
        _solver = Solver(0)
    state = {"kind": case["kind"], "solver": _solver}
    if case["kind"] == "text":
        state["text"] = _text(case, seed)
        return state
    if case["kind"] == "batch":
        g = _generator(seed)
        sizes = _batch_sizes(case)
        sizes = [sizes[k] for k in torch.randperm(len(sizes), generator=g, device="cuda").tolist()]
        graphs = [_rag(n, g) for n in sizes]
        state["i"], state["j"], state["c"] = (torch.cat([x[k] for x in graphs]) for k in range(3))
        state["edges"] = np.cumsum([0] + [x[2].numel() for x in graphs]).astype(np.int64)
        state["nodes"] = np.cumsum([0] + sizes).astype(np.int64)
        state["mode"] = case["mode"]
        return state
    state["i"], state["j"], state["c"] = _graph(case, seed)
    state["call"], state["mode"] = case["call"], case["mode"]
    if case["call"] == "host":
        state["i"], state["j"], state["c"] = (state[k].cpu().numpy() for k in "ijc")
    if case["call"] == "device":
        state["labels"] = torch.empty(int(state["j"].max()) + 1, dtype=torch.int32, device="cuda")
    else:
        state["options"] = rama_py.multicut_solver_options(case["mode"])
    return state


def run(state):
    solver = state["solver"]
    if state["kind"] == "text":
        return solver.parse_multicut(state["text"])
    if state["kind"] == "batch":
        labels, counts, bounds, status, _ = solver.solve_batch_device(state["i"], state["j"], state["c"], state["edges"],
                                                                      state["nodes"], mode=state["mode"])
        return labels, bounds, counts, status
    if state["call"] == "host":
        labels, bound, _, _ = rama_py.rama_cuda(state["i"], state["j"], state["c"], state["options"])
        return np.asarray(labels, dtype=np.int32), bound
    if state["call"] == "torch":
        labels, bound = rama_py.rama_torch(state["i"], state["j"], state["c"], state["options"])
        return labels, bound
    labels, bound = solver.solve_device(state["i"], state["j"], state["c"], mode=state["mode"], labels=state["labels"])
    return labels, bound


# ------------------------------------------------------------- work and results
def _rag_size(n):
    w = int(math.ceil(math.sqrt(n)))
    return 3 * n - 2 * (w + n / w) + 1


def _edges_and_nodes(case):
    """Edges (for rag and knn: about) and nodes of a case."""
    if case["kind"] == "grid2d":
        h, w = case["h"], case["w"]
        return h * (w - 1) + w * (h - 1), h * w
    if case["kind"] == "cube":
        s = case["side"]
        return 3 * s * s * (s - 1), s ** 3
    if case["kind"] == "voxels":
        x, y, z = case["nx"], case["ny"], case["nz"]
        return (6 * x * y * z - (1 + 4) * y * z - (1 + 4) * x * z - (1 + 2) * x * y), x * y * z
    if case["kind"] == "knn":
        return 0.55 * case["k"] * case["nodes"], case["nodes"]
    if case["kind"] == "batch":
        sizes = _batch_sizes(case)
        return sum(_rag_size(n) for n in sizes), sum(sizes)
    return _rag_size(case["nodes"]), case["nodes"]


def work(case):
    """Every edge read once (two ids and a cost), every label written once; a
    comparison and an addition per edge.  A text: its characters and the edges."""
    edges, nodes = _edges_and_nodes(case)
    if case["kind"] == "text":
        return {"bytes": (2 * math.log10(case["nodes"]) + 13 + 12) * edges, "flops": edges}
    return {"bytes": 12 * edges + (0 if case["mode"] == "D" else 4 * nodes), "flops": 2 * edges}


def tolerance(case):
    """Labels, counts and parsed ids are whole values and the same for every
    correct implementation of the solver's order of operations.  The bound
    without a dual is a 64-bit sum; with one, its messages are 32-bit floats
    (measured 1.8e-7 from the same messages in 64 bits).  A parsed cost is the
    nearest float."""
    if case["kind"] == "text":
        return "exact"
    return {"rel": 1e-10 if case["mode"] == "P" else 7e-7, "differ": 0.0}


def exact(case, seed):
    """The parsed values in 64 bits, and the bound without a dual: the sum of the
    negative costs.  Labels, and the bound after message passing, have no value
    that plain arithmetic gives without restating the solver."""
    if case["kind"] == "text":
        rows = np.array([line.split() for line in _text(case, seed).decode().splitlines()[1:]])
        return rows[:, 0].astype(np.int32), rows[:, 1].astype(np.int32), rows[:, 2].astype(np.float64)
    if case["mode"] != "P":
        return None
    if case["kind"] == "batch":
        state = prepare(case, seed)
        c = state["c"].double().clamp(max=0).cpu().numpy()
        return None, np.array([c[a:b].sum() for a, b in zip(state["edges"][:-1], state["edges"][1:])]), None, None
    bound = float(_graph(case, seed)[2].double().clamp(max=0).sum())
    return None, torch.tensor([bound], dtype=torch.float64) if case["call"] == "torch" else bound
