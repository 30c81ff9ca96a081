"""The searches that users of this package have it do, as timed cases.

Every case goes through the package's public entry points: CsrProblem and the
four enactors for single searches (synchronous, as the reference's driver
calls them, or queued with the *Async calls as a loop over many sources does),
b40c_enact_search_no_alloc for callers that own the device memory, BfsBatch
and BfsServer for many searches at once, and FromHostProblem .. ExtractResults
where the graph itself is new.  A graph is made on the GPU from the seed and
handed over as host CSR arrays, which is what the entry points take; the
source vertex is drawn from the same seed.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) graph uploaded, enactor or server made, queues allocated
    run(state)          one pass: Reset and search (or the whole batch, trace, load)
    exact(case, seed)   the labels by a level-synchronous search in plain torch
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import back40computing_b200 as b40c
from back40computing_b200._lib import lib
from back40computing_b200.batch import BfsBatch
from back40computing_b200.bfs import check
from back40computing_b200.graphs import CsrGraph
from back40computing_b200.serve import BfsServer

# ---- graphs ---------------------------------------------------------------------------


def _csr(nodes, rows, cols):
    """(row_offsets, column_indices) as int32 device tensors; rows keep list order."""
    order = torch.sort(rows, stable=True).indices
    col = cols[order].to(torch.int32)
    del order
    row = torch.zeros(nodes + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(torch.bincount(rows, minlength=nodes), 0)
    return row.to(torch.int32), col


def _rmat(scale, edge_factor, directed, gen):
    """R-MAT .57/.19/.19/.05, self-loops dropped, duplicates kept."""
    m = edge_factor << scale
    u = torch.zeros(m, dtype=torch.int32, device="cuda")
    v = torch.zeros(m, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device="cuda")
        u = u * 2 + (r >= 0.76).to(torch.int32)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).to(torch.int32)
    keep = u != v
    u, v = u[keep], v[keep]
    if directed:
        return _csr(1 << scale, u, v)
    return _csr(1 << scale, torch.cat((u, v)), torch.cat((v, u)))


def _random(nodes, degree, directed, gen):
    """Uniform random edges of mean (out-)degree `degree`."""
    m = nodes * degree if directed else nodes * degree // 2
    u = torch.randint(nodes, (m,), generator=gen, device="cuda", dtype=torch.int32)
    v = torch.randint(nodes, (m,), generator=gen, device="cuda", dtype=torch.int32)
    keep = u != v
    u, v = u[keep], v[keep]
    if directed:
        return _csr(nodes, u, v)
    return _csr(nodes, torch.cat((u, v)), torch.cat((v, u)))


def _grid(width, dims):
    """2 x dims neighbours per vertex, both directions stored."""
    n = width**dims
    me = torch.arange(n, dtype=torch.int32, device="cuda")
    near, there = [], []
    for d in range(dims):
        step = width**d
        at = (me // step) % width
        near += [me - step, me + step]
        there += [at > 0, at < width - 1]
    there = torch.stack(there, 1)
    col = torch.stack(near, 1)[there]
    row = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    row[1:] = torch.cumsum(there.sum(1), 0).to(torch.int32)
    return row, col


def _graph(case, gen):
    kind = case["graph"]
    if kind == "rmat":
        return _rmat(case["scale"], case["edge_factor"], case["directed"], gen)
    if kind == "random":
        return _random(case["nodes"], case["degree"], case["directed"], gen)
    return _grid(case["width"], 2 if kind == "grid2d" else 3)


def _size(case):
    """(vertices, CSR entries) of a case's graph; its random graphs lose a few self-loops."""
    kind = case["graph"]
    if kind == "rmat":
        return 1 << case["scale"], (case["edge_factor"] << case["scale"]) * (1 if case["directed"] else 2)
    if kind == "random":
        return case["nodes"], case["nodes"] * case["degree"]
    w = case["width"]
    return (w * w, 4 * w * (w - 1)) if kind == "grid2d" else (w**3, 6 * w * w * (w - 1))


def _mix(case):
    """The graphs of a batch or a server, sizes spread over the case's range.

    As in the package's own batched and served sets: R-MAT of mixed scale and
    edge factor, a quarter of the graphs random with mean degree 16, and, for
    the server, lattices among them.
    """
    lo, hi, k = case["min_scale"], case["max_scale"], case["graphs"]
    got = []
    for i in range(k):
        scale = lo + (hi - lo) * i // max(1, k - 1)
        if case["run"] == "serve" and i % 4 == 1:
            if i % 8 == 1:
                got.append({"graph": "grid2d", "width": int(2 ** (scale / 2.0))})
            else:
                got.append({"graph": "grid3d", "width": int(2 ** (scale / 3.0))})
        elif i % 4 == 3:
            got.append({"graph": "random", "nodes": (1 << scale) - 37, "degree": 16, "directed": False})
        else:
            got.append({"graph": "rmat", "scale": scale, "edge_factor": (8, 16, 32)[i % 3], "directed": False})
    return got


def _generator(seed, k=0):
    return torch.Generator("cuda").manual_seed(1_000_003 * seed + k)


def _sources(row, count, gen, lattice):
    """Vertices to search from: any vertex of a lattice, else of degree >= 4."""
    if lattice:
        return torch.randint(row.numel() - 1, (count,), generator=gen, device="cuda").tolist()
    have = torch.nonzero(row[1:] - row[:-1] >= 4).flatten()
    return have[torch.randint(have.numel(), (count,), generator=gen, device="cuda")].tolist()


def _inputs(case, seed):
    """[(row, col, sources)] of a case, on the device."""
    if case["run"] not in ("batch", "serve"):
        gen = _generator(seed)
        row, col = _graph(case, gen)
        return [(row, col, _sources(row, 1, gen, case["graph"].startswith("grid")))]
    got = []
    for k, c in enumerate(_mix(case)):
        gen = _generator(seed, k + 1)
        row, col = _graph(c, gen)
        got.append((row, col, _sources(row, case["searches"] // case["graphs"], gen, c["graph"].startswith("grid"))))
    return got


# ---- cases ----------------------------------------------------------------------------


def _one(name, graph, *, run="search", strategy=0, parents=False, queued=False, **sizes):
    c = {"run": run, "graph": graph, "strategy": strategy, "parents": parents, "queued": queued, **sizes}
    if graph in ("rmat", "random"):
        c.setdefault("directed", False)
    return dict(c, name=name) if name else c


def _many(name, run, graphs, searches, lo, hi):
    c = {"run": run, "graphs": graphs, "searches": searches, "min_scale": lo, "max_scale": hi}
    return dict(c, name=name) if name else c


EC, CE, TP, HY = 0, 1, 2, 3


def listed():
    return [
        # The smallest call: a thousand vertices, all launches and waits.
        _one("rmat10", "rmat", scale=10, edge_factor=16),
        # A caller that owns the device memory searches its own arrays, no allocation.
        _one("rmat16-no-alloc", "rmat", run="no_alloc", scale=16, edge_factor=16),
        # Parents instead of depths, as Graph500 asks for.
        _one("rmat18-parents", "rmat", scale=18, edge_factor=16, parents=True),
        # The benchmark's graph and default strategy, searches queued one after the other.
        _one("rmat22", "rmat", scale=22, edge_factor=16, queued=True),
        # The same family under contract-expand.
        _one("rmat21-contract", "rmat", strategy=CE, scale=21, edge_factor=16, queued=True),
        # A directed graph (the reference driver's default kind) under two-phase.
        _one("rmat20-directed", "rmat", strategy=TP, scale=20, edge_factor=16, directed=True),
        # A uniform random graph of odd size under the reference driver's default strategy.
        _one("random1m-hybrid", "random", strategy=HY, nodes=1_000_003, degree=16),
        # High diameter: the benchmark's 2D lattice, about a thousand levels or more.
        _one("grid2d-1024", "grid2d", strategy=CE, width=1024),
        # and its 3D lattice, whose levels are larger than the caches like.
        _one("grid3d-256", "grid3d", strategy=CE, width=256),
        # Many searches over graphs of uneven size in one launch, every label array read back.
        _many("batch-64", "batch", 16, 64, 10, 15),
        # A burst of queries to a server whose resident graphs are small and large, lattices among them.
        _many("serve-64", "serve", 16, 64, 10, 16),
        # A graph used once: uploaded, searched, its labels read back.
        _one("load-rmat18", "rmat", run="load", scale=18, edge_factor=16),
    ]


def draw(rng):
    run = rng.choice(["search"] * 6 + ["no_alloc", "load", "batch", "serve"])
    if run in ("batch", "serve"):
        lo = rng.randint(8, 11)
        graphs = rng.choice([4, 6, 8, 12, 16])
        return _many(None, run, graphs, graphs * rng.randint(1, 64 // graphs), lo, lo + rng.randint(2, 5))
    strategy = rng.choice([EC, EC, CE, TP, HY]) if run == "search" else EC
    options = {"run": run, "strategy": strategy, "parents": run == "search" and rng.random() < 0.25,
               "queued": run == "search" and rng.random() < 0.5}
    kind = rng.choice(["rmat", "rmat", "rmat", "random", "random", "grid2d", "grid3d"])
    if kind == "rmat":
        top = {"no_alloc": 17, "load": 19}.get(run, 21)
        return _one(None, kind, scale=rng.randint(9, top), edge_factor=rng.randint(8, 32 if top < 20 else 20),
                    directed=rng.random() < 0.3, **options)
    if kind == "random":
        top = {"no_alloc": 3e5, "load": 1e6}.get(run, 3e6)
        return _one(None, kind, nodes=int(math.exp(rng.uniform(math.log(500), math.log(top)))),
                    degree=rng.randint(8, 24), directed=rng.random() < 0.3, **options)
    if kind == "grid2d":
        return _one(None, kind, width=int(math.exp(rng.uniform(math.log(24), math.log(1000)))), **options)
    return _one(None, kind, width=int(math.exp(rng.uniform(math.log(8), math.log(100 if run == "no_alloc" else 200)))),
                **options)


# ---- state and pass -------------------------------------------------------------------


class _DeviceArray:
    """A problem's label array for torch.as_tensor (no copy); a tensor made of
    it keeps the problem, and so the memory, alive."""

    def __init__(self, problem):
        self.problem = problem
        address, count = problem.device_pointers()["d_labels"], problem.nodes
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 2}


def _host_graph(row, col):
    return CsrGraph(row.cpu().numpy(), col.cpu().numpy())


def prepare(case, seed):
    inputs = _inputs(case, seed)
    run = case["run"]
    if run in ("batch", "serve"):
        many = BfsBatch() if run == "batch" else BfsServer(max_slots=64, hbm_budget_bytes=1 << 30)
        ids, sources = [], []
        for row, col, src in inputs:
            gid = many.add_graph(_host_graph(row, col))
            ids += [gid] * len(src)
            sources += src
        return {"run": run, run: many, "ids": np.array(ids, np.int32), "sources": np.array(sources, np.int32),
                "arrivals": np.zeros(len(ids))}
    row, col, (source,) = inputs[0]
    if run == "no_alloc":
        torch.cuda.synchronize()  # the search runs on another stream than the arrays were made on
        return {"run": run, "row": row, "col": col, "source": source,
                "labels": torch.empty(row.numel() - 1, dtype=torch.int32, device="cuda")}
    graph = _host_graph(row, col)
    if run == "load":
        return {"run": run, "graph": graph, "source": source, "enactor": b40c.make_enactor(case["strategy"]),
                "problem": b40c.CsrProblem(case["parents"])}
    problem = b40c.CsrProblem(case["parents"]).from_graph(graph)
    enactor = b40c.make_enactor(case["strategy"])
    frontier = enactor.GetFrontierType()
    check(problem.Reset(frontier, 1.3))
    return {"run": "queued" if case["queued"] else "search", "problem": problem, "enactor": enactor,
            "frontier": frontier, "source": source, "labels": torch.as_tensor(_DeviceArray(problem), device="cuda")}


def run(state):
    kind = state["run"]
    if kind == "search":
        check(state["problem"].Reset(state["frontier"], 1.3))
        check(state["enactor"].EnactSearch(state["problem"], state["source"]))
        return state["labels"]
    if kind == "queued":
        check(state["problem"].ResetAsync(state["frontier"], 1.3))
        check(state["enactor"].EnactSearchAsync(state["problem"], state["source"]))
        return state["labels"]
    if kind == "no_alloc":
        row, col, labels = state["row"], state["col"], state["labels"]
        depth = ctypes.c_int()
        check(lib().b40c_enact_search_no_alloc(row.numel() - 1, col.numel(), row.data_ptr(), col.data_ptr(),
                                               state["source"], labels.data_ptr(), ctypes.byref(depth), None))
        return labels
    if kind == "load":
        problem, enactor = state["problem"], state["enactor"]
        problem.from_graph(state["graph"])
        check(problem.Reset(enactor.GetFrontierType(), 1.3))
        check(enactor.EnactSearch(problem, state["source"]))
        return problem.labels()
    if kind == "batch":
        state["batch"].run(state["ids"], state["sources"])
        return [state["batch"].labels(i) for i in range(len(state["ids"]))]
    return state["serve"].run_trace(state["ids"], state["sources"], state["arrivals"], keep_labels=True)[2]


def work(case):
    """Row offsets and column indices read once per search, labels written once."""
    if case["run"] in ("batch", "serve"):
        per = case["searches"] // case["graphs"]
        sizes = [_size(c) for c in _mix(case)] * per
    else:
        sizes = [_size(case)]
    return {"bytes": sum(4 * (n + 1) + 4 * m + 4 * n for n, m in sizes), "flops": 0}


def tolerance(case):
    """Depths are whole numbers and the same everywhere.  A vertex may have many
    valid parents, and which one is recorded depends on the order the GPU's
    warps run in and on the direction of a level: between expand-contract and
    two-phase 0.23 of the parents differ on R-MAT scale 18."""
    return {"differ": 0.9} if case.get("parents") else "exact"


# ---- the same in plain torch ------------------------------------------------------------


def _depths(row, col, source):
    row, col = row.to(torch.int64), col.to(torch.int64)
    n = row.numel() - 1
    label = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    label[source] = 0
    front, depth = torch.tensor([source], device="cuda"), 0
    while front.numel():
        start, count = row[front], row[front + 1] - row[front]
        first = torch.cumsum(count, 0) - count
        at = torch.arange(int(count.sum()), device="cuda")
        at += torch.repeat_interleave(start - first, count, output_size=at.numel())
        near = col[at]
        near = near[label[near] < 0]
        depth += 1
        label[near] = depth
        if near.numel() > n // 8:
            front = torch.nonzero(label == depth).flatten()
        else:
            front = torch.unique(near)
    return label.to(torch.int32)


def exact(case, seed):
    if case.get("parents"):
        return None
    got = [_depths(row, col, s) for row, col, sources in _inputs(case, seed) for s in sources]
    return got if case["run"] in ("batch", "serve") else got[0]
