"""The calls a program makes of this library, at the sizes it makes them, for timing and comparison.

Each case names a graph, a call and its options as plain values; `prepare` builds what such a
program holds before the call (the device-resident graph, the tree, the batches, in device or
page-locked host memory), `run` makes the call.

An update changes the graph and its tree, so one pass of an update case is two updates: a batch,
and then the batch that undoes it (its insertions deleted, its deletions put back with their old
weights, its weight changes reverted).  The graph is the same after every pass, both the
insertion-heavy and the deletion-heavy direction are in it, and the tree after each of the two
updates is an output.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dyng_b200 as dyng
from dyng_b200 import generators
from dyng_b200.scheduler import Scheduler

INFINITE = dyng.sssp.INFINITE_DISTANCE
DEVICE = "cuda:0"


def listed():
    return [
        # the smallest update: a handful of changes on a graph of a thousand vertices; all latency
        _update("update-tiny", 1024, 8, changes=32, memory="host"),
        # an undirected graph with rows in insertion order, an odd vertex count
        _update("update-undirected", 12345, 8, changes=601, memory="host", directed=False,
                ordered=False),
        # a multigraph with rows in insertion order: the properties of the MOSP file driver
        _update("update-multigraph", 65536, 16, changes=1000, memory="host", ordered=False,
                multi=True),
        # an ordinary batch on an ordinary graph
        _update("update-medium", 262144, 16, changes=9973),
        # mostly deletions: large invalidated subtrees, a long repair
        _update("update-deletions", 1 << 20, 16, changes=100_000, insert=0.25),
        # a small batch on a large graph, as a stream of updates to a big graph brings them
        _update("update-large-1k", 1 << 22, 16, changes=1000),
        # the benchmark workload: R-MAT scale 22, 100k changes, the learned schedule
        _update("update-large-100k", 1 << 22, 16, changes=100_000, learned=True),
        # the largest batches
        _update("update-large-1m", 1 << 22, 16, changes=1_000_000),
        # a road-like graph whose edges churn around the source: most of the tree is repaired
        _update("update-grid", 1000 * 1000, 0, changes=10_000, insert=0.5, side=1000),
        # from scratch: a power-law graph and a road-like one
        {"name": "compute-rmat", "call": "compute", "n": 1_000_003, "degree": 16, "side": 0},
        {"name": "compute-grid", "call": "compute", "n": 1024 * 1024, "degree": 0, "side": 1024},
        # three objectives: the batch applied once, three trees, the combined graph, path costs
        {"name": "mosp-k3", "call": "mosp", "n": 131072, "degree": 16, "side": 0, "k": 3,
         "changes": 5000, "insert": 0.5},
    ]


def _update(name, n, degree, *, changes, insert=0.75, memory="device", directed=True, ordered=True,
            multi=False, learned=False, side=0):
    return {"name": name, "call": "update", "n": n, "degree": degree, "side": side,
            "changes": changes, "insert": insert, "memory": memory, "directed": directed,
            "ordered": ordered, "multi": multi, "learned": learned}


def draw(rng):
    what = rng.random()
    grid = rng.random() < 0.2
    n = int(round(math.exp(rng.uniform(math.log(1024), math.log(1 << 21)))))
    side = 0
    if grid:
        side = max(32, int(math.sqrt(min(n, 1_000_000))))
        n = side * side
    degree = 0 if grid else rng.choice([8, 16])
    if what < 0.2:
        return {"call": "compute", "n": n, "degree": degree, "side": side}
    changes = int(round(math.exp(rng.uniform(math.log(16), math.log(min(500_000, n / 2))))))
    insert = rng.choice([0.25, 0.5, 0.75])
    if what < 0.3:
        n = min(n, 1 << 17)
        return {"call": "mosp", "n": n, "degree": degree or 8, "side": 0,
                "k": rng.choice([2, 3, 4]), "changes": min(changes, n // 16), "insert": insert}
    multi = rng.random() < 0.15 and n <= 1 << 18
    case = _update("", n, degree, changes=changes, insert=0.5 if grid else insert,
                   memory=rng.choice(["device", "host"]),
                   directed=multi or grid or rng.random() < 0.8, ordered=rng.random() < 0.7,
                   multi=multi, learned=rng.random() < 0.3, side=side)
    del case["name"]
    return case


# ---- inputs -----------------------------------------------------------------------------------

_shared = {}


def _stream():
    """One stream and one resources object per program; the library queues its work there."""
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
        _shared["resources"] = dyng.Resources(0, _shared["stream"].cuda_stream)
    return _shared["stream"]


def _resources():
    _stream()
    return _shared["resources"]


def _scheduler():
    if "scheduler" not in _shared:
        _shared["scheduler"] = Scheduler.load(resources=_resources())
    return _shared["scheduler"]


class _Base:
    """The graph before any batch: the edge list on the device and the library's graph.  It is the
    same for every seed (the batches and the sources differ), so it is built once per program and
    cloned."""

    def __init__(self, n, degree, side, directed=True, ordered=True, multi=False, k=1):
        if side:
            e = generators.grid(side, seed=3)
        else:
            e = generators.rmat(max(1, math.ceil(math.log2(n))), degree, device=DEVICE, seed=1)
        src = torch.from_numpy(e.src).to(DEVICE).long()
        dst = torch.from_numpy(e.dst).to(DEVICE).long()
        w = torch.from_numpy(e.weights).to(DEVICE)
        keep = (src < n) & (dst < n)
        if not directed:
            keep &= src < dst
        self.n, self.k, self.directed, self.side = n, k, directed, side
        self.key = ((src << 32) | dst)[keep]  # sorted, unique
        self.w = w[keep][:, None].repeat(1, k)  # (edges, k)
        gen = torch.Generator(DEVICE).manual_seed(5)
        if k > 1:
            self.w = torch.randint(1, 101, self.w.shape, generator=gen, device=DEVICE,
                                   dtype=torch.int32)
        # a multigraph holds parallel edges: one pair in twenty gets a second, heavier one
        self.single = torch.ones(self.key.numel(), dtype=torch.bool, device=DEVICE)
        key, w = self.key, self.w
        if multi:
            twice = torch.rand(key.numel(), generator=gen, device=DEVICE) < 0.05
            self.single = ~twice
            key = torch.cat([key, key[twice]])
            w = torch.cat([w, w[twice] + 7])
            key, order = torch.sort(key, stable=True)
            w = w[order]
        self.all_key, self.all_w = key, w
        # the library takes each undirected edge in both rows of its CSR
        if directed:
            rows, cols, weights = key >> 32, key & 0xFFFFFFFF, w
        else:
            both = torch.cat([key, ((key & 0xFFFFFFFF) << 32) | (key >> 32)])
            both, order = torch.sort(both)
            rows, cols, weights = both >> 32, both & 0xFFFFFFFF, torch.cat([w, w])[order]
        row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
        row_ptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
        self.props = dyng.GraphProperties(directed=directed, sorted=ordered, allow_multi=multi)
        self.graph = dyng.Graph.from_csr(row_ptr.cpu().numpy(), cols.to(torch.int32).cpu().numpy(),
                                         weights.t().contiguous().cpu().numpy(), self.props,
                                         num_weights=k, resources=_resources())
        self.edges = int(rows.numel())
        # grids start from the centre; the power-law graphs from vertex 0, their hub
        self.source = (side // 2) * side + side // 2 if side else 0


def _base(case):
    key = tuple(case.get(f, d) for f, d in (("n", 0), ("degree", 0), ("side", 0),
                                            ("directed", True), ("ordered", True),
                                            ("multi", False), ("k", 1)))
    bases = _shared.setdefault("bases", {})
    if key not in bases:
        bases[key] = _Base(*key)
    return bases[key]


def _parents(tree, n):
    return _view(tree.device_arrays()[1], n, "<i4", tree)


def _changes(base, case, seed, parents):
    """The batch of a case as sorted key arrays: inserted pairs (new), re-weighted edges, deleted
    edges.  Deletions are half tree edges and half any edges; on a grid half of all deletions lie
    within 64 hops of the source.  One insertion in twenty changes the weight of an edge."""
    gen = torch.Generator(DEVICE).manual_seed(1000 + seed)

    def rand(count, high):
        return torch.randint(0, max(high, 1), (count,), generator=gen, device=DEVICE)

    n, m = base.n, base.key.numel()
    total_ins = int(round(case["changes"] * case["insert"]))
    deletions = min(case["changes"] - total_ins, m // 4)
    reweighted = min(total_ins // 20, m // 8)
    # deletions: indices of edges without a parallel one
    picks = []
    if base.side:
        u = base.key >> 32
        x, y = u % base.side, u // base.side
        cx, cy = base.source % base.side, base.source // base.side
        near = torch.nonzero((x - cx).abs() + (y - cy).abs() <= 64).flatten()
        picks.append(near[rand(min(deletions // 2, near.numel() // 4), near.numel())])
    else:
        heads = torch.nonzero(parents >= 0).flatten()
        v = heads[rand(deletions // 2, heads.numel())]
        p = parents[v].long()
        if not base.directed:
            p, v = torch.minimum(p, v), torch.maximum(p, v)
        picks.append(torch.searchsorted(base.key, (p << 32) | v).clamp(max=m - 1))
    picks.append(rand(deletions - picks[0].numel(), m))
    delete = torch.unique(torch.cat(picks))
    delete = delete[base.single[delete]]
    change = torch.unique(rand(reweighted, m))
    change = change[base.single[change] & ~torch.isin(change, delete)]
    # new pairs, none of them an edge of the base graph
    u, v = rand(total_ins - change.numel(), n), rand(total_ins - change.numel(), n)
    if not base.directed:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    new = torch.unique((u << 32) | v)
    at = torch.searchsorted(base.key, new).clamp(max=m - 1)
    new = new[base.key[at] != new]
    top = 101 if base.k > 1 else (1001 if not base.side else 201)
    new_w = torch.randint(1, top, (new.numel(), base.k), generator=gen, device=DEVICE,
                          dtype=torch.int32)
    change_w = torch.randint(1, top, (change.numel(), base.k), generator=gen, device=DEVICE,
                             dtype=torch.int32)
    return delete, change, change_w, new, new_w


def _split(key):
    return (key >> 32).to(torch.int32), (key & 0xFFFFFFFF).to(torch.int32)


def _batch(ins_key, ins_w, del_key, memory, k, gen):
    """An edge batch in no particular order, and the arrays it points to."""
    order = torch.randperm(ins_key.numel(), generator=gen, device=DEVICE)
    ins_key, ins_w = ins_key[order], ins_w[order]
    del_key = del_key[torch.randperm(del_key.numel(), generator=gen, device=DEVICE)]
    arrays = [*_split(ins_key), ins_w.contiguous().reshape(-1), *_split(del_key)]
    if memory == "device":
        ptr = [a.data_ptr() for a in arrays]
        return dyng.EdgeBatch.device(ptr[0], ptr[1], ptr[2], ins_key.numel(), ptr[3], ptr[4],
                                     del_key.numel(), k), arrays
    arrays = [a.cpu().pin_memory() for a in arrays]
    host = [a.numpy() for a in arrays]
    return dyng.EdgeBatch.from_arrays(*host, num_weights=k), arrays


def _batches(base, case, seed, parents):
    delete, change, change_w, new, new_w = _changes(base, case, seed, parents)
    gen = torch.Generator(DEVICE).manual_seed(77 + seed)
    memory = case.get("memory", "host")
    there = _batch(torch.cat([new, base.key[change]]), torch.cat([new_w, change_w]),
                   base.key[delete], memory, base.k, gen)
    back = _batch(torch.cat([base.key[delete], base.key[change]]),
                  torch.cat([base.w[delete], base.w[change]]), new, memory, base.k, gen)
    return there, back


class _Pointer:
    """An array of the library's; keeps the result that owns it."""

    def __init__(self, ptr, n, kind, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False),
                                         "version": 2}


def _view(ptr, n, kind, owner):
    return torch.as_tensor(_Pointer(ptr, n, kind, owner), device=DEVICE)


def _tree_views(state, slot, tree):
    """The tree's distances and parents as tensors (made again only when the arrays moved)."""
    ptrs = tree.device_arrays()
    kept = state["views"].get(slot)
    if kept is None or kept[0] != ptrs:
        n = state["base"].n
        kept = state["views"][slot] = (ptrs, _view(ptrs[0], n, "<i8", tree),
                                       _view(ptrs[1], n, "<i4", tree))
    return kept[1], kept[2]


def _source(base, seed):
    """A source that has out-edges."""
    gen = torch.Generator(DEVICE).manual_seed(31 + seed)
    at = torch.randint(0, base.key.numel(), (1,), generator=gen, device=DEVICE)
    return int((base.key[at] >> 32).item())


def prepare(case, seed):
    _stream()
    base = _base(case)
    state = {"case": case, "base": base, "views": {}}
    if case["call"] == "compute":
        # a graph that is only read: every state solves the same one, from its own source
        state.update(graph=base.graph, source=_source(base, seed))
        return state
    graph = base.graph.clone()
    state["graph"] = graph
    if case["call"] == "mosp":
        state["result"] = dyng.mosp.compute(graph, base.source, preferences=[4, 1, 4, 2][:base.k])
        parents = _parents(state["result"].tree(0), base.n)
    else:
        state["tree"] = dyng.sssp.compute(graph, base.source)
        parents = _parents(state["tree"], base.n)
        state["scheduler"] = _scheduler() if case["learned"] else None
        state["middle"] = (torch.empty(base.n, dtype=torch.int64, device=DEVICE),
                           torch.empty(base.n, dtype=torch.int32, device=DEVICE))
    state["there"], state["back"] = _batches(base, case, seed, parents)
    return state


# ---- the pass -----------------------------------------------------------------------------------

def _counts(batch, *more):
    return np.array([batch.inserted_edges, batch.deleted_edges, batch.updated_edges, *more],
                    np.int64)


def run(state):
    return {"compute": _run_compute, "update": _run_update,
            "mosp": _run_mosp}[state["case"]["call"]](state)


def _run_compute(state):
    tree = dyng.sssp.compute(state["graph"], state["source"])
    state["tree"] = tree
    d, p = _tree_views(state, 0, tree)
    return {"distances": d, "parents": p}


def _run_update(state):
    graph, tree, scheduler = state["graph"], state["tree"], state["scheduler"]
    with torch.cuda.stream(_stream()):
        first = dyng.sssp.update(graph, state["there"][0], tree, scheduler=scheduler)
        d, p = _tree_views(state, 0, tree)
        state["middle"][0].copy_(d)
        state["middle"][1].copy_(p)
        second = dyng.sssp.update(graph, state["back"][0], tree, scheduler=scheduler)
        d, p = _tree_views(state, 0, tree)
    return {"distances_there": state["middle"][0], "parents_there": state["middle"][1],
            "counts_there": _counts(first.batch, first.invalidated, first.affected),
            "distances_back": d, "parents_back": p,
            "counts_back": _counts(second.batch, second.invalidated, second.affected)}


def _run_mosp(state):
    graph, result = state["graph"], state["result"]
    first = dyng.mosp.update(graph, state["there"][0], result)
    second = dyng.mosp.update(graph, state["back"][0], result)
    out = {"counts_there": _counts(first.batch, first.affected,
                                   *(s.affected for s in first.objectives)),
           "counts_back": _counts(second.batch, second.affected,
                                  *(s.affected for s in second.objectives)),
           "combined_distances": result.combined_distances,
           "combined_parents": result.combined_parents}
    for k in range(state["base"].k):
        out["distances_%d" % k], out["parents_%d" % k] = _tree_views(state, k, result.tree(k))
    return out


# ---- what a pass cannot do without, and what it gives -------------------------------------------

def _edges(case):
    """About how many edges the case's graph stores (a multigraph's and an undirected one's too)."""
    if case["side"]:
        return 4 * case["n"]
    return int(case["degree"] * case["n"] * 0.97)


def work(case):
    n, m = case["n"], _edges(case)
    if case["call"] == "compute":
        # every row read once (descriptor, columns, weights), every result written once
        return {"bytes": 8 * n + 8 * m + 12 * n, "flops": 0}
    k = case.get("k", 1)
    changes = case["changes"]
    directed = 1 if case.get("directed", True) else 2
    degree = m / n
    # per change and direction of the pass: the operation (12 bytes), its slot in both rows (a
    # column and k weights each), its edge index entry (16), both row descriptors (8 each)
    per_change = 12 + directed * (2 * (4 + 4 * k) + 16 + 16)
    # the repair: about one vertex per change gets another distance or parent (on a grid whose
    # source's surroundings churn, most vertices); it reads its in-row, its out-row and their
    # neighbours' words once and writes its result
    touched = 0.6 * n if case["side"] else min(n, changes)
    per_vertex = 16 + 2 * degree * 8 + degree * 8 + 12
    total = 2 * (changes * per_change + k * touched * per_vertex)
    if case["call"] == "update":
        total += 24 * n  # the first update's tree copied out
    else:
        total += 2 * n * (k * 12 + 12)  # the combined graph from the k parents, its tree
    return {"bytes": int(total), "flops": 0}


def tolerance(case):
    return "exact"  # ids, counts and distances are whole numbers, and ties go to the lowest parent


def _shortest(n, source, src, dst, w):
    """Distances and lowest-id tight parents by rounds of relaxing every edge."""
    dist = torch.full((n,), INFINITE, dtype=torch.int64, device=DEVICE)
    dist[source] = 0
    while True:
        offer = dist[src] + w
        new = dist.scatter_reduce(0, dst, offer, "amin")
        if torch.equal(new, dist):
            break
        dist = new
    # a path through an unreachable vertex is longer than INFINITE, so `dist` never takes it
    tight = (dist[src] + w == dist[dst]) & (dist[src] < INFINITE) & (dst != source)
    parents = torch.full((n,), n, dtype=torch.int64, device=DEVICE)
    parents.scatter_reduce_(0, dst[tight], src[tight], "amin")
    parents[parents == n] = -1
    return dist, parents.to(torch.int32)


def _solve(base, source, key, w):
    src, dst = key >> 32, key & 0xFFFFFFFF
    if not base.directed:
        src, dst, w = torch.cat([src, dst]), torch.cat([dst, src]), torch.cat([w, w])
    return _shortest(base.n, source, src, dst, w.long())


def exact(case, seed):
    if case["side"] > 512 or case["n"] > 1 << 21:
        return None  # thousands of rounds over millions of edges, or the largest graphs
    base = _base(case)
    if case["call"] == "compute":
        d, p = _solve(base, _source(base, seed), base.all_key, base.all_w[:, 0])
        return {"distances": d, "parents": p}
    before = [_solve(base, base.source, base.all_key, base.all_w[:, j]) for j in range(base.k)]
    if case["call"] == "mosp":
        out = {"counts_there": None, "counts_back": None, "combined_distances": None,
               "combined_parents": None}
        for j, (d, p) in enumerate(before):
            out["distances_%d" % j], out["parents_%d" % j] = d, p
        return out
    delete, change, change_w, new, new_w = _changes(base, case, seed, before[0][1])
    # deleted and re-weighted pairs have no parallel edge, so their keys name one edge each
    gone = torch.cat([base.key[delete], base.key[change]])
    keep = ~torch.isin(base.all_key, gone)
    key = torch.cat([base.all_key[keep], base.key[change], new])
    w = torch.cat([base.all_w[keep, 0], change_w[:, 0], new_w[:, 0]])
    there = _solve(base, base.source, key, w)
    return {"distances_there": there[0], "parents_there": there[1], "counts_there": None,
            "distances_back": before[0][0], "parents_back": before[0][1], "counts_back": None}
