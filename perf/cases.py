"""The calls that a user of the matching library makes, as cases to measure.

A case is one call (or one short chain of calls) through the package's public
entry points: a matching of a graph that stays on the device, a batch of
graphs in one call, the learned colouring, the whole way from host arrays to a
host result, one level of coarsening, and the check of a matching.  Graphs are
of the library's own families (grid, random geometric, R-MAT, Erdos-Renyi),
built on the GPU from the seed; colouring seeds are the host rand() values the
matchers draw.
"""
import importlib
import math

import numpy as np
import torch

mm = importlib.import_module("multicore-matching_b200")
policy = importlib.import_module("multicore-matching_b200.policy")

TYPES = {"random": mm.RANDOM, "random_maximal": mm.RANDOM_MAXIMAL,
         "weighted": mm.WEIGHTED, "weighted_maximal": mm.WEIGHTED_MAXIMAL}
BATCH_LO, BATCH_HI = 1 << 10, 1 << 18  # vertices of a batch's graphs, log-uniform


def _case(name, op, graph, n, deg, type_, lists="sorted", graphs=0):
    c = {"op": op, "graph": graph, "n": n, "deg": deg, "type": type_, "lists": lists, "graphs": graphs}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest call: a graph of a thousand vertices (a coarse level, a
        # mesh patch), where the call's own latency is all there is.
        _case("grid_1k", "match", "grid", 32 * 32, 4, "random_maximal"),
        # The 512 x 512 5-point grid, unweighted, to a maximal matching.
        _case("grid_262k", "match", "grid", 512 * 512, 4, "random_maximal"),
        # A random geometric graph (a mesh of points, degree 13), heavy edges first.
        _case("rgg_1m", "match", "rgg", 1 << 20, 13, "weighted_maximal"),
        # The large power-law graph: hubs, 45% isolated vertices, 0.26 G entries.
        _case("rmat_8m", "match", "rmat", 1 << 23, 16, "weighted_maximal"),
        # A power-law graph of odd size, unweighted, the fixed twenty rounds.
        _case("rmat_300k_fixed", "match", "rmat", 300_007, 16, "random"),
        # A graph as a file gives it, lists in no order: the general path.
        _case("er_200k_unsorted", "match", "er", 200_003, 8, "weighted", lists="unsorted"),
        # Many independent graphs of uneven sizes and kinds in one call.
        _case("batch_160", "batch", "mixed", 160, 0, "weighted_maximal", graphs=160),
        # The learned colouring with the shipped policy.
        _case("policy_rgg_1m", "policy", "rgg", 1 << 20, 13, "weighted_maximal"),
        # From pinned host arrays to a host result: upload, match, download, free.
        _case("host_rmat_1m", "host", "rmat", 1 << 20, 16, "weighted_maximal"),
        # The same for a small unweighted graph, where set-up is the cost.
        _case("host_grid_10k", "host", "grid", 100 * 100, 4, "random_maximal"),
        # One level of multilevel coarsening: the matched pairs contracted.
        _case("coarsen_rgg_1m", "coarsen", "rgg", 1 << 20, 13, "weighted_maximal"),
        # A matching judged on the device: weight, size, validity, maximality.
        _case("judge_rgg_1m", "judge", "rgg", 1 << 20, 13, "weighted_maximal"),
    ]


def draw(rng):
    op = rng.choice(["match"] * 6 + ["batch", "policy", "host", "host", "coarsen", "judge"])
    if op == "batch":
        k = int(round(math.exp(rng.uniform(math.log(8), math.log(160)))))
        return _case(None, "batch", "mixed", k, 0, rng.choice(sorted(TYPES)), graphs=k)
    graph = rng.choice(["grid", "rgg", "rmat", "er"])
    hi = {"match": 23, "policy": 20, "host": 19, "coarsen": 20, "judge": 20}[op]
    n = int(round(2 ** rng.uniform(10, hi)))
    deg = {"grid": 4, "rgg": rng.choice([8, 13, 20]), "rmat": rng.choice([8, 16]), "er": rng.choice([3, 8, 16])}[graph]
    type_ = rng.choice(sorted(TYPES))
    lists = "unsorted" if op in ("match", "host") and rng.random() < 0.2 else "sorted"
    return _case(None, op, graph, n, deg, type_, lists)


# ---- graphs ----------------------------------------------------------------


def _grid_shape(n):
    w = max(1, int(math.isqrt(n)))
    return w, max(1, n // w)


def _grid(n, deg, gen):
    w, h = _grid_shape(n)
    v = torch.arange(w * h, device="cuda", dtype=torch.int64)
    x, y = v % w, v // w
    a = [v[x > 0], v[x + 1 < w], v[y > 0], v[y + 1 < h]]
    d = (-1, 1, -w, w)
    return w * h, torch.cat(a), torch.cat([s + k for s, k in zip(a, d)])


def _rgg(n, deg, gen):
    # n points uniform in the unit square, an edge where closer than r; ids in
    # no spatial order.  Candidates come from the 3 x 3 cells around a point.
    r = math.sqrt(deg / (math.pi * n))
    g = max(1, int(1.0 / r))
    xy = torch.rand((n, 2), device="cuda", dtype=torch.float64, generator=gen)
    c = (xy * g).long().clamp_(max=g - 1)
    cell, order = torch.sort(c[:, 1] * g + c[:, 0])
    start = torch.searchsorted(cell, torch.arange(g * g + 1, device="cuda"))
    src, dst = [], []
    for dy in (-1, 0, 1):
        row = c[:, 1] + dy
        ok = (row >= 0) & (row < g)
        row = row.clamp(0, g - 1) * g
        lo = start[row + (c[:, 0] - 1).clamp(min=0)]
        hi = start[row + (c[:, 0] + 1).clamp(max=g - 1) + 1]
        cnt = torch.where(ok, hi - lo, torch.zeros_like(lo))
        s = torch.repeat_interleave(torch.arange(n, device="cuda"), cnt)
        k = torch.arange(s.numel(), device="cuda") - (torch.cumsum(cnt, 0) - cnt)[s] + lo[s]
        t = order[k]
        near = ((xy[s] - xy[t]).square().sum(1) < r * r) & (s != t)
        src.append(s[near])
        dst.append(t[near])
    return n, torch.cat(src), torch.cat(dst)


def _both_ways(n, u, v):
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.cat([u * n + v, v * n + u]))
    return n, key // n, key % n


def _rmat(n, deg, gen):
    # (a, b, c, d) = (0.57, 0.19, 0.19, 0.05); ids beyond an odd n are dropped
    scale = max(1, (n - 1).bit_length())
    m = deg * n
    u = torch.zeros(m, device="cuda", dtype=torch.int64)
    v = torch.zeros(m, device="cuda", dtype=torch.int64)
    for _ in range(scale):
        p = torch.rand(m, device="cuda", generator=gen)
        u.mul_(2).add_(p >= 0.76)
        v.mul_(2).add_(((p >= 0.57) & (p < 0.76)) | (p >= 0.95))
    if n != 1 << scale:
        keep = (u < n) & (v < n)
        u, v = u[keep], v[keep]
    return _both_ways(n, u, v)


def _er(n, deg, gen):
    e = torch.randint(0, n, (2, n * deg // 2), device="cuda", generator=gen)
    return _both_ways(n, e[0], e[1])


FAMILIES = {"grid": _grid, "rgg": _rgg, "rmat": _rmat, "er": _er}


def _shift(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _pair_weights(u, v, seed):
    # uniform in (0, 1], the same for both directions of an edge
    x = (torch.minimum(u, v) << 32 | torch.maximum(u, v)) ^ (seed * 0x2545F4914F6CDD1D + 0x1234567) % (1 << 62)
    x = (x ^ _shift(x, 30)) * -0x40A7B892E31B1A47
    x = (x ^ _shift(x, 27)) * -0x6B2FB644ECCEEE15
    return (_shift(x ^ _shift(x, 31), 40) + 1).to(torch.float32) / 16777216.0


def _csr(n, u, v, seed, gen, lists="sorted"):
    """(n, ranges, neighbours, weights) on the device, entries (u, v) by vertex."""
    if lists == "unsorted":
        v, u = v.clone(), u.clone()
        shuffle = torch.argsort(torch.rand(u.numel(), device="cuda", generator=gen))
        u, by = torch.sort(u[shuffle], stable=True)
        v = v[shuffle][by]
    else:
        key = torch.sort(u * n + v).values
        u, v = key // n, key % n
    end = torch.cumsum(torch.bincount(u, minlength=n), 0)
    ranges = torch.stack([torch.cat([end.new_zeros(1), end[:-1]]), end], 1).to(torch.int32)
    return n, ranges, v.to(torch.int32), _pair_weights(u, v, seed)


def _graph(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, u, v = FAMILIES[case["graph"]](case["n"], case["deg"], gen)
    return _csr(n, u, v, seed, gen, case["lists"])


def _matched(case, seed):
    """A graph with a maximal matching of it.  Edges and matching belong to the
    case, the numbering of the vertices and the weights to the seed, so that
    the contracted graph has one size."""
    n, ranges, nbrs, w = _graph(case, case["n"])
    match = _greedy(n, ranges, nbrs, w)
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), (ranges[:, 1] - ranges[:, 0]).long())
    v = nbrs.long()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    name = torch.randperm(n, device="cuda", generator=gen)
    pairs = (match[u] >= 4) & (match[u] == match[v])
    a, b = name[u[pairs]], name[v[pairs]]
    match = torch.zeros(n, device="cuda", dtype=torch.int32)
    match[a] = (4 + torch.minimum(a, b)).to(torch.int32)
    return _csr(n, name[u], name[v], seed, gen), match


def _batch(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(case["graphs"])  # the sizes belong to the case, the graphs to the seed
    sizes = np.exp(rng.uniform(math.log(BATCH_LO), math.log(BATCH_HI), case["graphs"])).astype(int)
    kinds = rng.integers(0, 3, case["graphs"])
    offsets, us, vs = [0], [], []
    for size, kind in zip(sizes.tolist(), kinds.tolist()):
        n, u, v = (_grid, _rgg, _er)[kind](size, (4, 13, 8)[kind], gen)
        us.append(u + offsets[-1])
        vs.append(v + offsets[-1])
        offsets.append(offsets[-1] + n)
    g = _csr(offsets[-1], torch.cat(us), torch.cat(vs), seed, gen)
    return g, np.array(offsets, dtype=np.int32)


def _weighted(case):
    return case["type"].startswith("weighted")


def _upload(n, ranges, nbrs, weights):
    """A device graph from arrays that are on the device (mm_graph_create_device)."""
    import ctypes

    handle = ctypes.c_void_p()
    status = mm.lib().mm_graph_create_device(n, ranges.data_ptr(), nbrs.numel(), nbrs.data_ptr(),
                                             None if weights is None else weights.data_ptr(), ctypes.byref(handle))
    if status != 0:
        raise mm.MatchError(status, mm.lib().mm_last_error().decode())
    return mm.DeviceGraph.adopt(handle.value)


def _greedy(n, ranges, nbrs, w):
    """A maximal matching by plain torch: unmatched vertices that are each
    other's heaviest unmatched neighbour pair up, until no edge is left."""
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), (ranges[:, 1] - ranges[:, 0]).long())
    v, w = nbrs.long(), w.clone()
    match = torch.zeros(n, device="cuda", dtype=torch.int32)
    while u.numel():
        best = torch.zeros(n, device="cuda").scatter_reduce_(0, u, w, "amax")
        top = (w == best[u]) & (w == best[v])  # ties: by the smallest pair of ids
        pair = torch.minimum(u, v)[top] * n + torch.maximum(u, v)[top]
        pick = torch.full((n,), 1 << 62, device="cuda", dtype=torch.int64)
        pick.scatter_reduce_(0, u[top], pair, "amin")
        lo, hi = pick // n, pick % n
        ids = torch.arange(n, device="cuda")
        other = torch.where(lo == ids, hi, lo)
        live = pick < (1 << 62)
        mutual = live & (pick[torch.where(live, other, ids)] == pick)
        match[mutual] = (4 + torch.minimum(ids, other)[mutual]).to(torch.int32)
        keep = (match[u] == 0) & (match[v] == 0)
        u, v, w = u[keep], v[keep], w[keep]
    return match


# ---- the cases -------------------------------------------------------------


def prepare(case, seed):
    state = {"case": case, "type": TYPES[case["type"]], "seeds": mm.rand_seeds(seed)}
    if case["op"] == "batch":
        (n, ranges, nbrs, w), offsets = _batch(case, seed)
    elif case["op"] in ("coarsen", "judge"):
        (n, ranges, nbrs, w), state["match"] = _matched(case, seed)
    else:
        n, ranges, nbrs, w = _graph(case, seed)
    if case["op"] == "host":
        # pinned host arrays, as a program that uploads graphs keeps them
        host = [t.cpu().pin_memory() for t in (ranges, nbrs, w)]
        state["pinned"] = host
        r, nb, ww = (t.numpy() for t in host)
        state["graph"] = mm.Graph(n, r, nb, ww if _weighted(case) else None)
        return state
    dg = _upload(n, ranges, nbrs, w if _weighted(case) else None)
    state["graph"] = dg
    if case["op"] in ("coarsen", "judge"):
        return state
    if case["op"] == "batch":
        dg.set_batch(offsets)
    if case["op"] == "policy":
        state["mlp"] = policy.load_policy()
    dg.prepare(state["type"])
    state["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return state


class _Array:
    """A device array of a coarse graph, which it keeps alive."""

    def __init__(self, owner, pointer, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"version": 3, "data": (pointer, False), "shape": shape, "typestr": kind}


def _view(owner, pointer, shape, kind):
    if math.prod(shape) == 0:
        return torch.empty(shape, dtype=torch.float32 if kind == "<f4" else torch.int32, device="cuda")
    return torch.as_tensor(_Array(owner, pointer, shape, kind), device="cuda")


def run(state):
    op, dg, type_, seeds = state["case"]["op"], state["graph"], state["type"], state["seeds"]
    if op == "match":
        return {"rounds": dg.match_device(type_, seeds, state["out"].data_ptr()), "match": state["out"]}
    if op == "batch":
        return {"rounds": dg.match_batch(type_, seeds, state["out"].data_ptr()), "match": state["out"]}
    if op == "policy":
        return {"rounds": dg.match_policy(type_, seeds, state["out"].data_ptr(), state["mlp"]), "match": state["out"]}
    if op == "host":
        with mm.DeviceGraph(dg, device=0) as device_graph:
            match, rounds = device_graph.match(type_, seeds)
        return {"rounds": rounds, "match": match}
    if op == "coarsen":
        cmap = torch.empty(dg.n, dtype=torch.int32, device="cuda")
        coarse = dg.contract(state["match"].data_ptr(), cmap.data_ptr())
        lib, h = mm.lib(), coarse.handle
        return {"cmap": cmap,
                "ranges": _view(coarse, lib.mm_graph_device_ranges(h), (coarse.n, 2), "<i4"),
                "neighbours": _view(coarse, lib.mm_graph_device_neighbours(h), (coarse.nnz,), "<i4"),
                "weights": _view(coarse, lib.mm_graph_device_weights(h), (coarse.nnz,), "<f4")}
    weight, size = dg.weight(state["match"].data_ptr())
    return {"weight": weight, "size": size, "counts": dg.check(state["match"].data_ptr())}


def _entries(case):
    """About how many adjacency entries the case's graph has."""
    n, d = case["n"], case["deg"]
    if case["op"] == "batch":
        return _vertices(case) * (4 + 13 + 8) / 3
    if case["graph"] == "grid":
        w, h = _grid_shape(n)
        return 2 * (w * (h - 1) + h * (w - 1))
    return n * d * (1.9 if case["graph"] == "rmat" else 1.0)


def _vertices(case):
    if case["op"] == "batch":  # the mean of the log-uniform sizes
        return case["graphs"] * (BATCH_HI - BATCH_LO) / math.log(BATCH_HI / BATCH_LO)
    return case["n"]


def work(case):
    # ranges, entries (with weights where they are used) and match values
    n, e = _vertices(case), _entries(case)
    b = 12 * n + (8 if _weighted(case) else 4) * e
    if case["op"] == "batch":
        b += 8 * case["graphs"]
    if case["op"] == "coarsen":  # the coarse map and a graph of about half the vertices
        b += 4 * n + 8 * n / 2 + 8 * 0.8 * e
    return {"bytes": b, "flops": 0}


def exact(case, seed):
    """Weight sums in 64 bits; the other outputs are whole numbers."""
    if case["op"] not in ("coarsen", "judge"):
        return None
    (n, ranges, nbrs, w), match = _matched(case, seed)
    if not _weighted(case):
        w = torch.ones_like(w)
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), (ranges[:, 1] - ranges[:, 0]).long())
    v, w = nbrs.long(), w.double()
    if case["op"] == "judge":
        return {"weight": float(w[(match[u] >= 4) & (match[u] == match[v])].sum() / 2), "size": None, "counts": None}
    ids = torch.arange(n, device="cuda")
    first = torch.where(match >= 4, match.long() - 4, ids)
    own = (first == ids).long()
    cid = (torch.cumsum(own, 0) - own)[first]
    cu, cv = cid[u], cid[v]
    keep = cu != cv
    key, at = torch.unique(cu[keep] * n + cv[keep], return_inverse=True)
    sums = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").scatter_add_(0, at, w[keep])
    return {"cmap": None, "ranges": None, "neighbours": None, "weights": sums}
