"""Contraction at the edges of its list classes (8, 16, 32, 64, 128 and 2048
entries of both members together, and beyond), with parallel edges that merge and
self-loops that vanish, and the matching checks on lists around 1024 entries and on
broken matchings.  Neighbour ids and ranges are whole numbers; weights are multiples
of 1/4, so their sums are exact and equal to numpy's."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph
from test_gpu_contract import _check_contraction

pytestmark = pytest.mark.gpu


def fans(degrees, rng):
    """Two centres for each degree, joined to each other and to d - 1 leaves each,
    half of the leaves shared; and the matching of the centres, with half of the
    leaves matched in pairs, so that entries merge."""
    edges, n, pairs = [], 0, []
    for d in degrees:
        a, b = n, n + 1
        k = max(1, d - 1)
        leaf = n + 2 + np.arange(k + (k + 1) // 2)
        n += 2 + len(leaf)
        edges.append((a, b))
        edges += [(a, int(x)) for x in leaf[:k]] + [(b, int(x)) for x in leaf[len(leaf) - k:]]
        pairs.append((a, b))
        pairs += [(int(leaf[i]), int(leaf[i + 1])) for i in range(0, len(leaf) - 1, 4)]
        edges += [(int(leaf[i]), int(leaf[i + 1])) for i in range(0, len(leaf) - 1, 4)]
    name = rng.permutation(n)
    e = name[np.array(edges)]
    u, v = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    w = ((lo * 7 + hi * 13) % 9 + 1) / 4
    by = np.lexsort((v, u))
    end = np.cumsum(np.bincount(u, minlength=n))
    g = SmallGraph(n, np.stack([end - np.bincount(u, minlength=n), end], 1), v[by], w[by].astype(np.float32))
    match = np.zeros(n, np.int32)
    for a, b in pairs:
        x, y = int(name[a]), int(name[b])
        match[x] = match[y] = 4 + min(x, y)
    return g, match


@pytest.mark.parametrize("degrees", [(2, 4, 5, 8, 9), (16, 17, 32, 33), (63, 64, 65, 66), (1023, 1024, 1025, 1026), (3000, 20000)])
def test_contract_list_classes(mm, orc, degrees):
    import torch

    g, match = fans(degrees, np.random.default_rng(sum(degrees)))
    with mm.DeviceGraph(g, device=0) as dg:
        _check_contraction(mm, torch, dg, g, match)
        d = torch.from_numpy(match).cuda()
        # the coarse graph takes the symmetric path and matches as the oracle says
        with dg.contract(d.data_ptr()) as cg:
            r, nb, w = cg.to_host()
            seeds = orc.rand_seeds(5, 256)
            want, rounds, _ = orc.match(SmallGraph(cg.n, r, nb, w), 9, seeds, 0x88B81733)
            got, rr = cg.match(9, seeds)
            assert rr == rounds and np.array_equal(got, want)


@pytest.mark.parametrize("degrees", [(3, 5, 40), (1023, 1024, 1025, 1026), (5000,)])
def test_checks_of_clean_and_broken_matchings(mm, orc, degrees):
    import torch

    rng = np.random.default_rng(len(degrees))
    g, match = fans(degrees, rng)
    paired = np.flatnonzero(match >= 4)
    cases = [match, match.copy(), match.copy(), match.copy(), match.copy(), match.copy()]
    cases[1][paired[0]] = 0                                   # a partner alone
    cases[2][np.flatnonzero(match == 0)[0]] = match[paired[1]]  # a third holder
    cases[3][paired] = rng.permutation(match[paired])         # values at the wrong vertices
    cases[4][paired[0]] = 4 + g.n + 7                         # names no vertex
    a, b = np.flatnonzero(match == 0)[:2]
    cases[5][[a, b]] = 4 + min(a, b)                          # a pair that is no edge
    with mm.DeviceGraph(g, device=0) as dg:
        for i, m in enumerate(cases):
            d = torch.from_numpy(np.ascontiguousarray(m)).cuda()
            want = orc.check(g, m)
            got = dg.check(d.data_ptr())
            assert {k: got[k] for k in want if k in got} == {k: want[k] for k in want if k in got}, i
            wt, size = dg.weight(d.data_ptr())
            ow = orc.weight(g, m)
            assert size == ow[1] and wt == pytest.approx(ow[0], rel=1e-12, abs=1e-12), i


def test_contract_takes_a_value_with_one_list_beside_its_vertex(mm):
    """Vertex 4 holds its pair's value too, and has no entries: it joins the pair's
    coarse vertex and adds nothing.  With entries of its own it is refused."""
    import torch

    ends = np.array([1, 3, 5, 6, 6])
    g = SmallGraph(5, np.stack([np.r_[0, ends[:-1]], ends], 1), np.array([1, 0, 2, 1, 3, 2]),
                   np.array([1, 1, 2, 2, 3, 3], np.float32))
    cmap = torch.empty(5, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph(g, device=0) as dg:
        m = torch.tensor([4, 4, 0, 0, 4], dtype=torch.int32).cuda()
        with dg.contract(m.data_ptr(), cmap.data_ptr()) as cg:
            r, nb, w = cg.to_host()
            assert cmap.tolist() == [0, 0, 1, 2, 0]
            assert r.tolist() == [[0, 1], [1, 3], [3, 4]] and nb.tolist() == [1, 0, 2, 1] and w.tolist() == [2, 2, 3, 3]
        m = torch.tensor([4, 4, 4, 0, 0], dtype=torch.int32).cuda()
        with pytest.raises(mm.MatchError):
            dg.contract(m.data_ptr())
