"""The round kernel's split of the vertices over blocks, at the sizes where it
changes: one block up to 4096 vertices, chunks of 64 dealt to the blocks beyond,
blocks with a remainder; and its three ways to scan a whole list (a warp up to 512
entries, the owning block up to 32768, all blocks beyond), at their edges, with
windows of odd and even length.  Match values and round counts are whole numbers:
equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph, random_graph

pytestmark = pytest.mark.gpu

BARRIER = 0x88B81733


@pytest.mark.parametrize("n", [1, 63, 65, 513, 4095, 4096, 4097, 4609, 9999, 75_777])
@pytest.mark.parametrize("sorted_", [True, False])
def test_block_shares(mm, orc, n, sorted_):
    if sorted_:
        g = mm.Graph.er(n, 5.0, seed=n) if n > 1 else mm.Graph.grid(1, 1)
    else:
        g = random_graph(np.random.default_rng(n), n, 4.0, symmetric=True, gaps=True, shuffle_ranges=True)
    seeds = orc.rand_seeds(n, 256)
    with mm.DeviceGraph(g, device=0) as dg:
        for t in mm.TYPES:
            want, rounds, _ = orc.match(g, t, seeds, BARRIER)
            got, r = dg.match(t, seeds)
            assert r == rounds and np.array_equal(got, want), (n, t)


def hubs_with_taken_windows(degrees):
    """Hubs whose 40 heaviest and first neighbours have six heavier neighbours each
    and are taken by them in round 0: a hub still unmatched then finds nothing in
    its window of 32, and its list has to be scanned whole."""
    edges, n = [], 0
    hub = [None] * len(degrees)
    front = []
    for d in degrees:  # the window's vertices and their suitors get the smallest ids
        k = min(40, d)
        leaf = n + np.arange(k)
        mates = n + k + np.arange(6 * k)
        n += 7 * k
        front.append(leaf)
        edges.append(np.stack([np.repeat(leaf, 6), mates, np.full(6 * k, 2.0)], 1))
    rng = np.random.default_rng(sum(degrees))
    names = n + rng.permutation(sum(d + 1 for d in degrees))  # hubs and other leaves in no order
    for h, d in enumerate(degrees):
        hub[h], names = names[0], names[1:]
        rest, names = names[:d - len(front[h])], names[d - len(front[h]):]
        leaf = np.concatenate([front[h], rest])
        edges.append(np.stack([np.full(d, hub[h]), leaf, np.linspace(1.0, 0.5, d)], 1))
    e = np.concatenate(edges)
    n = int(e[:, :2].max()) + 1
    u, v = e[:, 0].astype(int), e[:, 1].astype(int)
    a, b, w = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([e[:, 2], e[:, 2]])
    by = np.lexsort((b, a))
    end = np.cumsum(np.bincount(a, minlength=n))
    return SmallGraph(n, np.stack([end - np.bincount(a, minlength=n), end], 1), b[by], w[by].astype(np.float32))


@pytest.mark.parametrize("degrees", [(31, 32, 33, 34, 511, 512, 513), (2047, 2048, 2049, 5000), (32768, 32769, 40001)])
def test_whole_list_scans(mm, orc, degrees):
    g = hubs_with_taken_windows(degrees * 4)
    scanned = 0
    with mm.DeviceGraph(g, device=0) as dg:
        import torch

        out = torch.empty(g.n, dtype=torch.int32, device="cuda")
        for seed in (1, 2, 3):
            seeds = orc.rand_seeds(seed, 256)
            for t in mm.TYPES:
                want, rounds, _ = orc.match(g, t, seeds, BARRIER)
                got, r = dg.match(t, seeds)
                assert r == rounds and np.array_equal(got, want), (degrees, seed, t)
                r, st = dg.stats(t, seeds, out.data_ptr())
                assert r == rounds and np.array_equal(out.cpu().numpy(), want), (degrees, seed, t)
                scanned += int(st[:, mm.ST_STAGED_DEG].sum())
    assert scanned >= max(degrees)  # the longest list was scanned whole at least once
