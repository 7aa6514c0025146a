"""Small graphs with long lists: one block or several by the entries in lists longer
than a window, the lists of a round left to all blocks where they are many (random
types on dense graphs), on both sides of each line; and the places where a block's
own buffers end, more than 1024 lists to scan whole in a round (the rest goes to the
shared list at once, also from the one-block kernel) and more than 4800 blue items
(their requests go to global memory).  Match values, round counts and the counters'
round count are whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph

pytestmark = pytest.mark.gpu

BARRIER = 0x88B81733


def from_pairs(n, u, v, w, both=True):
    if both:
        u, v, w = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    by = np.lexsort((v, u))
    count = np.bincount(u, minlength=n)
    end = np.cumsum(count)
    return SmallGraph(n, np.stack([end - count, end], 1), v[by], w[by].astype(np.float32))


def random_dense(n, deg, seed):
    """About deg entries a vertex (all of them where deg >= n - 1), distinct weights."""
    rng = np.random.default_rng(seed)
    if deg >= n - 1:
        u, v = np.triu_indices(n, 1)
    else:
        e = np.unique(np.sort(rng.integers(0, n, (n * deg // 2, 2)), axis=1), axis=0)
        e = e[e[:, 0] != e[:, 1]]
        u, v = e[:, 0], e[:, 1]
    return from_pairs(n, u, v, rng.permutation(len(u)) / len(u) + 0.5)


def compare(mm, orc, g, seed, types, blocks=0, scanned=0):
    import torch

    seeds = orc.rand_seeds(seed, 256)
    out = torch.empty(g.n, dtype=torch.int32, device="cuda")
    staged = 0
    with mm.DeviceGraph(g, device=0) as dg:
        dg.tune(0, blocks)
        for t in types:
            want, rounds, _ = orc.match(g, t, seeds, BARRIER)
            for _ in range(2):
                got, r = dg.match(t, seeds)
                assert r == rounds and np.array_equal(got, want), (g.n, t)
            r, st = dg.stats(t, seeds, out.data_ptr())
            assert r == rounds and np.array_equal(out.cpu().numpy(), want), (g.n, t)
            staged = max(staged, int(st[:, mm.ST_STAGED_ITEMS].max()))
    assert staged >= scanned


# 2^17 entries in long lists (one block or several, random types) lie between 362 and
# 363 vertices that all list each other; 384 entries a vertex (dense) at 385, lists of
# 448 on average (left to all blocks) at 449
@pytest.mark.parametrize("n,deg", [(64, 63), (362, 361), (363, 362), (384, 383), (385, 384), (386, 385), (448, 447),
                                   (449, 448), (700, 699),
                                   (1023, 500), (2049, 64), (4095, 130), (4097, 130), (4096, 700), (9001, 450)])
def test_dense(mm, orc, n, deg):
    compare(mm, orc, random_dense(n, deg, n), n, mm.TYPES)


@pytest.mark.parametrize("n", [700, 3000])
def test_dense_learned(mm, orc, n):
    import importlib

    import torch

    mlp = importlib.import_module(mm.__name__ + ".policy").load_policy()
    g = random_dense(n, 600, n)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph(g, device=0) as dg:
        for t in mm.TYPES:
            dg.match_policy(t, orc.rand_seeds(n, 256), out.data_ptr(), mlp)
            c = orc.check(g, out.cpu().numpy())
            assert c["valid"] and (t in (mm.RANDOM, mm.WEIGHTED) or c["matchable"] == 0)


def taken_windows(n, k, both):
    """n vertices that all list the same k vertices first (and heaviest), and their
    neighbours on a ring; the k have partners of their own that they prefer."""
    ids = np.arange(n)
    front, mates = np.arange(k), k + np.arange(6 * k)
    body = 7 * k + ids
    nxt = np.roll(body, -1)
    total = 7 * k + n
    ring = (body, nxt, np.full(n, 0.5))
    mate = (np.repeat(front, 6), mates, np.full(6 * k, 4.0))
    to_front = (np.repeat(body, k), np.tile(front, n), np.tile(np.linspace(2.0, 1.0, k), n))
    two_way = [ring, mate] + ([to_front] if both else [])
    u, v, w = (np.concatenate([x[i] for x in two_way]) for i in range(3))
    u, v, w = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    if not both:
        u, v, w = (np.concatenate([a, b]) for a, b in zip((u, v, w), to_front))
    return from_pairs(total, u, v, w, both=False)


@pytest.mark.parametrize("n,both,blocks", [(2600, False, 0), (3500, True, 0), (400_000, True, 1)])
def test_more_lists_than_a_block_collects(mm, orc, n, both, blocks):
    """A block's buffer holds 1024 lists of a round; a block has some 1300 to 1700 here."""
    g = taken_windows(n, 34, both)
    compare(mm, orc, g, 5, mm.TYPES, blocks, scanned=1025 if n < 4096 else 1025 * 148)


def test_more_blue_items_than_requests_in_shared_memory(mm, orc):
    """1.6 million vertices in 148 blocks: some 5400 blue ones a block in round 0."""
    g = mm.Graph.er(1_600_000, 4.0, seed=2)
    compare(mm, orc, g, 3, (mm.RANDOM_MAXIMAL, mm.WEIGHTED), 1)
    rng = np.random.default_rng(1)
    w = rng.random(g.nnz).astype(np.float32)  # weights that differ by direction: the requests' key halves spill too
    compare(mm, orc, mm.Graph(g.n, g.ranges, g.nbrs, w), 3, (mm.WEIGHTED,), 1)
