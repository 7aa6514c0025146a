"""The finish phase off the symmetric path: lists that tile the arrays and are
symmetric in structure, but in any order, with parallel edges, self-loops, weights
that differ in the two directions or can never be picked.  Equal to the oracle's
matchings, with the finish phase (its items are counted) and without it."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SPECIAL_WEIGHTS, SmallGraph

pytestmark = pytest.mark.gpu

BARRIER = 0x88B81733


def lists(n, avg, seed, order, weights, loops):
    rng = np.random.default_rng(seed)
    m = n * avg // 2
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    u, v = u[u != v], v[u != v]
    again = rng.random(len(u)) < 0.05  # parallel edges, in both lists
    u, v = np.concatenate([u, u[again]]), np.concatenate([v, v[again]])
    a, b = np.concatenate([u, v]), np.concatenate([v, u])
    if weights == "equal":
        w = rng.integers(1, 9, len(u)) / 4
        w = np.concatenate([w, w])
    else:
        w = rng.integers(1, 9, len(a)) / 4
        odd = rng.random(len(a)) < 0.2
        w[odd] = SPECIAL_WEIGHTS[rng.integers(0, len(SPECIAL_WEIGHTS), odd.sum())]
    if loops:
        s = rng.integers(0, n, n // 50)
        a, b, w = np.concatenate([a, s]), np.concatenate([b, s]), np.concatenate([w, np.ones(len(s))])
    key = rng.permutation(len(a)) if order == "any" else b
    by = np.lexsort((key, a))
    end = np.cumsum(np.bincount(a, minlength=n))
    return SmallGraph(n, np.stack([end - np.bincount(a, minlength=n), end], 1), b[by], w[by].astype(np.float32))


@pytest.mark.parametrize("n", [4097, 20_011])
@pytest.mark.parametrize("avg", [3, 12])
@pytest.mark.parametrize("order,weights,loops", [("any", "equal", False), ("any", "odd", True), ("sorted", "odd", False)])
def test_finish_phase_of_unsorted_and_asymmetric_lists(mm, orc, n, avg, order, weights, loops):
    import torch

    g = lists(n, avg, n + avg, order, weights, loops)
    seeds = orc.rand_seeds(n, 256)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph(g, device=0) as dg:
        for t in mm.TYPES:
            want, rounds, ost = orc.match(g, t, seeds, BARRIER)
            played = 0
            for div in (0, 2, 3, -1):
                dg.tune(div, 0)
                got, r = dg.match(t, seeds)
                assert r == rounds and np.array_equal(got, want), (t, div)
                r, st = dg.stats(t, seeds, out.data_ptr())
                assert r == rounds and np.array_equal(out.cpu().numpy(), want), (t, div)
                assert np.array_equal(st[:, :8], ost[:, :8]), (t, div)
                played += int(st[:, mm.ST_FINISH_ITEMS].sum())
            assert played > 0
