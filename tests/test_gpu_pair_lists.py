"""Weight and check of a matching over the forms that take the pass over the lists its
ways: symmetric graphs without self-loops (one list a pair), with some (both lists
for the weight, since a self-loop ahead of the partner is what getWeight finds),
symmetric in structure only, and neither; list lengths around the pass's steps (16, 32
and 128 entries) and its last, partly filled 32 vertices.  Weights are multiples of
1/4: their sums are exact."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph
from test_gpu_check import _compare, _corruptions

pytestmark = pytest.mark.gpu


def build(n, avg, form, rng):
    u, v = rng.integers(0, n, (2, n * avg // 2))
    if form != "loops":
        u, v = u[u != v], v[u != v]
    key = np.unique(np.concatenate([u * n + v, v * n + u]))
    if form == "general":
        key = key[rng.random(len(key)) < 0.8]  # some entries one way only
    u, v = key // n, key % n
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    w = ((lo * 7 + hi * 13) % 9 + 1) / 4
    if form == "structure":
        w = ((u * 5 + v * 11) % 9 + 1) / 4
    end = np.cumsum(np.bincount(u, minlength=n))
    return SmallGraph(n, np.stack([end - np.bincount(u, minlength=n), end], 1), v, w.astype(np.float32))


@pytest.mark.parametrize("form", ["symmetric", "loops", "structure", "general"])
@pytest.mark.parametrize("n,avg", [(31, 4), (33, 16), (257, 18), (1000, 40), (1025, 130)])
def test_forms_and_sizes(mm, orc, n, avg, form):
    import torch

    rng = np.random.default_rng(n + avg)
    g = build(n, avg, form, rng)
    # a matching of some of the graph's edges, in the matchers' values
    match = np.zeros(n, np.int32)
    for a in rng.permutation(n):
        for b in g.nbrs[g.ranges[a, 0]:g.ranges[a, 1]]:
            if a != b and not match[a] and not match[b] and rng.random() < 0.6:
                match[a] = match[b] = 4 + min(a, b)
    with mm.DeviceGraph(g, device=0) as dg:
        _compare(mm, orc, torch, g, dg, match)
        for x in _corruptions(match, n, rng):
            _compare(mm, orc, torch, g, dg, x)
