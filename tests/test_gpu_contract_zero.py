"""Sums of weights that are zero: every way to merge a coarse list (8, 16, 32, 64, 128
and 2048 entries, and beyond) takes the sum from 0, so an entry of weight -0 becomes
+0 in the coarse graph, whatever its list's length; both ends of a coarse edge then
carry the same bits, and the coarse graph takes the symmetric path."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degrees", [(3, 7, 8), (9, 16, 17, 31, 32), (33, 63, 64, 65, 127, 128), (129, 2048), (2049, 5000)])
def test_negative_zero_weights(mm, degrees):
    import torch

    # hubs with d leaves each: every leaf is one entry long, so the two ends of an edge
    # are merged in different ways; no two entries merge
    edges, n = [], 0
    for d in degrees:
        edges += [(n, n + 1 + k) for k in range(d)]
        n += 1 + d
    e = np.array(edges)
    u, v = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    by = np.lexsort((v, u))
    end = np.cumsum(np.bincount(u, minlength=n))
    g = SmallGraph(n, np.stack([end - np.bincount(u, minlength=n), end], 1), v[by], np.full(len(u), -0.0, np.float32))
    with mm.DeviceGraph(g, device=0) as dg:
        with dg.contract(torch.zeros(n, dtype=torch.int32, device="cuda").data_ptr()) as cg:
            r, nb, w = cg.to_host()
            assert np.array_equal(r, g.ranges) and np.array_equal(nb, g.nbrs)
            assert not w.view(np.uint32).any()
