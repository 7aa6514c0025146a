"""A matching whose counts look like clean pairs but whose values clash: one value held
by three vertices, another by its own vertex alone.  The pass over the lists finds
that out while its blocks run; weight and check then are the reference's walk, equal
to the oracle's on every run, wherever the clash stands."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", [0, 1, 2])
@pytest.mark.parametrize("n", [40, 20_000, 600_000])
def test_three_holders_and_one(mm, orc, n, where):
    import torch

    g = mm.Graph.rgg(n, 8.0, seed=n)
    seeds = orc.rand_seeds(3, 256)
    match, _, _ = orc.match(g, 9, seeds, mm.DEFAULT_BARRIER)
    ids = np.arange(g.n)
    named = np.flatnonzero(match == 4 + ids)          # vertices that their own value names
    pick = [(0, 1), (len(named) // 2, len(named) - 1), (len(named) - 1, 0)][where]
    a, b = int(named[pick[0]]), int(named[pick[1]])
    v = int(np.flatnonzero((match == 4 + b) & (ids != b))[0])
    match = match.copy()
    match[v] = 4 + a                                  # a's value has three holders, b's one
    with mm.DeviceGraph(g, device=0) as dg:
        d = torch.from_numpy(match).cuda()
        want, ow = orc.check(g, match), orc.weight(g, match)
        for _ in range(5):
            got = dg.check(d.data_ptr())
            assert {k: got[k] for k in want if k in got} == {k: want[k] for k in want if k in got}
            weight, size = dg.weight(d.data_ptr())
            assert size == ow[1] and weight == pytest.approx(ow[0], rel=1e-12)
