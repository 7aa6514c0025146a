"""What a contraction writes into the caller's arrays: the coarse map may be the match
array itself (wholly, or shifted into it), with the result of a map apart; a call that
is refused leaves the map as it was."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matched(mm, orc, n):
    g = mm.Graph.rgg(n, 9.0, seed=n)
    match, _, _ = orc.match(g, 9, orc.rand_seeds(1, 256), mm.DEFAULT_BARRIER)
    return g, match


@pytest.mark.parametrize("n", [50, 4097, 300_000])
def test_map_in_place_of_the_matching(mm, orc, n):
    import torch

    g, match = matched(mm, orc, n)
    with mm.DeviceGraph(g, device=0) as dg:
        d = torch.from_numpy(match).cuda()
        apart = torch.empty_like(d)
        with dg.contract(d.data_ptr(), apart.data_ptr()) as cg:
            want = cg.to_host()
        for shift in (0, 1, 1000 % n):
            buf = torch.full((n + shift,), -7, dtype=torch.int32, device="cuda")
            buf[shift:] = d
            with dg.contract(buf[shift:].data_ptr(), buf.data_ptr()) as cg:
                assert all(np.array_equal(x, y) for x, y in zip(cg.to_host(), want)), shift
            assert torch.equal(buf[:n], apart), shift


def test_refused_call_leaves_the_map(mm, orc):
    import torch

    g, match = matched(mm, orc, 20_000)
    a = int(np.flatnonzero(match == 4 + np.arange(g.n))[7])
    bad = [match.copy() for _ in range(3)]
    bad[0][a] = 0                                                  # the named vertex does not hold its value
    bad[1][np.flatnonzero(match >= 4)[3]] = 4 + g.n + 5            # names no vertex
    third = np.flatnonzero((match < 4) & (g.ranges[:, 1] > g.ranges[:, 0]))[0]
    bad[2][third] = 4 + a                                          # a third holder with entries
    cmap = torch.full((g.n,), -7, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph(g, device=0) as dg:
        for m in bad:
            with pytest.raises(mm.MatchError) as e:
                dg.contract(torch.from_numpy(m).cuda().data_ptr(), cmap.data_ptr())
            assert e.value.status == 1
            assert int((cmap != -7).sum()) == 0
        with dg.contract(torch.from_numpy(match).cuda().data_ptr(), cmap.data_ptr()) as cg:
            assert int(cmap.max()) == cg.n - 1
