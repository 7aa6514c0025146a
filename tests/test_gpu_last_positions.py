"""Lists that end at the last position an array can have (2^31 - 1 entries): scans
step past a list's end, and that must not wrap to positions before it.  The lists
stand at the end of otherwise unused arrays; the matching does not depend on where
they stand, so it equals the oracle's on the same lists at the front.  One long list
of each way it is scanned (window, a warp, a block, all blocks) stands last."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from graphs_small import SmallGraph
from test_gpu_blocks import BARRIER, hubs_with_taken_windows

pytestmark = pytest.mark.gpu

ENTRIES = 2**31 - 1
DEGREES = (40, 513, 2049, 5000, 40001)


@pytest.fixture(scope="module")
def arrays(mm):
    import torch

    if torch.cuda.mem_get_info()[0] < 64 << 30:
        pytest.skip("needs 64 GB of device memory")
    nbrs = torch.zeros(ENTRIES, dtype=torch.int32, device="cuda")
    w = torch.zeros(ENTRIES, dtype=torch.float32, device="cuda")
    yield nbrs, w
    del nbrs, w
    torch.cuda.empty_cache()
    mm.lib().mm_release_cached_memory(0)


@pytest.mark.parametrize("last", DEGREES)
def test_lists_at_the_end_of_the_arrays(mm, orc, arrays, last):
    import torch

    nbrs, w = arrays
    g = hubs_with_taken_windows(DEGREES)
    deg = (g.ranges[:, 1] - g.ranges[:, 0]).astype(np.int64)
    # lists in another order, the one of `last` entries at the end; so the ranges do not tile the arrays
    by = np.argsort(deg, kind="stable")
    hub = np.flatnonzero(deg == last)
    by = np.concatenate([by[~np.isin(by, hub[:1])], hub[:1]])
    end = np.zeros(g.n, np.int64)
    end[by] = np.cumsum(deg[by])
    at = np.concatenate([np.arange(g.ranges[v, 0], g.ranges[v, 1]) for v in by])
    total = len(at)
    low = SmallGraph(g.n, np.stack([end - deg, end], 1), g.nbrs[at], g.weights[at])
    shift = ENTRIES - total
    nbrs[shift:] = torch.from_numpy(low.nbrs).cuda()
    w[shift:] = torch.from_numpy(low.weights).cuda()
    ranges = torch.from_numpy((low.ranges.astype(np.int64) + shift).astype(np.int32)).cuda()
    assert int(ranges.max()) == ENTRIES
    torch.cuda.synchronize()
    handle = ctypes.c_void_p()
    assert mm.lib().mm_graph_create_device(g.n, ranges.data_ptr(), ENTRIES, nbrs.data_ptr(), w.data_ptr(), ctypes.byref(handle)) == 0
    out = torch.empty(g.n, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph.adopt(handle.value) as dg:
        for seed in (1, 2):
            seeds = orc.rand_seeds(seed, 256)
            for t in mm.TYPES:
                want, rounds, _ = orc.match(low, t, seeds, BARRIER)
                r = dg.match_device(t, seeds, out.data_ptr())
                assert r == rounds and np.array_equal(out.cpu().numpy(), want), (last, seed, t)
        got = dg.check(out.data_ptr())
        expect = orc.check(low, want)
        assert {k: got[k] for k in expect if k in got} == {k: expect[k] for k in expect if k in got}
        weight, size = dg.weight(out.data_ptr())
        ow = orc.weight(low, want)
        assert size == ow[1] and weight == pytest.approx(ow[0], rel=1e-12)
        # a list searched to its end: the hub paired with a vertex it does not list
        hubs = int(hub[0])
        other = int(np.setdiff1d(np.arange(g.n), np.append(low.nbrs[low.ranges[hubs, 0]:low.ranges[hubs, 1]], hubs))[0])
        m = np.zeros(g.n, np.int32)
        m[[hubs, other]] = 4 + min(hubs, other)
        out.copy_(torch.from_numpy(m))
        got, expect = dg.check(out.data_ptr()), orc.check(low, m)
        assert {k: got[k] for k in expect if k in got} == {k: expect[k] for k in expect if k in got}
