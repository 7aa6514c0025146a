"""A graph uploaded, matched and given back, over and over: the device memory that the
first round took serves all later ones, and a first matching takes about the same
time every time (the memory for it is there: nothing is mapped or moved inside the
call)."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [19, 23])
def test_steps_take_no_more_memory_and_no_odd_time(mm, scale):
    import torch

    g = mm.Graph.rmat(scale, 16, seed=1)
    host = [torch.from_numpy(np.ascontiguousarray(x)).pin_memory() for x in (g.ranges, g.nbrs, g.weights)]
    pinned = mm.Graph(g.n, *(x.numpy() for x in host))
    seeds = mm.rand_seeds(12345, 255)
    ms, free, first = [], [], None
    for _ in range(20):
        with mm.DeviceGraph(pinned, device=0) as dg:
            torch.cuda.mem_get_info()
            t0 = time.perf_counter()
            match, rounds = dg.match(mm.WEIGHTED_MAXIMAL, seeds)
            ms.append((time.perf_counter() - t0) * 1e3)
            if first is None:
                first = (match, rounds)
            assert rounds == first[1] and np.array_equal(match, first[0])
        free.append(torch.cuda.mem_get_info()[0])
    assert min(free[1:]) == max(free[1:])
    # (a matching with its result to pageable memory: 1 ms at 2^19, 9 ms at 2^23; one
    # step may be the host's own hiccup)
    assert sorted(ms[2:])[-2] < 2.0 * np.median(ms[2:]) + 1.0, ms
    mm.lib().mm_release_cached_memory(0)
