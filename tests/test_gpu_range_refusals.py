"""Ranges whose ends lie so far apart that their difference does not fit 32 bits are
refused in validation, whichever vertex they stand at, on both sides of the size from
which an upload is pipelined (2^19 entries), from host and from device arrays."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_gpu_upload import SMALL, ring

pytestmark = pytest.mark.gpu

INT_MAX, INT_MIN = 2**31 - 1, -(2**31)


@pytest.mark.parametrize("entries", [1000, SMALL + 1])
@pytest.mark.parametrize("pair", [(-1, INT_MAX), (-2, INT_MAX), (INT_MIN, 1), (INT_MIN, INT_MAX), (0, INT_MAX), (-1, 1)])
def test_wide_ranges_are_refused(mm, entries, pair):
    import torch

    for weighted in (False, True):
        for at in (0, 7, entries // 2 - 1):
            g = ring(entries, weighted, "tiled")
            g.ranges[at] = pair
            with pytest.raises(mm.MatchError) as e:
                mm.DeviceGraph(g, device=0)
            assert e.value.status == 2
            r, nb = torch.from_numpy(g.ranges).cuda(), torch.from_numpy(g.nbrs).cuda()
            handle = ctypes.c_void_p()
            assert mm.lib().mm_graph_create_device(g.n, r.data_ptr(), g.nnz, nb.data_ptr(), None, ctypes.byref(handle)) == 2
            assert not handle.value
    # reversed and negative empty ranges are lists without entries
    g = ring(1000, False, "tiled")
    g.ranges[3], g.ranges[4], g.ranges[5] = (INT_MAX, INT_MIN), (-5, -7), (INT_MIN, INT_MIN)
    with mm.DeviceGraph(g, device=0) as dg:
        assert dg.n == g.n
