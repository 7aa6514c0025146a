"""Contraction of a graph of 2^26 vertices and more: a coarse id no longer leaves six
bits of a 32-bit sort key for an entry's place, so lists of up to 128 entries are
sorted by 64-bit keys.  On both sides of that line, against the same sums by numpy:
coarse ids, ranges and neighbours are whole numbers, weights multiples of 1/4."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 26) - 2, (1 << 26) - 1, (1 << 26) + 3])
def test_key_width(mm, n):
    import torch

    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    rng = np.random.default_rng(n)
    # lists of 1 to 128 entries (of both members together), ends all over the ids and the last ones among them
    centre = np.append(rng.choice(n - 64, 4000, replace=False), n - 1 - np.arange(8))
    deg = rng.integers(1, 61, len(centre))
    u = np.repeat(centre, deg)
    v = np.where(rng.random(len(u)) < 0.3, n - 1 - rng.integers(0, 64, len(u)), rng.integers(0, n, len(u)))
    u, v = u[u != v], v[u != v]
    key = np.unique(np.concatenate([u.astype(np.int64) * n + v, v.astype(np.int64) * n + u]))
    u, v = key // n, key % n
    w = ((np.minimum(u, v) * 7 + np.maximum(u, v) * 13) % 9 + 1) / 4
    match = np.zeros(n, np.int32)
    for a, b in zip(u[::7].tolist(), v[::7].tolist()):
        if match[a] == 0 and match[b] == 0:
            match[a] = match[b] = 4 + min(a, b)
    # expected
    ids = np.arange(n, dtype=np.int64)
    first = np.where(match >= 4, match.astype(np.int64) - 4, ids)
    own = first == ids
    cid = np.cumsum(own) - own
    cmap = cid[first]
    nc = int(own.sum())
    cu, cv = cmap[u], cmap[v]
    keep = cu != cv
    ckey, at = np.unique(cu[keep] * n + cv[keep], return_inverse=True)
    sums = np.bincount(at, w[keep])
    count = np.bincount(ckey // n, minlength=nc)
    end = np.cumsum(count)

    start = np.cumsum(np.bincount(u, minlength=n))
    ranges = torch.from_numpy(np.stack([start - np.bincount(u, minlength=n), start], 1).astype(np.int32)).cuda()
    nbrs, wt = torch.from_numpy(v.astype(np.int32)).cuda(), torch.from_numpy(w.astype(np.float32)).cuda()
    handle = ctypes.c_void_p()
    assert mm.lib().mm_graph_create_device(n, ranges.data_ptr(), len(v), nbrs.data_ptr(), wt.data_ptr(), ctypes.byref(handle)) == 0
    got_map = torch.empty(n, dtype=torch.int32, device="cuda")
    with mm.DeviceGraph.adopt(handle.value) as dg:
        with dg.contract(torch.from_numpy(match).cuda().data_ptr(), got_map.data_ptr()) as cg:
            r, nb, cw = cg.to_host()
    assert np.array_equal(got_map.cpu().numpy(), cmap)
    assert cg.n == nc and np.array_equal(r[:, 1], end) and np.array_equal(r[:, 0], end - count)
    assert np.array_equal(nb, ckey % n) and np.array_equal(cw, sums.astype(np.float32))
    del ranges, got_map
    torch.cuda.empty_cache()
    mm.lib().mm_release_cached_memory(0)
