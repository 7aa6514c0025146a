"""Uploads on both sides of the size from which copies and checks are pipelined
(2^19 entries), with a last chunk of one entry and of all: the graph read back is the
one given, matchings equal the oracle's, and what must be refused is refused wherever
in the arrays it stands."""
from __future__ import annotations

import numpy as np
import pytest

from graphs_small import SmallGraph

pytestmark = pytest.mark.gpu

BARRIER = 0x88B81733
SMALL = 1 << 19


def ring(m, weighted, layout):
    """A cycle of about m / 2 vertices with m entries (two a vertex, one hub entry
    list padded to m), sorted lists; layout: 'tiled' or 'gaps'."""
    n = m // 2
    v = np.arange(n)
    nb = np.sort(np.stack([(v - 1) % n, (v + 1) % n], 1), 1).ravel()
    r = np.stack([2 * v, 2 * v + 2], 1)
    if m > 2 * n:  # one more entry: a self-loop of the last vertex
        nb = np.append(nb, n - 1)
        r[-1, 1] += 1
        nb[r[-1, 0]:r[-1, 1]].sort()
    if layout == "gaps":
        nb = np.append(nb, 0)  # an entry of no list
    lo, hi = np.minimum(np.repeat(v, r[:, 1] - r[:, 0]), nb[:m]), np.maximum(np.repeat(v, r[:, 1] - r[:, 0]), nb[:m])
    w = (((lo * 2654435761 + hi * 40503) >> 7) % 1000 + 1) / 1024
    w = np.append(w, 1.0)[:len(nb)].astype(np.float32)
    return SmallGraph(n, r, nb, w if weighted else None)


@pytest.mark.parametrize("entries", [SMALL - 1, SMALL, SMALL + 1, 24 * 65536, 24 * 65536 + 1, 2_000_001])
@pytest.mark.parametrize("layout", ["tiled", "gaps"])
def test_upload_sizes(mm, orc, entries, layout):
    seeds = orc.rand_seeds(entries, 256)
    for weighted in (False, True):
        g = ring(entries, weighted, layout)
        t = 9 if weighted else 7
        want, rounds, _ = orc.match(g, t, seeds, BARRIER)
        with mm.DeviceGraph(g, device=0) as dg:
            r, nb, w = dg.to_host()
            assert np.array_equal(r, g.ranges) and np.array_equal(nb, g.nbrs)
            assert np.array_equal(w, g.weights if weighted else np.ones(g.nnz, np.float32))
            got, rr = dg.match(t, seeds)
            assert rr == rounds and np.array_equal(got, want)


@pytest.mark.parametrize("entries", [1000, SMALL + 1, 2_000_001])
def test_upload_refusals(mm, entries):
    for where in (0, entries // 2, entries - 1):
        g = ring(entries, True, "tiled")
        g.nbrs[where] = g.n
        with pytest.raises(mm.MatchError) as e:
            mm.DeviceGraph(g, device=0)
        assert e.value.status == 2
        g = ring(entries, True, "gaps")
        g.nbrs[where] = -1
        with pytest.raises(mm.MatchError) as e:
            mm.DeviceGraph(g, device=0)
        assert e.value.status == 2
        g = ring(entries, False, "tiled")
        g.ranges[where // 2 - (where // 2 == g.n), 1] = entries + 1
        with pytest.raises(mm.MatchError) as e:
            mm.DeviceGraph(g, device=0)
        assert e.value.status == 2
    g = ring(entries, True, "tiled")  # the library goes on
    with mm.DeviceGraph(g, device=0) as dg:
        assert dg.n == g.n
    assert mm.lib().mm_release_cached_memory(0) == 0
    with mm.DeviceGraph(g, device=0) as dg:
        assert dg.nnz == g.nnz
