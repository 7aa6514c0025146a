"""Round counts of a batch whose graphs fill, cut and share the 1024-vertex spans
that the counts are taken over: single vertices, empty graphs, graphs of 1023 to
1025 vertices and one of several spans, graph by graph equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 1, 2, 1023, 1024, 1025), (1024, 1024, 4096), (700, 0, 0, 324, 5000, 0, 3), (16,) * 200])
def test_batch_round_counts(mm, orc, sizes):
    import torch

    graphs = [mm.Graph.er(n, 4.0, seed=i + 1) if n > 1 else mm.Graph.grid(1, 1) for i, n in enumerate(sizes) if n]
    u, off = mm.Graph.union(graphs)
    full, k = [0], 0
    for n in sizes:  # empty graphs take no vertices
        k += n > 0
        full.append(int(off[k]))
    seeds = orc.rand_seeds(11, 256)
    with mm.DeviceGraph(u, device=0) as dg:
        dg.set_batch(np.array(full, np.int32))
        out = torch.empty(u.n, dtype=torch.int32, device="cuda")
        for t in mm.TYPES:
            rounds = dg.match_batch(t, seeds, out.data_ptr())
            got, it = out.cpu().numpy(), iter(graphs)
            for i, n in enumerate(sizes):
                if not n:
                    assert rounds[i] == (1 if t in (7, 9) else 20)
                    continue
                want, want_rounds, _ = orc.match(next(it), t, seeds, 0x88B81733)
                assert rounds[i] == want_rounds and np.array_equal(got[full[i]:full[i + 1]], want), (i, t)
