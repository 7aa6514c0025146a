"""The 4096-graph batch where the reference's own build is absent: 12 graphs of its
sample against the restatement (bit-exact match values and round counts), and all
graphs valid and maximal.  (With that build,
test_batch4096_graphs_match_reference compares with the reference itself.)"""
from __future__ import annotations

import sys

import numpy as np
import pytest

from test_gpu_fullsize import BARRIER, ROOT

pytestmark = pytest.mark.gpu


def test_batch4096_graphs_match_restatement(mm, orc):
    import torch

    sys.path.insert(0, str(ROOT))
    import bench

    u, batch = bench.make_batch(mm, 4096, seed=3)
    off = batch["offsets"]
    seeds = orc.rand_seeds(12345, 256)
    with mm.DeviceGraph(u, device=0) as dg:
        dg.set_batch(off)
        out = torch.empty(u.n, dtype=torch.int32, device="cuda")
        rounds = dg.match_batch(9, seeds, out.data_ptr())
        # all graphs at once, in the union's numbering
        base = torch.from_numpy(np.repeat(off[:-1], np.diff(off)).astype(np.int32)).cuda()
        chk = dg.check(torch.where(out >= 4, out + base, out).data_ptr())
        assert chk["valid"] and chk["matchable"] == 0
        got = out.cpu().numpy()
    assert len(rounds) == 4096
    for i, x in batch["sample"][::4]:
        want, r, _ = orc.match(x, 9, seeds, BARRIER)
        assert np.array_equal(got[off[i]:off[i + 1]], want), i
        assert rounds[i] == r, i
    mm.lib().mm_release_cached_memory(0)
