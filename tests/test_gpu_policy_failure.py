"""A learned matching whose features find no memory, on a stream of the caller's: it
ends with nothing in flight there, so the next call on the graph may come on another
stream at once; the matchings that follow equal those of an untouched graph."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

from test_gpu_failure import ALLOC, USED, debug

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 400_000])
def test_out_of_memory_between_state_and_features(mm, orc, n):
    import torch

    policy = importlib.import_module(mm.__name__ + ".policy")
    mlp = policy.load_policy()
    g = mm.Graph.rgg(n, 13.0, seed=5)
    seeds = orc.rand_seeds(12345, 256)
    want, rounds, _ = orc.match(g, 9, seeds, mm.DEFAULT_BARRIER)
    out = torch.empty(n, dtype=torch.int32, device="cuda")

    def limited(dg, limit, stream):
        debug(mm, ALLOC, limit)
        try:
            dg.match_policy(9, seeds, out.data_ptr(), mlp, stream=stream)
        except mm.MatchError as e:
            assert e.status == 4
            return False
        finally:
            debug(mm, ALLOC, -1)
        return True

    with mm.DeviceGraph(g, device=0) as dg:
        dg.prepare(9)
        learned = dg.match_policy(9, seeds, out.data_ptr(), mlp)
        learned_match = out.cpu().numpy()
    # how much memory is enough for the state but not for the features (8 bytes a vertex)
    room = 0
    with mm.DeviceGraph(g, device=0) as dg:
        dg.prepare(9)
        used = debug(mm, USED)
        while debug(mm, USED) == used:
            room += 4 * n
            assert not limited(dg, used + room, 0)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(5):
        with mm.DeviceGraph(g, device=0) as dg:
            dg.prepare(9)
            assert not limited(dg, debug(mm, USED) + room, a.cuda_stream)
            r = dg.match_device(9, seeds, out.data_ptr(), stream=b.cuda_stream)
            assert r == rounds and np.array_equal(out.cpu().numpy(), want)
            assert dg.match_policy(9, seeds, out.data_ptr(), mlp, stream=a.cuda_stream) == learned
            assert np.array_equal(out.cpu().numpy(), learned_match)
