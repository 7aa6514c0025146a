"""The autotuner's baseline is what an untuned graph gets: the pair (0, 0), the
library's own choice, is timed, and a class keeps it unless another pair beats it
clearly; so DeviceGraph.tune_for never pins a pair that is no better than none.  No
device: the timing rows are given."""
from __future__ import annotations

import json

from test_tune_host import ROOT, _rows, _tune


def test_own_choice_is_the_baseline():
    t = _tune()
    assert (0, 0) == t.DEFAULT and 0 in t.FIN_DIVS and 0 in t.BLOCKS
    # a pair that ties with the library's own choice is not pinned, whatever 12 takes
    choice, dflt, wins = t.pick(_rows({(0, 0): 0.796, (24, 2): 0.794, (12, 2): 0.802, (16, 2): 0.80}))
    assert not wins and choice is dflt and (choice["finish_div"], choice["blocks_per_sm"]) == (0, 0)
    # one that beats it clearly is
    choice, dflt, wins = t.pick(_rows({(0, 0): 1.0, (16, 1): 0.9, (12, 2): 1.2}))
    assert wins and (choice["finish_div"], choice["blocks_per_sm"]) == (16, 1) and dflt["ms"] == 1.0


def test_shipped_table_names_the_own_choice_or_a_faster_pair():
    table = json.loads((ROOT / "multicore-matching_b200" / "tuned.json").read_text())
    for name, c in table.items():
        if not (c["finish_div"] == 0 and c["blocks_per_sm"] == 0):
            assert c["ms"] < 0.97 * c["default_ms"], name
