"""What the bench line says of its CPU baseline: without a build of the reference the
repository's own restatement runs, and the line then neither names the reference's
matcher as what ran nor claims bit-exactness against it."""
from __future__ import annotations

import importlib.util
import json

from test_bench_reference import ROOT, _run


def _bench():
    spec = importlib.util.spec_from_file_location("bench_labels_mod", ROOT / "bench.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_reference_arm_says_what_ran(orc):
    line = json.loads(_run().stdout)
    cb = line["cpu_baseline"]
    assert cb["kind"] == ("reference" if orc.ref_available() else "port")
    assert ("restatement" in cb["runs"]) == (cb["kind"] == "port")


def test_parity_is_claimed_against_what_ran():
    b = _bench()
    cpu = {"parity": True, "valid": True, "maximal": True, "gpu_weight": 2.0, "gpu_size": 4}
    port, ref = b.parity_line({**cpu, "kind": "port"}), b.parity_line({**cpu, "kind": "reference"})
    assert port["bit_exact_vs_reference"] is None and port["bit_exact_vs_restatement"] is True
    assert ref["bit_exact_vs_reference"] is True and ref["bit_exact_vs_restatement"] is None
    assert "matchtbb" not in b.runs_what("port") and "matchtbb" in b.runs_what("reference")
