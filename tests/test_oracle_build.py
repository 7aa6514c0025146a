"""The oracle's two layers are told apart when one is missing: the reference's own
build may be absent (its tests skip), the restatement may not."""
from __future__ import annotations

from pathlib import Path

import pytest


def test_missing_reference_build_is_its_own_error(orc):
    with pytest.raises(orc.ReferenceNotBuilt):
        orc._load(Path(orc.__file__).parent / "_ref" / "no_such.so", {})
    with pytest.raises(OSError) as e:
        orc._load(Path(orc.__file__).parent / "no_such.so", {})
    assert not isinstance(e.value, orc.ReferenceNotBuilt)


def test_reference_tests_skip_without_the_build(orc):
    if orc.ref_available():
        pytest.skip("the reference's build is here")
    with pytest.raises(orc.ReferenceNotBuilt):
        orc.ref_lib()
