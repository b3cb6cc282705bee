"""Rules of the kernels' inline PTX that no run shows."""

from __future__ import annotations

import re

import pytest
from conftest import ROOT

SOURCES = sorted((ROOT / "acoustic_spaces_b200" / "csrc").glob("*.cuh"))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_barriers_do_not_assume_a_converged_warp(path):
    """The aligned form of a barrier is undefined where a warp's threads reach it apart, and the steps' loops end lane
    by lane."""
    assert not re.findall(r"barrier\.[\w.:]*\.aligned", path.read_text())
