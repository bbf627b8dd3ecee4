"""How the kernels' warps wait, as their sources state it."""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).parent.parent / "csrc").rglob("*.cu*"))


@pytest.mark.parametrize("source", SOURCES, ids=lambda p: p.name)
def test_no_lane_waits_for_another(source):
    """A barrier that one lane alone has waited for, joined by a vote, has published nothing to the lane that is elected to issue: votes order no memory."""
    one_lane = re.findall(r"if \(lane == \d+\)\s*\{?\s*(?:\w+ &?= )mbar_wait\(.*", source.read_text())
    assert not one_lane, one_lane
