"""Rules of the CUDA sources that no run shows reliably, checked on the text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blind-spiking-lstm_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))


def code(name):
    """A source without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


@pytest.mark.parametrize("name", SOURCES)
def test_warp_collectives_name_their_lanes(name):
    """__activemask() says which lanes happen to be converged, not which have to
    take part: a vote, shuffle or __syncwarp over it may run in parts."""
    assert "__activemask" not in code(name)


@pytest.mark.parametrize("name", ["ks_tc.cu", "lstm_linear.cuh"])
def test_launches_follow_the_devices_sm_count(name):
    """Tiles, parts and grids are chosen for the SMs there are (148 on a B200)."""
    assert not re.search(r"\b(148|296)(LL)?\b", code(name))
