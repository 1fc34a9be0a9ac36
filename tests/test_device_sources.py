"""Rules of the device code that its sources show (no GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pandora-2.0_b200", "csrc")


def test_warp_exchanges_name_their_lanes():
    """A shuffle or vote names a fixed set of lanes that all reach it: __activemask() gives the
    lanes that happen to be converged, so inside a branch that parts a warp the lane a value
    comes from need not be among them."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(CSRC, name)).read()
        code = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
        assert "__activemask" not in code, name
