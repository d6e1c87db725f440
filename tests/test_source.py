"""Rules of the device code that a run cannot show to be kept, read from the sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "polar_b200" / "csrc"


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """An aligned barrier that a diverged warp reaches is undefined, and may hang: every arrival
    is the statement after a __syncwarp, every wait the one after its arrival."""
    seen = 0
    for f in sorted(CSRC.glob("*.cu*")):
        stmts = [s.strip() for s in re.split(r"[;{}]", re.sub(r"//[^\n]*", "", f.read_text()))]
        for i, s in enumerate(stmts):
            if "barrier.cluster.arrive" in s and ".aligned" in s:
                assert stmts[i - 1] == "__syncwarp()", f.name
                seen += 1
            if "barrier.cluster.wait" in s and ".aligned" in s:
                assert "barrier.cluster.arrive" in "".join(stmts[i - 2:i]), f.name
    assert seen
