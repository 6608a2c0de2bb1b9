"""An aligned cluster barrier is undefined for a warp whose lanes have not reconverged, and a loop that lanes leave at
different times does not bring them together by itself: every function of the sources that issues one converges the
warp (__syncwarp) right in front of it."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_aligned_cluster_barrier_converges_its_warp_first():
    seen = 0
    for name in sorted(glob.glob(os.path.join(ROOT, "karume_b200", "csrc", "*.cu*"))):
        with open(name) as fh:
            lines = [line.split("//")[0].strip() for line in fh]
        lines = [line for line in lines if line]
        for at, line in enumerate(lines):
            if re.search(r"barrier\.cluster\.arrive\S*\.aligned", line):
                seen += 1
                assert lines[at - 1] == "__syncwarp();", (os.path.basename(name), line)
    assert seen > 0
