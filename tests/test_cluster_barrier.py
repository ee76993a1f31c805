"""The cluster barrier's halves stand behind loops that a warp's lanes leave at
different times, so they are the unaligned forms (the aligned ones are undefined
for a diverged warp)."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_aligned_cluster_barrier():
    found = 0
    for path in glob.glob(os.path.join(ROOT, "codesthesis_dir_gb300", "csrc", "*.cu*")):
        for m in re.finditer(r'"(barrier\.cluster\.[^"]*)"', open(path).read()):
            found += 1
            assert "aligned" not in m.group(1), (os.path.basename(path), m.group(1))
    assert found == 2
