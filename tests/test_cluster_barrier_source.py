"""The aligned cluster barrier instructions want the whole warp converged, and a
warp that arrives in parts counts wrongly or waits for good, which no test may try
on a device: the check is of the source. Every such instruction has a __syncwarp
in front of it, with nothing in between that could take the lanes apart again."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfdrs_b200", "csrc")


def barrier_lines(path):
    lines = [re.sub(r"//.*", "", s).strip() for s in open(path)]
    lines = [s for s in lines if s]
    return [(lines[i - 1], s) for i, s in enumerate(lines) if re.search(r"barrier\.cluster\.\w+[.\w]*\.aligned", s)]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_aligned_cluster_barriers_behind_syncwarp(path):
    for before, line in barrier_lines(path):
        assert before == "__syncwarp();", (os.path.basename(path), before, line)


def test_the_barriers_are_there():
    assert sum(len(barrier_lines(p)) for p in glob.glob(os.path.join(CSRC, "*.cu*"))) >= 2
