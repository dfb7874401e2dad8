"""CPU checks of rules that the kernels' sources keep and that no run on a GPU shows reliably."""
import glob
import os

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "webgpt_b200", "csrc", "*.cu*")))


def test_cluster_barriers_are_reached_by_whole_warps():
    """The .aligned forms of barrier.cluster want all lanes of a warp together; a branch on tid just before does not promise
    that, so each is issued right behind a __syncwarp() (or behind another barrier.cluster)."""
    found = 0
    for path in SOURCES:
        lines = open(path).read().splitlines()
        for i, line in enumerate(lines):
            if 'asm volatile("barrier.cluster.' in line:
                found += 1
                assert "__syncwarp();" in lines[i - 1] or "barrier.cluster." in lines[i - 1], f"{path}:{i + 1}"
    assert found >= 5
