"""Rules of the CUDA sources that no run on a GPU can be relied on to show: what breaks them may work by chance."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amdmigraphx_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_cluster_barriers_stand_behind_a_reconvergence(path):
    """barrier.cluster.*.aligned is undefined where the lanes of a warp do not execute it together; after code that
    divided the lanes only __syncwarp() directly in front brings them together again."""
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r'asm volatile\(\s*"[^;]*barrier\.cluster\.', text):
        before = text[:m.start()].rstrip()
        assert before.endswith("__syncwarp();"), text[max(0, m.start() - 100):m.end()]
