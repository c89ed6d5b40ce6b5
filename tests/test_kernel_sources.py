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


def test_stages_released_from_another_cta_are_waited_for_at_the_end():
    """tc_commit_pair arrives on the barriers of both CTAs of a pair.  A producer that waits for a stage only before it
    fills it again leaves the last release of every stage unobserved, and its CTA may be gone when that arrives: behind
    its loop over the tiles it waits for all stages once more."""
    for path in SOURCES:
        with open(path) as f:
            text = f.read()
        if "tc_commit_pair(&empty_bar" not in text:
            continue
        producer = text[text.index("TMA producer\n"):text.index("MMA issuer\n")]
        assert re.search(r"if constexpr\(PAIR\)\s*\{[^{}]*for\([^{}]*S::stages[^{}]*\{[^{}]*mbar_wait_warp\(&empty_bar\[s\]", producer), path
