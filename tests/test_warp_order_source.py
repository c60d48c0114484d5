"""One lane often signals for its whole warp: it arrives on a barrier for what all lanes wrote or read, or issues MMAs on data that other
lanes' waits have seen.  A vote (`__all_sync`) is no memory barrier, `__syncwarp()` is; no run on the GPU can be relied on to show a missing
one.  Checked here by reading the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "train_gpt_b200", "csrc")
FILES = ["gemm_fp8.cu", "gemm_ring.cu", "gemm_skinny.cu"]


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", " ", text, flags=re.S))


@pytest.mark.parametrize("name", FILES)
def test_a_warps_arrival_follows_its_syncwarp(name):
    text = _source(name)
    calls = [m.start() for m in re.finditer(r"\bmbar_arrive(?:_cluster)?_if\((?!uint32_t)", text)]
    assert calls
    marks = [(m.start(), m.group()) for m in re.finditer(r"__syncwarp\(\);|__all_sync\(|\bmbar_wait\(|cp\.async|cp_async_4\(|\btmem_wait_ld\w*\(", text)]
    for at in calls:
        assert [what for where, what in marks if where < at][-1] == "__syncwarp();", text[max(0, at - 300):at + 60]


@pytest.mark.parametrize("name", FILES)
def test_lanes_that_wait_for_different_barriers_meet_before_the_issue(name):
    text = _source(name)
    waits = [m.end() for m in re.finditer(r"__all_sync\(0xffffffffu, mbar_wait\([^;]*stage_lane[^;]*;", text)]
    assert waits
    for at in waits:
        assert "__syncwarp();" in text[at:text.index("elect_one()", at)], text[at - 200:at + 100]
