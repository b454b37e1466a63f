"""CPU, by reading the sources: a warp that goes on to warp-collective instructions (tcgen05.ld / st, votes, __syncwarp) may not
leave the loop at a bounded wait with some of its lanes only. In the attention kernels these are the softmax and the
epilogue warps, and the readers of the unit queue that are whole warps: they leave at votes of all lanes."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashomni_b200", "csrc")


@pytest.mark.parametrize("name", ["attention.cu", "attention_streams.cu"])
def test_whole_warps_leave_their_loops_together(name):
    src = open(os.path.join(CSRC, name)).read()
    kernel = src[src.index("} else if (warp >= kWarpEpilogue) {"):src.index("common exit")]
    assert len(re.findall(r"\bmbar_wait\w*\(", kernel)) >= 5
    # no way out of the loop hangs on the outcome of one lane's wait
    for stmt in re.findall(r"if \([^;{]*mbar_wait\w*\([^;{]*[;{]", kernel):
        if "break" in stmt or "return" in stmt or stmt.endswith("{"):
            assert "mbar_wait_all(" in stmt or "__all_sync(" in stmt, stmt
    assert "__all_sync(" in kernel
    reader = src[src.index("struct ItemRead {"):]
    assert re.search(r"kWholeWarp \? mbar_wait_all\(", reader[:reader.index("\n};")])
