"""The tensor-core contractions give up a wait after a limit.  Every role of the block then ends its own loop, and one
that had nothing left to wait for ends as if nothing had happened, so the block itself waits for the copies and MMAs
in flight after its last barrier, before it frees TMEM and its shared memory.  A wait that gives up cannot be brought
about in the built kernels, so the sources are read."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amber_b200", "csrc")


@pytest.mark.parametrize("name,full,commit", [("contract_i8.cu", "st_full", "umma_commit_bar"),
                                              ("contract_tc.cu", "b_full", "umma_commit")])
def test_block_drains_after_its_last_barrier(name, full, commit):
    src = open(os.path.join(CSRC, name), encoding="utf-8").read()
    end = src[:src.index("tcgen05.dealloc")]
    end = end[end.rindex("fence_before();"):]
    m = re.search(r"__syncthreads\(\);\s*if \(\*abort_flag\) \{(.*)__syncthreads\(\);", end, re.S)
    assert m, "no drain between the last barrier and the release of TMEM"
    assert re.search(r"warp == WARP_TMA.*WAIT_LIMIT && !mbar_try_wait\(&" + full, m[1], re.S)
    assert re.search(r"warp == WARP_MMA.*" + commit + r"\(.*WAIT_LIMIT && !mbar_try_wait\(d", m[1], re.S)
