"""How the insertion kernels give a lock back.  The lane that stores a tet's lock word is
often not the lane that wrote the tet, so the release is: the writes, a warp barrier, then
a fence in every lane and its plain stores, or compare-and-swaps with release ordering.
On a GPU a missed ordering would show as a rare stale read at most, so the source is
checked."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "del3d_b200", "csrc")
STEPS = r"m\.kill|T\.kill|__syncwarp|m\.fence|m\.set|unlock_if"


@pytest.mark.parametrize("name,start,end,order", [
    ("insert_groups.cuh", "// ---- re-star: new tet", "return outcome;", ["m.kill", "__syncwarp", "m.fence", "m.set"]),
    ("build.cu", "// Re-star (as k_restar), reading", "return ok ? AI_DONE : AI_LEAVE;",
     ["T.kill", "__syncwarp", "unlock_if"]),
])
def test_writes_barrier_fence_release(name, start, end, order):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    assert text.count(start) == 1
    part = text[text.index(start):]
    part = re.sub(r"//[^\n]*", "", part[:part.index(end)])
    steps = re.findall(STEPS, part)
    last_write = steps.index(order[0])
    assert not {"m.set", "unlock_if"} & set(steps[:last_write])     # nothing is given back before
    assert steps[last_write:last_write + len(order)] == order
