"""Rules that the tensor-core kernels' sources have to keep so that a stuck call ends with an error (read on the CPU; nothing runs)."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "sentinel_b200", "csrc")


def roles(text):
    """The bodies of a file's warp roles, without comments: what lies between two of the branches that tell warps apart."""
    text = re.sub(r"//[^\n]*", "", text)
    return re.split(r"\n    (?:if \(warp|\} else (?:if \(warp|\{))", text)


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith("_sm100.cu")))
def test_warps_agree_after_bounded_waits_before_they_meet_in_a_named_barrier(name):
    """A named barrier has no limit.  If one warp's wait gives up and another's does not, and the second then stands in a barrier that
    counts the first, neither ever leaves.  So between a wait (or a call that waits) and a named barrier comes named_barrier_all, at
    which all of them learn that one has given up."""
    with open(os.path.join(CSRC, name)) as f:
        bodies = roles(f.read())
    met = 0
    for body in bodies:
        agreed = True
        for token in re.findall(r"\b(?:mbar_wait\w*|get|next|wait|named_barrier_all|named_barrier_sync|push_dq_tile)\b(?=[(<])", body * 2):   # (twice: loops)
            if token == "named_barrier_all":
                met += 1
                agreed = True
            elif token in ("named_barrier_sync", "push_dq_tile"):
                met += 1
                assert agreed, f"{name}: {token} behind a wait that may have given up in one warp alone"
            else:
                agreed = False
    assert met > 0 or name not in ("attn_fwd_sm100.cu", "attn_bwd_sm100.cu")
