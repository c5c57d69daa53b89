"""The strip kernels' shared memory between the lanes and the copies: an elected
lane's asynchronous copies overwrite rows that all lanes have read and written,
and fence.proxy.async orders only the accesses of the thread that executes it.
A missing fence is a race that a run does not show reliably, so the order is
checked in the source: every elected block that issues copies follows
hand_to_copies(), in which each lane fences its own accesses before the warp
meets, with nothing but the row's bound between the two."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcv_sw_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def test_hand_over_fences_every_lane_before_the_warp_meets():
    body = re.search(r"void hand_to_copies\(\)\s*\{(.*?)\}", source("mcv_strip.cuh"), re.S)
    assert body and body.group(1).split() == ["fence_proxy_async();", "__syncwarp();"]


@pytest.mark.parametrize("name", ["mcv_strip.cuh", "mcv_strip64.cuh"])
def test_every_elected_copy_follows_a_hand_over(name):
    text = source(name)
    blocks = [m.start() for m in re.finditer(r"if \(elect_one\(\)\) \{", text)]
    assert len(blocks) == 3  # a strip's start, the next input rows, the next update's operands
    for at in blocks:
        before = re.sub(r"if \(c < r1\) \{\s*$", "", text[:at].rstrip()).rstrip()
        assert before.endswith("hand_to_copies();"), before[-120:]
