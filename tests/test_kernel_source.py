"""CPU tests of rules that the kernels' source keeps and no healthy run can show."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "e_natten_b200", "csrc")


def scopes_of(text, pattern):
    """(matched text, heads of the braces it lies in) of every match."""
    text = re.sub(r"//[^\n]*", "", text)
    for match in re.finditer(pattern, text):
        heads, start = [], 0
        for i, c in enumerate(text[:match.start()]):
            if c == "{":
                heads.append(text[start:i])
            elif c == "}":
                heads.pop()
            if c in "{};":
                start = i + 1
        yield match.group(), heads


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "na2d_tc_*.cuh"))), ids=os.path.basename)
def test_a_wait_that_decides_a_branch_decides_it_for_its_warp(path):
    """A bounded wait ends in each lane by itself: where a role leaves its loop when one gives up, it is a role of one lane, or
    its lanes vote.  Lanes that part there leave the others at a warp barrier for good."""
    for call, heads in scopes_of(open(path).read(), r"\blt\.acquire(_warp)?\("):
        one_lane = any(re.search(r"\bif \(lane == 0\)\s*$", head) for head in heads)
        assert one_lane == (call == "lt.acquire(")
