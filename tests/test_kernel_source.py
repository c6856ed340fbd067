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


def test_box_loads_over_ordinary_stores_come_behind_a_fence():
    """The second halo of the box kernels lands where their row maxima and sums were written with ordinary stores; only a proxy fence
    of the threads that wrote them orders those before the copy (the count of the warps does not)."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "na2d_box.cuh")).read())
    places = [m.start() for m in re.finditer(r"\bloads\.last\(3\)", text)]
    assert len(places) == 2                                       # fwd_kernel, dq_kernel
    for at in places:
        assert re.search(r"fence_proxy_async\(\);\s*if \($", text[:at])


@pytest.mark.parametrize("name", ["na2d_box.cuh", "na2d_box_key.cuh"])
def test_box_loads_stop_when_a_wait_has_given_up(name):
    """Loads::expect says whether a load may still start (no wait of the thread that asks has given up, and so the barrier's last phase is
    over); no barrier is armed and no load issued without asking it."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    asked = re.findall(r"(if \()?uint64_t\* bar = loads\.expect\([^;{]*?\)(\)|;\s*if \(!bar\) return;)", text)
    assert len(asked) == len(re.findall(r"\bexpect\(", text)) - text.count("uint64_t* expect(") > 0
    assert all((before == "if (") == (after == ")") for before, after in asked)
    assert all("bar" in call.split(",")[2] for call in re.findall(r"tma_load_5d\(([^;]*)\);", text))
    for call, heads in scopes_of(text, r"mbar_expect_tx\("):
        assert "uint64_t* expect(" in heads[-1]
        assert re.search(r"if \(gave_up\) return nullptr;\s*na2d_ptx::$", text[:text.index(call)])
