"""Instructions of a whole warp in the CUDA sources stand where all its lanes come by: a lane that asks a barrier or a word in shared
memory gets an answer of its own, so what depends on the answer has to be decided by a vote."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nfai_b200", "csrc")
LANE_WISE = re.compile(r"\b(bar_try|bar_try_cluster|bar_wait|bar_wait_cluster|dead)\s*\(")
VOTE = re.compile(r"\b__(all|any)_sync\s*\(")
WHOLE_WARP = re.compile(r"_sync\s*\(\s*0xffffffff|__syncwarp\s*\(|\belect_one\s*\(|\btmem_(ld|st|st_wait)\s*\(|\bwarp_wait(_cluster)?\s*\(|\.sync\.aligned")


def closing(text, at, pair):
    """Index of the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError(f"unbalanced at {at}")


def plain(text):
    """Without comments (asm strings stay: they hold instructions of a whole warp)."""
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def outside_votes(condition):
    for m in list(VOTE.finditer(condition))[::-1]:
        condition = condition[:m.start()] + condition[closing(condition, m.end() - 1, "()") + 1:]
    return condition


def lane_wise_branches(text):
    """(condition, what it controls) of every branch or loop whose condition a lane answers for itself."""
    for m in re.finditer(r"\b(if|while|for)\s*(constexpr\s*)?\(", text):
        end = closing(text, m.end() - 1, "()")
        condition = text[m.end():end]
        if m.group(1) == "for":
            condition = condition.split(";", 2)[1] if condition.count(";") >= 2 else ""
        if not LANE_WISE.search(outside_votes(condition)):
            continue
        at = end + 1
        while text[at].isspace():
            at += 1
        last = closing(text, at, "{}") if text[at] == "{" else text.index(";", at)
        yield condition, text[at:last + 1]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_no_whole_warp_instruction_behind_a_lanes_own_answer(name):
    with open(os.path.join(CSRC, name)) as f:
        text = plain(f.read())
    for condition, body in lane_wise_branches(text):
        assert not WHOLE_WARP.search(body), f"{name}: {condition.strip()} decides lane by lane on {body.strip()[:200]}"


def test_the_scan_sees_both_shapes():
    loop = "for (uint32_t k = 0; k < end && dead(sh) < 2; ++k) { if (elect_one()) go(); }"
    branch = "if (!bar_try(full, turn)) { wait(); if (__any_sync(0xffffffffu, dead(sh) >= 2)) return; }"
    voted = "if (!__all_sync(0xffffffffu, bar_try(full, turn))) { wait(); if (__any_sync(0xffffffffu, dead(sh) >= 2)) return; }"
    found = [any(WHOLE_WARP.search(body) for _, body in lane_wise_branches(t)) for t in (loop, branch, voted)]
    assert found == [True, True, False]
