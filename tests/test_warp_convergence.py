"""CPU checks of the kernels' sources for what a warp-wide operation needs.

A function that holds a full-mask warp intrinsic (peers_of: a match and a
ballot) is one call that all lanes make together: in an arm of a conditional
expression, or behind && or ||, the lanes stand at different call sites and the
result depends on whether the compiler merges them.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "single-clustering_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))

# one call for the whole warp: a match, a ballot or a shuffle with the full mask inside
WARP_CALLS = r"(?:peers_of|__match_any_sync|__reduce_\w+_sync|warp_best|group_best\s*<\s*\w+\s*>)"


def _code(name):
    src = open(os.path.join(CSRC, name)).read()
    src = re.sub(r"/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group(0)), src, flags=re.S)
    return re.sub(r"//[^\n]*", "", src)


def _statement_before(src, at):
    """The statement's text in front of src[at]."""
    return src[max(src.rfind(c, 0, at) for c in ";{}") + 1:at]


def _per_lane_calls(src):
    found = []
    for m in re.finditer(WARP_CALLS + r"\s*\(", src):
        head = _statement_before(src, m.start())
        # only what still encloses the call counts: drop closed parentheses
        while re.search(r"\([^()]*\)", head):
            head = re.sub(r"\([^()]*\)", "", head)
        if re.search(r"\?|&&|\|\|", head):
            found.append(" ".join((head + m.group(0)).split()))
    return found


@pytest.mark.parametrize("name", FILES)
def test_warp_wide_calls_stand_outside_conditional_expressions(name):
    assert _per_lane_calls(_code(name)) == []


def test_the_check_sees_a_call_in_an_arm():
    assert _per_lane_calls("{ m = ok ? peers_of(c, ok) & g : peers_of(c, ok); }")
    assert _per_lane_calls("{ if (a(b) && __match_any_sync(F, c)) x(); }")
    assert not _per_lane_calls("{ m = peers_of(c, x ? 1 : 0); n = ok ? m : 0; }")
    assert not _per_lane_calls("{ const unsigned same = __match_any_sync(F, key); }")
