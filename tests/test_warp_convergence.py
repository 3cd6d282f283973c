"""CPU checks of the kernels' sources for what a warp-wide operation needs.

A function that holds a full-mask warp intrinsic (peers_of: a match and a
ballot) is one call that all lanes make together: in an arm of a conditional
expression, or behind && or ||, the lanes stand at different call sites and the
result depends on whether the compiler merges them.

A load from tensor memory (tmem_ld8, tmem_ld64: tcgen05.ld.sync.aligned) needs
its warp converged: in the block of code that makes it, a warp-wide operation
stands in front of it, whatever the lanes did in the round before. A barrier
written as PTX (bar.sync, barrier.cluster.arrive / wait with .aligned) needs the
same.

The flag that ends the kNN scan early is read by a whole warp (__any_sync) where
its lanes go on to warp-wide operations: lanes that read it one by one could part
there, and some would wait for the others.
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


def _block_before(src, at):
    """The text of the innermost block around src[at] up to there, without the blocks closed in it."""
    depth, i, text = 0, at - 1, []
    while i >= 0:
        c = src[i]
        if c == "}":
            depth += 1
        elif c == "{":
            if depth == 0:
                return "".join(reversed(text))
            depth -= 1
        elif depth == 0:
            text.append(c)
        i -= 1
    return "".join(reversed(text))


def _unconverged_loads(src):
    found = []
    for m in re.finditer(r"\btmem_ld(?:8|64)\s*\(", src):
        if re.search(r"\bvoid\s+$", src[:m.start()]):
            continue  # its definition
        if not re.search(r"__syncwarp\s*\(|__(?:all|any|ballot)_sync\s*\(", _block_before(src, m.start())):
            found.append(src.count("\n", 0, m.start()) + 1)
    return found


@pytest.mark.parametrize("name", FILES)
def test_tensor_memory_loads_follow_a_warp_wide_operation(name):
    assert _unconverged_loads(_code(name)) == []


def test_the_check_sees_a_load_behind_predicated_stores():
    assert _unconverged_loads("{ __syncwarp(); while (g) { float x[8]; tmem_ld8(a, x); if (x[0] < t) s[0] = x[0]; } }")
    assert not _unconverged_loads("{ while (g) { __syncwarp(); tmem_ld8(a, x); } }")
    assert not _unconverged_loads("{ if (!__all_sync(F, w(b))) { break; } tmem_ld64(a, r); }")


def _unconverged_barriers(src):
    found = []
    for m in re.finditer(r'asm\s+volatile\s*\(\s*"(bar\.sync|barrier\.cluster\.arrive[^"]*\.aligned)', src):
        if not re.search(r"__syncwarp\s*\(", _block_before(src, m.start())):
            found.append(m.group(1))
    return found


@pytest.mark.parametrize("name", FILES)
def test_aligned_barriers_follow_a_warp_barrier(name):
    assert _unconverged_barriers(_code(name)) == []


def test_the_scan_stops_by_the_warp():
    src = _code("sc_knn.cu")
    kernel = src[src.index("k_knn_tc(const __grid_constant__"):]
    kernel = kernel[kernel.index("else if (warp == 1)"):]  # behind the producer, which is one lane
    kernel = kernel[:kernel.index("__syncthreads()")]
    reads = [m.start() for m in re.finditer(r"\*abort_flag(?!\s*=[^=])", kernel)]
    assert reads
    assert all(kernel[:at].endswith("__any_sync(0xFFFFFFFFu, ") for at in reads)
