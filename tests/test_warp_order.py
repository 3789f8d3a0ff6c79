"""Shared memory that one lane of a warp writes and another reads needs a
__syncwarp (or a barrier) in between: votes and shuffles order no memory. The
order holds by chance where a warp's accesses issue in program order, so no run
shows the mistake; this reads the source instead."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sptc-smat_gb300", "csrc")


def code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def between(text, first, second):
    """The text from the only match of `first` to the next match of `second`."""
    starts = list(re.finditer(first, text))
    assert len(starts) == 1, first
    tail = text[starts[0].end():]
    end = re.search(second, tail)
    assert end, second
    return tail[:end.start()]


def test_gather_list_is_ordered():
    part = between(code("spmm_tc.cu"), r"reinterpret_cast<int4\*>\(glist\)\[lane\]\s*=", r"gather_tile<")
    assert "__syncwarp()" in part


def test_row_table_is_ordered():
    part = between(code("spmm_tc.cu"), r"rows\[x \* 32 \+ lane\]\s*=", r"store_rows16<")
    assert "__syncwarp()" in part


def test_warp_wait_orders_the_other_lanes():
    part = between(code("spmm_tc.cu"), r"__device__ __forceinline__ bool warp_wait\(", r"\n}")
    assert "__syncwarp()" in part


def test_roles_wait_for_the_launch_before_ahead_of_their_limits():
    """A kernel launched behind another one starts while that one runs. A role's bounded
    waits must not count it (they are too coarse to see that in a run: the launch
    before would have to take milliseconds with all of its blocks resident)."""
    tc, s24 = code("spmm_tc.cu"), code("spmm24.cu")
    assert "grid_wait();" in between(tc, r"const int ct = \(threadIdx\.x", r"take_item_warp\(")        # converters
    assert "grid_wait();" in between(tc, r"const uint32_t stall =", r"take_item_one\(")                # MMAs
    assert "grid_wait();" in between(s24, r"bool ok = true, issued = false;", r"w24\(")                # MMAs
    part = between(s24, r"bool ok = true, behind = false;", r"!w24_warp\(smem_u32\(&a_free")           # converters
    assert "grid_wait();" in part and part.count("wait_before(") == 2
    stages = between(s24, r"if \(warp == 1\) \{", r"!w24\(smem_u32\(&s_free")                          # stage copies
    assert "grid_wait();" in stages
