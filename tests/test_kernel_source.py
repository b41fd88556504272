"""Rules of the kernels' sources that no run on a healthy GPU shows."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "super_gemma_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["attn_prefill_wide.cu", "attn_prefill_int8.cu"])
def test_v_loader_warps_agree_on_a_wait_that_ran_out(name):
    """The V loader is a whole warp that breaks out of its loop, with __syncwarp() inside: every wait of its is voted on."""
    s = _source(name)
    role = s[s.index("warp == V_W"):s.index("warp == MMA_W")]
    assert "__syncwarp" in role and "break" in role
    assert len(re.findall(r"\bmbar_wait_warp\(", role)) == 2 and not re.search(r"\bmbar_wait\(", role)


def test_decode_warps_stop_at_a_wait_that_ran_out():
    """A warp whose copy did not arrive asks for no more (a slot would have two copies under way and its barrier more arrivals
    than it counts), and lets those in flight land before their target is used for the merge or left to another CTA."""
    s = _source("attn_decode_rows.cu")
    waits = re.findall(r"[^\n]*\bmbar_wait(?:_warp)?\([^\n]*", s)
    assert len(waits) == 2 and all(re.search(r"if \(!mbar_wait_warp\(.*\) break;", w) for w in waits)
    assert 0 < s.index("if (failed) let_copies_land();", s.rindex("mbar_wait_warp("))
    s = _source("attn_decode_paged.cu")
    refill = s.index("n_iter && !failed)", s.index("mbar_wait("))
    assert s.index("issue(it + NSTAGES", refill) < s.index("let_copies_land();", refill)


def test_dependent_kernels_read_nothing_as_constant():
    """A kernel that waits for its predecessor (pdl_wait) lives while that one still writes: no ld.global.nc, neither asked for nor
    invited by a const __restrict__ pointer."""
    names = sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh")))
    dependent = [n for n in names if "pdl_wait()" in _source(n)]
    assert len(dependent) >= 6
    for n in names:
        assert not re.search(r"\b__ldg\b|ld\.global\.nc", _source(n)), n
    for n in dependent:
        assert not re.search(r"\bconst\s+[\w ]+\*\s*__restrict__", _source(n)), n


def test_a_failed_launch_is_reported_by_its_own_message():
    """What breaks a launch while recording can end the capture too; the launcher's message must not be lost to that."""
    s = _source("sgb_runtime.cu")
    body = s[s.index("e->fn(a)"):]
    assert body.index("record_after(") < body.index("set_error(r,") < body.index("return recorded")


def test_tensor_memory_is_taken_behind_the_wait_for_the_kernel_before():
    """tcgen05.alloc waits without a limit.  A CTA that holds columns while it waits for its predecessor's end, beside a CTA of the
    predecessor that has yet to allocate, would wait for ever."""
    found = 0
    for n in sorted(os.listdir(CSRC)):
        if not n.endswith(".cu"):
            continue
        for kernel in re.split(r"__global__", _source(n))[1:]:
            if re.search(r"\btmem_alloc(_pair)?\(", kernel) and "pdl_wait()" in kernel:
                assert kernel.index("pdl_wait()") < re.search(r"\btmem_alloc(_pair)?\(", kernel).start(), n
                found += 1
    assert found >= 3


def test_settled_parts_change_hands_over_barriers_of_the_cta():
    """The settled parts of O lie in global memory and go back and forth between two roles of one CTA.  Arrivals on the even CTA's barriers
    order only what the tensor pipe reads, so neither side may rest on them: each waits for a barrier that the other arrives on."""
    s = _source("attn_prefill_int8.cu")
    keys = s[s.index("warp >= SOFT_WARPS && warp < MMA_W"):s.index("warp == V_W")]
    softmax = s[s.rindex("} else {", 0, s.index("const int key0")):]
    assert 0 < keys.index("mbar_wait_warp(&bar.parts_here") < keys.index("fetch_settled(") < keys.index("__threadfence_block()") < keys.index("mbar_arrive(&bar.settle_here)")
    assert "mbar_arrive(&bar.parts_here)" in softmax
    raised = softmax[softmax.index("if (raise)"):]
    wait = re.search(r"if \((.*)\) mbar_wait\(&bar.settle_here", raised)
    assert wait.group(1) == "it >= SETTLE_FROM" and wait.start() < raised.index("fetch_settled(") < raised.index("__threadfence_block()")
    assert raised.index("__threadfence_block()") < raised.index("mbar_arrive(&bar.parts_here)")
