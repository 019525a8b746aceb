"""Rules for the bounded waits of the convolution kernels that no run can show cheaply: a bound takes seconds to run out,
and what it guards against is a fault.  They are checked on the kernels' source text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "excalibur_b200", "csrc")


def _part(name, start, end):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", lambda m: m.group(0) if m.group(0) in (start, end) else "", text)
    a = text.index(start)
    return text[a:text.index(end, a + len(start))]


MMA_ROLES = {
    "conv_tc.cu": ("// ------------------------------- MMA issuer ----------------------------------------",
                   "// ------------------------------- epilogue ------------------------------------------"),
    "conv_split.cu": ("} else if (warp == 1) {", "uint4 res[kSplitMaxItems];"),
}


@pytest.mark.parametrize("name", sorted(MMA_ROLES))
def test_mma_role_waits_for_the_previous_kernel_before_it_polls_for_loads(name):
    """The activations are asked for behind griddepcontrol.wait, so a bounded wait for them that starts before it also
    counts whatever is left of the previous kernel, and gives up when that is long."""
    role = _part(name, *MMA_ROLES[name])
    assert "pdl_wait();" in role
    assert role.index("pdl_wait();") < role.index("full0 +")


@pytest.mark.parametrize("name", sorted(MMA_ROLES))
def test_mma_role_that_gives_up_pauses_for_the_loads_in_flight(name):
    """With a reduction that fits the ring the producer has left by then: nobody else would wait before the shared memory
    becomes the partial tile or another block's."""
    role = _part(name, *MMA_ROLES[name])
    if name == "conv_split.cu":      # no commit either: it would let the epilogue write over the ring
        assert re.search(r"if \(ok\) ptx::tc_commit_u32\(ptx::smem_u32\(&done_bar\), leader\);\s*else ptx::give_up\(", role)
    else:
        assert "if (!ok) ptx::give_up(" in role


def test_giving_up_sets_the_error_word_and_pauses():
    body = _part("ptx_sm100.cuh", "void give_up(", "}\n\n")
    assert re.search(r"atomicExch\(error, code\);\s*for \(int i = 0; i < 2000; \+\+i\) __nanosleep\(100\);", body)
