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
