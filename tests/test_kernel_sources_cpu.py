"""Rules of the kernel sources that no run can be trusted to break: what would go wrong is a matter of how the lanes of a
warp happen to be scheduled, or of where the compiler puts a load."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msa-for-sail_b200", "csrc")


def code(name):
    """Source without comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("name,begin,end", [("fmha_sparse_tc.cu", "const int gt =", "const uint64_t dk_hi")])
def test_warps_wait_as_one(name, begin, end):
    """A role of a tcgen05 kernel is one or more whole warps, each of which goes on as one: a bounded wait is voted on
    (mbar_wait_warp).  The loaders of the sparse kernel: a lane that lagged could miss a phase for good."""
    text = code(name)
    role = text[text.index(begin):text.index(end)]
    assert "mbar_wait_warp(" in role
    assert not re.search(r"\bmbar_wait\(", role)
