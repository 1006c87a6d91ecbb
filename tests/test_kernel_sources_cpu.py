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


@pytest.mark.parametrize("name", ["fmha_tc.cu", "fmha_sparse_tc.cu", "fmha_decode_tc.cu"])
def test_warps_wait_as_one(name):
    """A role of a tcgen05 kernel is one or more whole warps, each of which goes on as one: every bounded wait is voted on
    (mbar_wait_warp).  A lane that lagged in a wait of its own could miss a phase for good; one that gave up alone would
    leave the others in a warp-wide instruction."""
    text = code(name)
    assert "mbar_wait_warp(" in text
    assert not re.search(r"\bmbar_wait\(", text)
    assert not re.search(r"&& \*abort_flag", text)           # the other way out of a loop: read by each lane, decided by the warp


@pytest.mark.parametrize("name", ["fmha_tc.cu", "fmha_sparse_tc.cu", "fmha_decode_tc.cu"])
def test_a_timeout_outlasts_the_copies_in_flight(name):
    """After a wait gave up, shared memory and TMEM are given back only once nothing that was issued can still land there."""
    end = code(name).rsplit("if (*abort_flag) {", 1)[1]
    assert end.index("outlast_async_work();") < end.index("tmem_dealloc(")


def test_sparse_loader_leaves_before_the_wait():
    """A loader warp without a unit in the last chunk of a list may not wait for that chunk's buffer (the phase it waits for
    can be over by then).  That the condition is right for every group size and chunk is asserted when the file is compiled."""
    loop = code("fmha_sparse_tc.cu").split("int ent = entry_of(0);")[1]
    leave = loop.index("if (!loader_has_unit(warp - GATHER_WARP0, upt, min(tpc, item.z - (item.y + c * tpc)))) break;")
    assert leave < loop.index("mbar_wait")


@pytest.mark.parametrize("name", sorted(n for n in os.listdir(CSRC) if n.endswith(".cu")))
def test_chained_kernels_wait_and_read_coherently(name):
    """A kernel launched with launch_chained() is up while the one before it still writes: it waits with chain_begin(), and
    reads global memory in no way that takes the data to be constant during the kernel."""
    text = code(name)
    kernels = text.split("__global__")[1:]
    if "launch_chained(" in text:
        assert kernels and all("chain_begin();" in k for k in kernels)
        for k in kernels:
            assert not re.search(r"__restrict__|__ldg\b|\.nc\b", k)
