"""Rules of the kernels' source that no run can show without a hang or a race: read from the text."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eet_b200", "csrc")


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name", ["gemm_tc.cu", "gemm_pair.cu"])
def test_warps_whose_wait_ran_out_join_the_barrier_of_the_epilogue(name):
    """Between a tile's loop over its k-blocks and epi_bar_or, a barrier that counts all 256 threads of the transform
    warps, nothing may leave: a warp that gives up there would keep the warps that finished their loop waiting for ever.
    And the waits in that loop answer a whole warp alike, so that no warp arrives in two parts."""
    text = _source(name)
    role = text[text.index("const int lane_base = (warp & 3) * 32;"):]
    at = role.index("epi_bar_or(")
    depth, body_end = 0, None
    start = role.index("{", role.index("for (int kb = "))
    for i in range(start, at):
        depth += {"{": 1, "}": -1}.get(role[i], 0)
        if depth == 0:
            body_end = i
            break
    assert body_end is not None, "the loop over the k-blocks encloses the barrier"
    assert not re.search(r"\b(break|return|continue|goto)\b", role[body_end:at])
    waits = re.findall(r"\btc_wait\w*\(", role[start:at])
    assert len(waits) == 3 and set(waits) == {"tc_wait_warp("}


@pytest.mark.parametrize("name", ["gemm_row.cu", "gemm_skinny.cu"])
def test_what_the_preceding_kernel_writes_is_not_read_as_constant(name):
    """These kernels begin before the one in front of them has ended.  __ldg promises that nobody writes the memory during the
    kernel's lifetime: true of weights, scales and norm weights, not of what is read behind pdl_wait."""
    text = _source(name)
    assert "__ldg" not in text[text.index("pdl_wait();"):]


@pytest.mark.parametrize("name,push", [("attention.cu", "map_shared_rank("), ("gemm_row.cu", "st.shared::cluster"),
                                       ("gemm_tc.cu", "st.shared::cluster")])
def test_no_store_into_another_cta_before_it_is_known_to_run(name, push):
    """A CTA may write another's shared memory only once that one has begun: a cluster barrier comes first."""
    text = _source(name)
    before = text[:text.index(push)]
    assert "barrier.cluster.wait" in before or "this_cluster().sync()" in before
