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


def _body(text, head):
    """The braces behind `head`, and what they hold."""
    start = text.index("{", text.index(head))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError(head)


@pytest.mark.parametrize("name,remote", [("gemm_tc.cu", "st.shared::cluster"), ("gemm_pair.cu", "mbar_arrive_cluster("),
                                         ("gemm_ts.cu", "ts_exchange<")])
def test_no_cta_leaves_while_another_of_its_cluster_may_address_it(name, remote):
    """Also where a wait has run out: between a kernel's last remote access and the release of its tensor memory stands a
    barrier of the whole cluster, and nothing jumps over it."""
    text = _source(name)
    tail = text[text.rindex(remote):]
    tail = tail[:tail.index("tcgen05.dealloc")]
    assert re.search(r"this_cluster\(\)\.sync\(\)|\bcluster_wait\(\)", tail)
    assert not re.search(r"\b(return|goto)\b", tail)


def test_exchange_arrives_at_the_cluster_barrier_once_behind_its_last_store():
    """gemm_ts: every way through the exchange arrives once - before it waits for what the others send, behind its own stores -
    and only a CTA whose MMAs have completed, and which knows that of the others, stores into them or lets them store."""
    text = _source("gemm_ts.cu")
    body = _body(text, "void ts_exchange(")
    left = _body(body, "if (warp < 3 ||")
    assert re.fullmatch(r"\{\s*cluster_arrive\(\);\s*return;\s*\}", left)
    rest = body[body.index(left) + len(left):]
    assert "return" not in rest and rest.count("cluster_arrive()") == 1
    assert rest.rindex("st.async") < rest.index("cluster_arrive()") < rest.index("&sm.partials, 0")
    stores = rest[:rest.index("cluster_arrive()")]
    assert "send = tc_wait_warp(&sm.peers_done, 0, &sm.abort) && summed;" in stores
    assert re.search(r"for \([^)]*&& send;", stores)
    kernel = _body(text, "gemm_ts_kernel(")
    assert "summed = ok && tc_wait_warp(&sm.accum" in kernel
    assert re.search(r"if \([^)]*\bsummed\b.*\) mbar_arrive_cluster\(cluster_addr\(&sm.peers_done", kernel)
