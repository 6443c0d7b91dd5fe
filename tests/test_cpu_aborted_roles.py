"""Roles that meet at a named barrier after a device-side wait has given up.  Such a barrier has no limit of its own, so all warps
of the role have to come to it equally often whatever their waits returned: one warp reads the work item for all of them.  Checked
here on a model of the hand-over, and by reading that the kernels do it."""
import itertools
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pku-aiprogramming_b200", "csrc")
WARPS, TILES = 4, (2, 1, 3)     # tiles per work item, two barriers each


def arrivals(gives_up_at, one_reads):
    """How often each warp comes to the barrier when its wait for item gives_up_at[warp] is its first that fails."""
    if one_reads:   # warp 0: a barrier behind every read, and what it read counts for all
        n = gives_up_at[0]
        return [n + 1 + 2 * sum(TILES[:n])] * WARPS
    return [2 * sum(TILES[:n]) for n in gives_up_at]


def test_an_abort_leaves_no_warp_at_the_barrier():
    every = list(itertools.product(range(len(TILES) + 1), repeat=WARPS))
    assert any(len(set(arrivals(w, False))) > 1 for w in every)      # each on its own: some would wait for the others for good
    assert all(len(set(arrivals(w, True))) == 1 for w in every)


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.mark.parametrize("name,role,barrier,reader", [
    ("attn_bwd_fused_sm100.cu", "the adding warpgroup: dQ_t out of tensor memory", "named_bar_sync(1, 128)", 8),
    ("attn_decode_gq_sm100.cu", "softmax: thread = key of the tile", "bar_sync_128(1)", 0)])
def test_one_warp_reads_the_item_for_its_role(name, role, barrier, reader):
    src = source(name)
    loop = src.index("for (int", src.index(role))
    head = src[loop:src.index(barrier, loop)]       # from the top of the item loop to its first barrier
    assert re.search(r"if \(warp == %d\) \{[^}]*next_item\(" % reader, head), head
    assert "take_item(" not in head and head.count("next_item(") == 1


@pytest.mark.parametrize("name", ["attn_bwd_fused_sm100.cu", "attn_decode_gq_sm100.cu", "attn_fwd_sm100.cu", "attn_bwd_sm100.cu",
                                  "attn_fwd_pair_sm100.cu", "attn_bwd_pair_sm100.cu"])
def test_a_warp_takes_or_leaves_an_item_as_one(name):
    src = source(name)
    body = src[src.index("auto next_item ="):]
    body = body[:body.index("};")]
    assert re.search(r"__all_sync\(0xffffffffu, (mbar_wait|ok)", body)
    if "kVoteHere" in body:      # some instantiations leave it to the two roles that call
        assert src.count("if (kVoteHere ? item < 0 : __any_sync(0xffffffffu, item < 0)) break;") == 2


@pytest.mark.parametrize("name", ["attn_bwd_fused_sm100.cu", "attn_fwd_sm100.cu"])
def test_the_loader_leaves_a_slot_alone_that_was_not_released(name):
    """These two publish a packed item's geometry beside its number: half of it overwritten would name rows of another sequence."""
    src = source(name)
    at = src.index("if (kVarlen) packed[slot] = pi;")
    wait = src.rindex("mbar_wait(&bar_sched_empty[slot]", 0, at)
    assert re.search(r"if \(!__all_sync\(0xffffffffu, mbar_wait\(&bar_sched_empty\[slot\].*\) break;", src[wait - 40:at])
