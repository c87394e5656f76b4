"""The rule that cuts a GEMM's contraction over clusters of CTA pairs (host code of the extension)."""

import itertools

import pytest

from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.skipif(not native.available(), reason="the extension is not built")


def _rule(*a):
    return native.load().gemm_pairs_per_tile(*a)


def test_split_needs_room_for_its_clusters():
    """A share of a GPU that has no room for a cluster of four or eight CTAs takes what is left."""
    for tiles, kb in itertools.product((1, 8, 16, 37), (8, 32, 128, 1568)):
        assert _rule(tiles, kb, 74, 0, 0) == 1
        assert _rule(tiles, kb, 74, 37, 0) in (1, 2) and _rule(tiles, kb, 74, 0, 18) in (1, 4)
    assert _rule(16, 32, 74, 37, 0) == 2 and _rule(16, 32, 74, 0, 18) == 4


def test_split_takes_the_fewest_k_blocks_in_a_row():
    for tiles, kb, c2, c4 in itertools.product((1, 3, 8, 16, 19, 32, 37, 38, 64), (4, 7, 8, 9, 12, 16, 32, 33, 128, 1568), (30, 36, 37), (12, 16, 18)):
        cost = {1: kb, 2: -(-tiles // c2) * (-(-kb // 2) + 6), 4: -(-tiles // c4) * (-(-kb // 4) + 6)}
        got = _rule(tiles, kb, 74, c2, c4)
        if 2 * tiles > 74 or kb < 8:
            assert got == 1
        else:
            assert cost[got] == min(cost.values()) and not (got > 1 and cost[1] == cost[got]) and not (got == 2 and cost[4] == cost[2])


def test_launches_of_several_weights():
    """One launch from 256 rows on while CTA-pair tiles are on, else one for each weight."""
    ops = native.load()
    was = ops.gemm_pair_mode(1)
    try:
        assert [ops.gemm_group_launches(m, 3) for m in (8, 255, 256, 5000)] == [3, 3, 1, 1]
        ops.gemm_pair_mode(0)
        assert [ops.gemm_group_launches(m, 2) for m in (8, 255, 256, 5000)] == [2, 2, 2, 2]
    finally:
        ops.gemm_pair_mode(was)
