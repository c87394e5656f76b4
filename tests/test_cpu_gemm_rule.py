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


def _split_costs(tiles, kb, c2, c4, c3):
    """k-blocks in a row, by pairs per tile, with the exchange of partial tiles in k-blocks; clusters that the GPU has no room for left out."""
    cost = {1: kb, 2: c2 and -(-tiles // c2) * (-(-kb // 2) + 6), 3: c3 and -(-tiles // c3) * (-(-kb // 3) + 12),
            4: c4 and -(-tiles // c4) * (-(-kb // 4) + 6)}
    return {s: c for s, c in cost.items() if c}


def test_split_takes_the_fewest_k_blocks_in_a_row():
    """Ties go to fewer pairs, but to four where two take the same."""
    for tiles, kb, c2, c4, c3 in itertools.product((1, 3, 8, 16, 18, 19, 32, 37, 38, 64), (4, 7, 8, 9, 12, 16, 32, 33, 41, 128, 129, 1568), (0, 30, 33, 37),
                                                   (0, 12, 15, 16), (0, 20, 22)):
        cost = _split_costs(tiles, kb, c2, c4, c3)
        got = _rule(tiles, kb, 74, c2, c4, c3)
        if 2 * tiles > 74 or kb < 8:
            assert got == 1
        else:
            best = min(cost.values())
            ties = [s for s in cost if cost[s] == best]
            assert got == (4 if ties[0] == 2 and 4 in ties else ties[0]), (tiles, kb, c2, c4, c3)


def test_three_pairs_are_taken_where_four_do_not_fit():
    assert _rule(18, 128, 74, 33, 15, 22) == 3 and _rule(18, 128, 74, 33, 15, 0) == 2 and _rule(18, 128, 74, 33, 15) == 2
    assert _rule(16, 128, 74, 33, 15, 22) == 3 and _rule(16, 128, 74, 33, 16, 22) == 4


def _stream(tiles, kb, pairs=74, c2=33, c4=15, c3=22):
    return native.load().gemm_stream_plan(tiles, kb, pairs, c2, c4, c3)


def test_shared_contraction_is_taken_where_it_is_faster():
    """Launches that took longer than clusters do (256 x 256 from K = 12,288, 512 x 256, 256 x 768, 4096 x 768) stay with clusters; the
    projections of a prompt (K = 100,352, 4 to 24 and 48 tiles) and other long contractions go over all pairs."""
    for tiles, k in ((1, 12288), (1, 16384), (1, 32768), (2, 12288), (2, 16384), (3, 12288), (3, 16384), (8, 16384), (48, 12288), (48, 16384),
                     (32, 100352), (64, 100352)):
        assert not _stream(tiles, k // 64)[0], (tiles, k)
    for tiles, k in ((1, 100352), (2, 32768), (3, 32768), (4, 32768), (8, 32768), (4, 100352), (8, 100352), (12, 100352), (16, 100352),
                     (24, 100352), (48, 100352)):
        assert _stream(tiles, k // 64)[0], (tiles, k)
    assert not _stream(0, 2000)[0] and not _stream(75, 2000)[0] and not _stream(4, 73)[0]
    assert not _stream(16, 1568, c4=16)[0]          # sixteen clusters of four pairs at once are faster


def test_every_k_block_is_taken_once():
    """The pairs of a tile take every per_tile-th of its first k-blocks, the pairs of the tail equal parts of the last ones of all tiles."""
    for pairs, kb in itertools.product((2, 9, 36, 66, 73, 74), (74, 75, 128, 513, 1568)):
        for tiles in range(1, pairs + 1):
            if kb < pairs:
                continue
            _, per_tile, extra, tail = _stream(tiles, kb, pairs)
            assert per_tile >= 1 and per_tile * tiles + extra <= pairs and kb - tail >= per_tile and (tail > 0) == (extra > 0)
            taken = [[0] * kb for _ in range(tiles)]
            for pair in range(per_tile * tiles):
                for k in range(pair // tiles, kb - tail, per_tile):
                    taken[pair % tiles][k] += 1
            for e in range(extra):
                lo, hi = e * tiles * tail // extra, (e + 1) * tiles * tail // extra
                assert hi > lo and (hi - 1) // tail - lo // tail + 1 <= 3       # three partial tiles have a place
                for g in range(lo, hi):
                    taken[g // tail][kb - tail + g % tail] += 1
            assert all(n == 1 for t in taken for n in t), (pairs, kb, tiles)


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


def _few_rows(Z, R, N, K):
    return native.load().skinny_rows(1, K, 1, True, False, False, Z, R, N, K)


def test_few_row_kernel_is_taken_where_it_is_faster():
    """Measured slower there and back with the wide kernel: the second layer of 28 blocks' modulation from three rows on, weights of up to 64
    elements a row with many columns, half-empty lanes. Measured faster with the weights from HBM: the first layer, few columns, calls whose
    reduction the wide kernel splits."""
    for Z, R, N, K in ((84, 3, 6144, 256), (84, 4, 6144, 256), (84, 4, 2048, 256), (84, 4, 256, 64), (84, 1, 768, 8), (84, 2, 6144, 64), (6, 2, 6144, 64),
                       (84, 4, 2048, 512), (28, 2, 3072, 264), (3, 2, 6144, 1032), (28, 1, 6144, 264), (84, 3, 256, 128), (84, 1, 1024, 192)):
        assert not _few_rows(Z, R, N, K), (Z, R, N, K)
    for Z, R, N, K in ((84, 1, 256, 2048), (84, 2, 256, 2048), (84, 4, 256, 2048), (84, 1, 6144, 256), (84, 2, 6144, 256), (1, 1, 4096, 256), (1, 2, 4096, 256), (1, 4, 4096, 256),
                       (1, 4, 256, 2048), (1, 2, 6144, 2048), (84, 4, 64, 2048), (84, 4, 64, 256), (1, 4, 4096, 64), (1, 1, 1, 8), (12, 2, 1024, 520),
                       (84, 2, 768, 1024), (84, 1, 3072, 248), (12, 4, 3072, 2048), (84, 3, 768, 1024)):
        assert _few_rows(Z, R, N, K), (Z, R, N, K)
    ops = native.load()
    assert not ops.skinny_rows(1, 2056, 1, True, False, False, 1, 1, 8, 2056) and not _few_rows(1, 5, 64, 2048)
    assert not ops.skinny_rows(1, 264, 1, True, True, False, 1, 1, 8, 256) and not ops.skinny_rows(2, 256, 1, True, False, False, 1, 1, 8, 256)
    assert not ops.skinny_rows(1, 260, 1, True, False, False, 1, 1, 8, 256) and not ops.skinny_rows(1, 1, 256, True, False, False, 1, 1, 8, 256)
