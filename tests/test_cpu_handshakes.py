"""Models of kernel handshakes whose failure would be a hang: every interleaving of the warps is explored on the CPU."""

import itertools
import pathlib

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "cosmos_predict25_b200" / "ops" / "csrc"


def explore(start, successors):
    """All reachable states, and those from which nothing can happen."""
    seen, todo, stuck = {start}, [start], []
    while todo:
        s = todo.pop()
        nxt = list(successors(s))
        if not nxt:
            stuck.append(s)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return seen, stuck


TILES = 4
ACC, SUM, READ, GONE = range(4)


def _passed(done, n):
    """mbarrier.try_wait on the parity of phase ``n`` when ``done`` phases are complete: it tells neighbouring phases apart only."""
    return (done ^ n) & 1 == 1


def _exchange(bounded):
    """The two epilogue warps of a lane quarter in the convolution with a fused norm. Per tile: wait for the accumulator (bounded: it
    may run out for one warp and not for the other), write the sum of squares into the tile's buffer, meet, read the partner's.
    ``bounded``: they meet at a barrier with a bounded wait (an mbarrier per buffer, two arrivals), else at a named barrier.
    State: tiles finished by the tensor pipe, abort flag, per warp (tile, step), the tile whose sum lies in each warp's two buffers,
    arrivals per warp and buffer."""

    def successors(s):
        ready, abort, warps, bufs, arrived = s
        if ready < TILES:
            yield ready + 1, abort, warps, bufs, arrived
        for i in (0, 1):
            tile, step = warps[i]
            if step == GONE:
                continue
            b = tile & 1

            def to(w, abort=abort, bufs=bufs, arrived=arrived):
                return ready, abort, warps[:i] + (w,) + warps[i + 1:], bufs, arrived

            if step == ACC:
                if ready > tile:                                        # the sum is written and announced
                    nb = tuple(tuple(tile if (j, k) == (i, b) else bufs[j][k] for k in (0, 1)) for j in (0, 1))
                    na = tuple(tuple(arrived[j][k] + ((j, k) == (i, b)) for k in (0, 1)) for j in (0, 1))
                    yield to((tile, SUM), bufs=nb, arrived=na)
                yield to((tile, GONE), abort=1)                          # the limit, or the abort flag, at any moment
            elif step == SUM:
                if bounded:
                    if _passed((arrived[0][b] + arrived[1][b]) // 2, tile >> 1):
                        yield to((tile, READ))
                    yield to((tile, GONE), abort=1)
                elif arrived[1 - i][b] == arrived[i][b] or warps[1 - i][0] > tile:
                    yield to((tile, READ))
            else:
                yield to((tile + 1, ACC) if tile + 1 < TILES else (tile, GONE))

    return (0, 0, ((0, ACC), (0, ACC)), ((-1, -1), (-1, -1)), ((0, 0), (0, 0))), successors


@pytest.mark.parametrize("bounded", [True, False])
def test_exchange_of_sums_between_two_epilogue_warps(bounded):
    seen, stuck = explore(*_exchange(bounded))
    hung = [s for s in stuck if any(w[1] != GONE for w in s[2])]
    if not bounded:
        assert hung, "the model has to show the hang of a named barrier whose partner gave up"
        return
    assert not hung
    for (_, _, warps, bufs, _), i in itertools.product(seen, (0, 1)):
        if warps[i][1] == READ:
            tile = warps[i][0]
            assert bufs[1 - i][tile & 1] == tile, "a warp reads a sum of another tile"


def test_convolution_warps_meet_at_bounded_waits():
    """The convolution kernel is the bounded variant of the model above: no named barrier."""
    assert "bar.sync" not in (CSRC / "conv3d_cl.cu").read_text()
