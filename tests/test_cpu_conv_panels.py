"""How the convolution kernel walks over a list of taps (host code of the extension)."""

import itertools

import pytest

from cosmos_predict25_b200.ops import native

pytestmark = pytest.mark.skipif(not native.available(), reason="the extension is not built")

SQUARE = [(i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)]
_LISTS = {"3x3x3": [(t, i, j) for t in (0, 1, 2) for i, j in SQUARE], "1x3x3": [(0, i, j) for i, j in SQUARE],
          "shuffled": [(t, i, j) for j in (1, -1, 0) for t in (2, 0, 1) for i in (0, 1, -1)], "2x2": [(0, i, j) for j in (0, 1) for i in (-1, 0)],
          "3x1x1": [(t, 0, 0) for t in (0, 1, 2)], "rows": [(0, i, 0) for i in (-1, 0, 1)], "columns": [(0, 0, j) for j in (1, 0, -1)],
          "3x2": [(0, i, j) for i in (-1, 0, 1) for j in (0, 1)], "2x1": [(t, i, 4) for t in (1, 0) for i in (3, 2)], "one": [(0, 1, -2)]}


def _panels(name, cin, n_tile, stride=1):
    taps = _LISTS[name]
    out = native.load().conv_panels([v for t in taps for v in t], stride, cin, n_tile)
    run, cols, n = out[:3]
    assert len(out) == 3 + n * (3 + run * cols)
    panels = [out[3 + g * (3 + run * cols):][:3 + run * cols] for g in range(n)]
    return run, cols, [(p[:3], p[3:]) for p in panels]


@pytest.mark.parametrize("name", sorted(_LISTS))
def test_every_tap_is_read_once_at_its_offset(name):
    for cin, n_tile, stride in itertools.product((16, 32, 96), (16, 32, 192), (1, 2)):
        run, cols, panels = _panels(name, cin, n_tile, stride)
        seen = []
        for (dt, dh, dw), taps in panels:
            for (i, j), k in zip(itertools.product(range(cols), range(run)), taps):
                assert _LISTS[name][k] == (dt, dh + j, dw + i)
                seen.append(k)
        assert sorted(seen) == list(range(len(_LISTS[name])))
        assert [p[0][0] for p in panels] == sorted(p[0][0] for p in panels)   # frames that are all padding are skipped from the front


def test_shapes():
    """Squares share a box; not where a layer has 16 input or output channels, which goes by columns; lists of whole columns do too."""
    for name in ("3x3x3", "1x3x3", "shuffled"):
        assert [_panels(name, *c)[:2] for c in ((96, 96), (384, 192), (96, 32), (32, 16))] == [(3, 3)] * 4
        assert [_panels(name, *c)[:2] for c in ((96, 16), (384, 16), (16, 192), (16, 16))] == [(3, 1)] * 4
        assert _panels(name, 96, 96, 2)[:2] == (1, 1)
    assert [_panels(n, 96, 96)[:2] for n in ("2x2", "3x1x1", "rows", "columns", "3x2", "2x1", "one")] == [(2, 2), (1, 1), (3, 1), (1, 1), (3, 1), (2, 1), (1, 1)]
