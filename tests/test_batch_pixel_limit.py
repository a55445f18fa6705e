"""Workspace sizes of batches at the pixel limit (total pixels below 2^31 - 1): the alignment of the
images in the label planes does not count against it."""
import ctypes as C

import pytest

LIMIT = 2**31 - 1
SIDE = 8191  # odd: images do not end on a multiple of four pixels


def _size(nsgb_ffi, shapes):
    tiles = (nsgb_ffi.Tile * len(shapes))(*[nsgb_ffi.Tile(4096, 8192, h, w, w, 0, 0, 0) for h, w in shapes])
    return nsgb_ffi.lib.nsgb_batch_workspace_size(0, tiles, len(shapes))


@pytest.mark.parametrize("below", [0, 1, 2, 7, 200])
def test_total_just_below_the_limit(below):
    ffi = pytest.importorskip("nsgb._ffi")
    left = LIMIT - below
    shapes = []
    while left >= SIDE * SIDE:
        shapes.append((SIDE, SIDE))
        left -= SIDE * SIDE
    shapes.append((left // SIDE, SIDE))
    if left % SIDE:
        shapes.append((1, left % SIDE))
    assert sum(h * w for h, w in shapes) == LIMIT - below
    assert (_size(ffi, shapes) > 0) == (below > 0)
    assert (_size(ffi, shapes[::-1]) > 0) == (below > 0)
