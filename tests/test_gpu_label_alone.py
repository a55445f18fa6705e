"""Labelling of tiles with many single pixels: around the number from which they are treated apart (256 of
a 32 x 32 tile), singles beside runs that touch them straight or diagonally, several classes, uneven
edges; labels, areas and counts against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(32, 32), (33, 31), (64, 95), (97, 130)]


def _images(h, w, rng):
    y, x = np.arange(h)[:, None], np.arange(w)[None, :]
    grid = ((y % 2 == 0) & (x % 2 == 0)).astype(np.uint8) * 255  # 256 singles of a full tile
    yield "256", grid
    less = grid.copy()
    less[::32, ::32] = 0
    yield "255", less
    bridged = grid.copy()  # some joined to the next column, row or diagonal
    bridged[rng.random((h, w)) < 0.05] = 255
    yield "bridged", bridged
    yield "checkerboard", ((x + y) % 2).astype(np.uint8) * 9
    yield "256 classes", rng.integers(0, 256, (h, w)).astype(np.uint8)
    yield "12 classes", rng.integers(0, 12, (h, w)).astype(np.uint8)
    mixed = rng.integers(1, 200, (h, w)).astype(np.uint8)
    mixed[h // 3:2 * h // 3] = 77  # a run of a whole row between singles
    mixed[:, w // 2] = 78
    yield "mixed", mixed


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("conn", [4, 8])
def test_many_single_pixels(nsgb, oracle, shape, conn):
    for name, img in _images(*shape, np.random.default_rng(shape[0])):
        t = torch.from_numpy(img).cuda()
        for relab in (True, False):
            got, n = nsgb._bwlabel(t, conn, relab)
            exp, exp_n = oracle.bwlabel2(img, conn, relab)
            assert np.array_equal(got.cpu().numpy(), exp) and (n == exp_n or not relab), (name, relab)
        for lo, hi in ((1, 2), (2, 30)):
            got, kept = nsgb.bwareaopen2(t, False, False, lo, hi, conn)
            exp, exp_kept = oracle.bwareaopen2(img, False, False, lo, hi, conn)
            assert kept == exp_kept and np.array_equal(got.cpu().numpy(), exp), (name, lo)
