"""Tile-local labelling on patterns whose runs meet in every way a 32 x 32 tile allows: combs,
spirals, diagonals, checkerboards and noise, at sizes around the tile edge, one class and
several, all connectivities; labels, areas and roots against the CPU oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 70), (70, 1), (31, 33), (32, 32), (33, 31), (64, 96), (65, 97)]


def _patterns(h, w):
    y, x = np.mgrid[0:h, 0:w]
    rng = np.random.default_rng(h * 1000 + w)
    spiral = np.zeros((h, w), bool)
    for r in range(0, max(1, min(h, w) // 2), 2):  # nested rings, each opened at one pixel
        spiral[r, r:w - r] = spiral[h - 1 - r, r:w - r] = True
        spiral[r:h - r, r] = spiral[r:h - r, w - 1 - r] = True
        spiral[min(r + 1, h - 1), r] = False
    yield "comb", (x % 2 == 0) | (y == h - 1)
    yield "comb_up", (x % 2 == 0) | (y == 0)
    yield "comb_rows", (y % 2 == 0) | (x == w - 1)
    yield "diagonals", (x + y) % 3 == 0
    yield "antidiagonals", (x - y) % 3 == 0
    yield "checkerboard", (x + y) % 2 == 0
    yield "rings", spiral
    yield "full", np.ones((h, w), bool)
    yield "empty", np.zeros((h, w), bool)
    for p in (0.3, 0.41, 0.59, 0.9):
        yield f"noise{p}", rng.random((h, w)) < p


@pytest.mark.parametrize("conn", [4, 8])
@pytest.mark.parametrize("shape", SIZES)
def test_label_patterns(nsgb, oracle, shape, conn):
    h, w = shape
    rng = np.random.default_rng(7 * h + w)
    for name, on in _patterns(h, w):
        for img in (np.where(on, 255, 0).astype(np.uint8),
                    (on * rng.integers(1, 4, (h, w))).astype(np.uint8),       # several classes
                    np.where(on, 7, 200).astype(np.uint8)):                   # no background
            t = torch.from_numpy(img).cuda()
            for relab in (True, False):
                got = nsgb.bwlabel2(t, conn, relab).cpu().numpy()
                assert np.array_equal(got, oracle.bwlabel2(img, conn, relab)[0]), (name, relab)
            got, kept = nsgb.bwareaopen2(t, False, False, 2, 40, conn)
            exp, exp_kept = oracle.bwareaopen2(img, False, False, 2, 40, conn)
            assert kept == exp_kept and np.array_equal(got.cpu().numpy(), exp), name


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32])
@pytest.mark.parametrize("shape", SIZES)
def test_two_class_patterns(nsgb, oracle, shape, dtype):
    """Hole fill and labelling in one forest (both classes), for both dual pairs."""
    scale = {np.uint8: 1, np.uint16: 257, np.int32: 1000}[dtype]
    for name, on in _patterns(*shape):
        mask = (np.where(on, 200, 60) * scale).astype(dtype)
        marker = (mask - 10 * scale).astype(dtype)
        for fill_conn, label_conn in ((4, 8), (8, 4)):
            kw = dict(thr=128 * scale, fill_conn=fill_conn, label_conn=label_conn, area_min=2, area_max=200)
            got = nsgb.chain(torch.from_numpy(marker).cuda(), torch.from_numpy(mask).cuda(), **kw)
            exp = oracle.chain(marker, mask, 8, 128 * scale, fill_conn, label_conn, 2, 200)
            for key in ("recon", "fill", "labels", "area"):
                assert np.array_equal(got[key].cpu().numpy(), exp[key]), (name, key)
            assert got["n_labels"] == exp["n_labels"] and got["n_kept"] == exp["n_kept"], name
