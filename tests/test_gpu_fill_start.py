"""Grayscale hole filling from an estimated level (sides of 1280 and more): images whose level is
found at once, after others, or not at all give the oracle's fill, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

H, W = 1291, 1407


def _image(kind, dtype, rng):
    lo, hi = {np.uint8: (0, 255), np.uint16: (0, 65535), np.int32: (-2**31, 2**31 - 1)}[dtype]
    scale = {np.uint8: 1, np.uint16: 257, np.int32: 1000}[dtype]
    if kind == "noise":  # few levels, dark objects
        img = rng.integers(185, 216, (H, W))
        img[rng.random((H, W)) < 0.1] = 50
        return (img * scale).astype(dtype)
    if kind == "two_levels":
        return (np.where(rng.random((H, W)) < 0.55, 40, 200) * scale).astype(dtype)
    if kind == "many_levels":  # no level is shared
        return rng.integers(lo, hi, (H, W), endpoint=True).astype(dtype)
    if kind == "constant":
        return np.full((H, W), hi if rng.random() < 0.5 else lo, dtype)
    if kind == "slope":  # the level rises along the image
        return ((np.arange(W)[None, :] * 60 // W + rng.integers(100, 120, (H, W))) * scale).astype(dtype)
    img = rng.integers(100, 131, (H, W))  # "walls": closed boxes of several heights
    for k, v in enumerate(range(140, 240, 20)):
        a = 100 + 90 * k
        img[a:H - a, a] = img[a:H - a, W - 1 - a] = v
        img[a, a:W - a] = img[H - 1 - a, a:W - a] = v
    return (img * scale).astype(dtype)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32])
@pytest.mark.parametrize("kind", ["noise", "two_levels", "many_levels", "constant", "slope", "walls"])
def test_fill_matches_oracle(nsgb, oracle, kind, dtype):
    rng = np.random.default_rng(len(kind))
    img = _image(kind, dtype, rng)
    for conn in (4, 8):
        got = nsgb.imfillHoles(torch.from_numpy(img).cuda(), False, conn).cpu().numpy()
        assert np.array_equal(got, oracle.imfill_holes(img, False, conn)), conn
