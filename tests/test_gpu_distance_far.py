"""Distance transform with far pixels: around 32 words of rows (where the column pass changes), 128-row
chunks and the number of near tiles from which fewer threads work on each; rows whose far pixels are few,
in the middle of near ones; bit for bit against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _masks(h, w, rng):
    noise = np.where(rng.random((h, w)) < 0.02, 0, 255).astype(np.uint8)
    hole = noise.copy()  # near rows with a far disk in them, over a chunk's end
    y, x = np.arange(h)[:, None], np.arange(w)[None, :]
    hole[(y - min(h - 1, 128)) ** 2 + (x - w // 2) ** 2 < 60 ** 2] = 255
    yield "far disk", hole
    sparse = np.full((h, w), 255, np.uint8)
    sparse[37::90, 11::90] = 0
    yield "sparse", sparse
    ends = np.full((h, w), 1, np.uint8)  # columns with zeros at their ends only, and columns without any
    ends[0, ::3] = 0
    ends[h - 1, 1::3] = 0
    yield "ends", ends
    top = noise.copy()
    top[h // 2:] = 255
    yield "top half", top


@pytest.mark.parametrize("shape", [(127, 90), (128, 513), (129, 129), (1023, 70), (1024, 65), (1025, 64), (1157, 200),
                                   (320, 3905)])
@pytest.mark.parametrize("basins", [False, True])
def test_far_pixels(nsgb, oracle, shape, basins):
    rng = np.random.default_rng(shape[0] + shape[1])
    for name, m in _masks(*shape, rng):
        got = nsgb.distanceTransform(torch.from_numpy(m).cuda(), basins=basins).cpu().numpy()
        assert np.array_equal(got, oracle.distance_transform(m, basins=basins)), name
