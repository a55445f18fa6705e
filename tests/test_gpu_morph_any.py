"""Openings by elements that are not centred runs: dense and sparse random ones of the smallest to the
largest size, single pixels at the ends of a row, gaps wider than a word; against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _elements(k, rng):
    yield "dense", (rng.random((k, k)) < 0.6).astype(np.uint8)
    yield "sparse", (rng.random((k, k)) < 1.5 / k).astype(np.uint8)
    ends = np.zeros((k, k), np.uint8)  # first and last column, first and last row
    ends[0, 0] = ends[k - 1, k - 1] = ends[k // 2, 0] = ends[k // 2, k - 1] = 1
    yield "ends", ends
    one = np.zeros((k, k), np.uint8)
    one[k - 1, 0] = 1
    yield "one corner", one
    yield "diagonal", np.eye(k, dtype=np.uint8)


@pytest.mark.parametrize("k", [3, 5, 7, 9, 11, 19, 33, 61, 63])
@pytest.mark.parametrize("shape", [(5, 3), (127, 129), (130, 261)])
def test_any_element(nsgb, oracle, k, shape):
    rng = np.random.default_rng(k)
    img = rng.integers(0, 256, shape).astype(np.uint8)
    img[rng.random(shape) < 0.6] //= 4
    for name, e in _elements(k, rng):
        if not e.any():
            continue
        got = nsgb.morphOpen(torch.from_numpy(img).cuda(), e).cpu().numpy()
        assert np.array_equal(got, oracle.morph_open(img, e)), name
