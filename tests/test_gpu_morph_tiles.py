"""Opening at the edges of its 128 x 128 tiles and for elements whose rows form long vertical runs,
pairs of single rows or only far radii (each a branch of the centred path); against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _elements():
    def rows(k, widths):  # centred rows of the given widths (0: empty)
        e = np.zeros((k, k), np.uint8)
        for i, w in enumerate(widths):
            if w:
                e[i, k // 2 - w // 2:k // 2 + w // 2 + 1] = 1
        return e

    return {
        "rect15": np.ones((15, 15), np.uint8),
        "vline17": rows(17, [1] * 17),
        "hline63": rows(63, [0] * 31 + [63] + [0] * 31),
        "bars21": rows(21, [21, 0, 21] + [0] * 15 + [21, 0, 21]),
        "cross21": rows(21, [1] * 10 + [21] + [1] * 10),
        "hourglass25": rows(25, [25 - 2 * min(i, 24 - i) for i in range(25)]),
        "rect63": np.ones((63, 63), np.uint8),
    }


@pytest.mark.parametrize("name", list(_elements()))
@pytest.mark.parametrize("shape", [(127, 129), (129, 320), (257, 383)])
def test_elements_at_tile_edges(nsgb, oracle, name, shape):
    rng = np.random.default_rng(shape[0])
    img = rng.integers(0, 256, shape).astype(np.uint8)
    img[rng.random(shape) < 0.6] //= 4
    k = _elements()[name]
    got = nsgb.morphOpen(torch.from_numpy(img).cuda(), k).cpu().numpy()
    assert np.array_equal(got, oracle.morph_open(img, k))
