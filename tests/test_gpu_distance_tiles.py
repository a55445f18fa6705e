"""Distance transform around the near pass's tiles (32 rows x 128 columns, 32 columns of halo):
distances of 31 .. 34 in every direction, rows of the near and of the far pass in one image, odd
sizes, unaligned rows; bit for bit against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _masks(h, w, rng):
    yield "all zero", np.zeros((h, w), np.uint8)
    one = np.full((h, w), 255, np.uint8)
    one[h // 2, w // 2] = 0
    yield "one zero", one
    grid = np.full((h, w), 7, np.uint8)
    grid[::65, ::65] = 0  # up to 32 in each direction: the last exact offset
    yield "grid 65", grid
    grid = np.full((h, w), 1, np.uint8)
    grid[::67, ::63] = 0
    yield "grid 67 63", grid
    half = np.where(rng.random((h, w)) < 0.02, 0, 255).astype(np.uint8)
    half[:, w // 2:] = 255  # near rows, far pixels in the same rows
    yield "half", half
    yield "noise", np.where(rng.random((h, w)) < 0.5, 0, 128).astype(np.uint8)
    stripes = np.full((h, w), 255, np.uint8)
    stripes[:, ::33] = 0
    stripes[h // 3:h // 2] = 255  # a band whose nearest zeros are above and below
    yield "band", stripes


@pytest.mark.parametrize("shape", [(1, 1), (1, 300), (300, 1), (32, 128), (33, 129), (65, 127), (131, 263), (97, 400)])
@pytest.mark.parametrize("basins", [False, True])
def test_near_and_far_pixels(nsgb, oracle, shape, basins):
    rng = np.random.default_rng(shape[0] + shape[1])
    for name, m in _masks(*shape, rng):
        got = nsgb.distanceTransform(torch.from_numpy(m).cuda(), basins=basins).cpu().numpy()
        exp = oracle.distance_transform(m, basins=basins)
        assert np.array_equal(got, exp), name


def test_unaligned_rows(nsgb, oracle):
    rng = np.random.default_rng(1)
    full = np.where(rng.random((90, 211)) < 0.03, 0, 255).astype(np.uint8)
    t = torch.from_numpy(full).cuda().reshape(-1)
    from nsgb import _ffi
    import ctypes as C

    h, w, pitch, off = 80, 150, 211, 3
    m = full.reshape(-1)[off:off + pitch * h].reshape(h, pitch)[:, :w]
    out = torch.full((h, w + 5), -1.0, dtype=torch.float32, device="cuda")
    need = _ffi.lib.nsgb_workspace_size(_ffi.OP_DISTANCE, _ffi.U8, h, w)
    ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    st = _ffi.lib.nsgb_distance_transform(t.data_ptr() + off, out.data_ptr(), h, w, pitch, (w + 5) * 4, 0,
                                          (ws.data_ptr() + 255) & ~255, need,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    assert st == 0
    got = out.cpu().numpy()
    assert np.array_equal(got[:, :w], oracle.distance_transform(np.ascontiguousarray(m), basins=False))
    assert (got[:, w:] == -1.0).all()
