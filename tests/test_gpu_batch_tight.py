"""Batches whose images lie in the label planes without padding (what a batch within a few pixels of
the limit of 2^31 - 1 gets): the chain's outputs on images that start at no multiple of four pixels.
The layout is made by moving the images in the prepared table."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(33, 65), (1, 97), (97, 1), (7, 11), (64, 131), (129, 31), (1, 1), (200, 303), (5, 5), (45, 1025)]


def _table(ws, tiles):
    """Offset and stride of the image table in a workspace's bytes: images hold their marker's address."""
    raw = ws.tobytes()
    at = [raw.index(np.uint64(t.marker).tobytes()) for t in tiles]
    step = at[1] - at[0]
    assert all(b - a == step for a, b in zip(at, at[1:]))
    return at[0], step


@pytest.mark.parametrize("dtype", ["u8", "i32"])
def test_chain_on_unpadded_images(nsgb, oracle, dtype):
    from nsgb import _ffi, synth

    tiles = [synth.tile_u8(h, w, synth.ellipses_for(h, w), 50 + k) for k, (h, w) in enumerate(SIZES)]
    scale = 1
    if dtype == "i32":
        tiles, scale = [synth.scale(m, dtype) for m, _ in tiles], 1000
    masks = [torch.from_numpy(m).cuda() for m, _ in tiles]
    markers = [torch.from_numpy(k).cuda() for _, k in tiles]
    plan = nsgb.BatchPlan(markers, masks)
    torch.cuda.synchronize()
    structs = [_ffi.Tile(m.data_ptr()) for m in markers]
    host = plan._ws.cpu().numpy()
    start, step = _table(host, structs)
    table = host[start:start + step * len(SIZES)].view(np.int32).reshape(len(SIZES), step // 4)
    px = np.array([h * w for h, w in SIZES])
    padded = np.concatenate([[0], np.cumsum((px + 3) // 4 * 4)[:-1]])
    column = [c for c in range(table.shape[1]) if np.array_equal(table[:, c], padded)]
    assert len(column) == 1  # the first pixel of each image in the label planes
    tight = np.concatenate([[0], np.cumsum(px)[:-1]])
    assert (tight[1:] % 4 != 0).any()
    table[:, column[0]] = tight
    plan._ws.copy_(torch.from_numpy(host))
    nl, nk = plan.chain(thr=128.0 * scale)
    for i, (m, k) in enumerate(tiles):
        exp = oracle.chain(k, m, thr=128 * scale)
        got = {"recon": markers[i], "fill": plan.fill[i], "labels": plan.labels[i], "area": plan.area[i]}
        for name, t in got.items():
            assert np.array_equal(t.cpu().numpy(), exp[name]), (i, SIZES[i], name)
        assert nl[i] == exp["n_labels"] and nk[i] == exp["n_kept"], i
