"""The grayscale hole fill's start on images of several kinds: the fill is the oracle's, bit for bit, and no
level is labelled where the image has none of its own, or where a wall closes it off (labelling the
image for nothing made a fill up to 2.6 times as long).  The control words of the start stay in the last region of the workspace."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SCALE = {np.uint8: 1, np.uint16: 257, np.int32: 1000}
BAND = 3  # index of the band among the labellings; 0 .. 2 are the levels


def _image(kind, h, w, rng):
    noise = rng.integers(185, 216, (h, w))
    noise[rng.random((h, w)) < 0.1] = 50
    y, x = np.arange(h)[:, None], np.arange(w)[None, :]
    if kind == "noise":
        return noise
    if kind in ("frame", "rim"):  # a bright border, one pixel or many
        t = 1 if kind == "frame" else h // 9
        img = noise // 2
        img[:t] = img[h - t:] = 240
        img[:, :t] = img[:, w - t:] = 240
        return img
    if kind == "surround":  # bright noise around a dark noisy disk
        r = (y / h - 0.5) ** 2 + (x / w - 0.5) ** 2
        return np.where(r > 0.16, rng.integers(236, 245, (h, w)), noise // 2)
    if kind == "slope":
        return x * 150 // w + rng.integers(20, 51, (h, w))
    if kind == "many":
        return rng.integers(0, 256, (h, w))
    a = 100  # "wall": a closed wall between the outermost crops and the next
    noise[a:h - a, a] = noise[a:h - a, w - 1 - a] = 250
    noise[a, a:w - a] = noise[h - 1 - a, a:w - a] = 250
    return noise


def _fill(img, conn):
    """The fill and which labellings its start made."""
    from nsgb import _ffi

    h, w = img.shape
    dt = {np.dtype(np.uint8): 0, np.dtype(np.uint16): 1, np.dtype(np.int32): 2}[img.dtype]
    need = _ffi.lib.nsgb_workspace_size(_ffi.OP_FILL_HOLES, dt, h, w)
    ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    base = (ws.data_ptr() + 255) & ~255
    src = torch.from_numpy(img).cuda()
    out = torch.empty_like(src)
    st = _ffi.lib.nsgb_imfill_holes(dt, src.data_ptr(), out.data_ptr(), h, w, w * img.itemsize, 0, conn, base, need,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    assert st == 0
    at = base - ws.data_ptr() + need - (h * w + 255) // 256 * 256
    go = ws[at:at + 16].cpu().numpy().view(np.int32)
    return out.cpu().numpy(), [k for k in range(4) if go[k]]


# sides of 1280, below and above 2^23 pixels (where the band begins), a tall and a wide one
@pytest.mark.parametrize("h,w", [(1280, 1283), (2896, 2896), (2896, 2897), (4500, 1281), (1290, 6600)])
@pytest.mark.parametrize("kind", ["noise", "frame", "rim", "surround", "slope", "many", "wall"])
def test_levels_and_result(nsgb, oracle, kind, h, w):
    dtype = {"noise": np.int32, "surround": np.uint16}.get(kind, np.uint8)
    img = (_image(kind, h, w, np.random.default_rng(h + w)) * SCALE[dtype]).astype(dtype)
    for conn in (4, 8):
        got, tried = _fill(img, conn)
        assert np.array_equal(got, oracle.imfill_holes(img, False, conn)), conn
        if kind in ("noise", "frame", "rim"):  # the level of the noise, or of the border around it
            assert 0 in tried, (conn, tried)
        elif kind in ("slope", "many"):
            assert tried == [], (conn, tried)
        elif kind == "wall" and h * w > 1 << 23:
            assert tried in ([], [BAND]), (conn, tried)
