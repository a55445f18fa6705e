"""Row widths and alignments around the 16-byte accesses of threshold, h-minima marker and bounding
boxes: every remainder, rows that start unaligned, against numpy and the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(rng, dtype, h, w, pitch, off):
    """A h x w view with the given row pitch and start (elements), on host and device."""
    top = {np.uint8: 256, np.uint16: 65536, np.int32: 2**31 - 1, np.float32: 1}[dtype]
    flat = (rng.random(off + pitch * h + 8) * top).astype(dtype)
    t = torch.from_numpy(flat).cuda()
    host = flat[off:off + pitch * h].reshape(h, pitch)[:, :w]
    return np.ascontiguousarray(host), t, t.data_ptr() + off * flat.itemsize


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32, np.float32])
@pytest.mark.parametrize("w", [1, 3, 7, 8, 15, 16, 17, 31, 33, 64, 4097])
def test_threshold_rows(nsgb, dtype, w):
    from nsgb import _ffi

    rng = np.random.default_rng(w)
    code = {np.uint8: 0, np.uint16: 1, np.int32: 2, np.float32: 3}[dtype]
    for pitch, off in ((w, 0), (w + 3, 1), ((w + 31) // 16 * 16, 0), ((w + 31) // 16 * 16, 4)):
        h = 5
        host, keep, ptr = _rows(rng, dtype, h, w, pitch, off)
        thr = {np.uint8: 100, np.uint16: 30000, np.int32: 10**9, np.float32: 0.4}[dtype]
        for po in (w, (w + 31) // 16 * 16):
            out = torch.full((h, po), 7, dtype=torch.uint8, device="cuda")
            st = _ffi.lib.nsgb_threshold(code, ptr, out.data_ptr(), h, w, pitch * host.itemsize, po, float(thr),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0
            got = out.cpu().numpy()
            assert np.array_equal(got[:, :w], np.where(host > host.dtype.type(thr), 255, 0)), (pitch, off, po)
            assert (got[:, w:] == 7).all()


@pytest.mark.parametrize("w", [1, 3, 4, 5, 31, 33, 130])
def test_bounding_box_rows(nsgb, oracle, w):
    from nsgb import _ffi

    rng = np.random.default_rng(w)
    h = 9
    for pitch, off in ((w, 0), (w + 1, 1), ((w + 7) // 4 * 4, 0)):
        lab = np.zeros((h, pitch), np.int32)
        lab[:, :w] = rng.integers(-1, h * w + 1, (h, w)) if w == 31 else rng.integers(1, h * w + 1, (h, w))
        flat = np.zeros(off + h * pitch, np.int32)
        flat[off:] = lab.reshape(-1)
        t = torch.from_numpy(flat).cuda()
        exp = oracle.bounding_box(np.ascontiguousarray(lab[:, :w]), 0)
        cap = h * w
        boxes = torch.zeros((5, cap), dtype=torch.int32, device="cuda")
        n = C.c_int32(0)
        need = _ffi.lib.nsgb_workspace_size(_ffi.OP_BOUNDING_BOX, _ffi.I32, h, w)
        ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
        st = _ffi.lib.nsgb_bounding_boxes(t.data_ptr() + 4 * off, h, w, 4 * pitch, 0, boxes.data_ptr(), cap, C.byref(n),
                                          None, (ws.data_ptr() + 255) & ~255, need,
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
        assert st == 0
        assert np.array_equal(boxes[:, :n.value].cpu().numpy(), np.asarray(exp).reshape(5, -1))
