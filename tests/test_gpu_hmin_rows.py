"""h-minima marker and zero-sign pass on rows of every remainder, pitch and start (through the C ABI),
against the oracle on dense copies."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 7, 8, 31, 33, 130])
def test_hmin_rows(nsgb, oracle, dtype, w):
    from nsgb import _ffi

    rng = np.random.default_rng(w)
    code = {np.uint8: 0, np.uint16: 1, np.float32: 3}[dtype]
    h, item = 6, np.dtype(dtype).itemsize
    # one pitch for image and result; starts in elements
    for pitch, off_in, off_out in ((w, 0, 0), (w + 3, 1, 0), ((w + 7) // 4 * 4, 0, 0), ((w + 7) // 4 * 4, 4, 1),
                                   ((w + 7) // 4 * 4, 0, 4)):
        vals = rng.integers(0, 40, (h, pitch))
        flat_in = np.zeros(off_in + h * pitch + 4, dtype)
        if dtype == np.float32:
            vals = vals * 0.25 - 3.0  # zeros of the inverted domain, and negative values
        flat_in[off_in:off_in + h * pitch] = vals.astype(dtype).reshape(-1)
        host = np.ascontiguousarray(flat_in[off_in:off_in + h * pitch].reshape(h, pitch)[:, :w])
        src = torch.from_numpy(flat_in).cuda()
        out = torch.from_numpy(np.full(off_out + h * pitch + 4, 7, dtype)).cuda()
        need = _ffi.lib.nsgb_workspace_size(_ffi.OP_HMIN, code, h, w)
        ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
        for conn in (4, 8):
            st = _ffi.lib.nsgb_imhmin(code, src.data_ptr() + off_in * item, out.data_ptr() + off_out * item, h, w,
                                      pitch * item, 3.0, conn, (ws.data_ptr() + 255) & ~255, need,
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
            assert st == 0
            got = out.cpu().numpy()
            body = got[off_out:off_out + h * pitch].reshape(h, pitch)
            exp = oracle.imhmin(host, 3.0, conn)
            assert np.array_equal(body[:, :w].view(f"u{item}"), np.asarray(exp, dtype).view(f"u{item}")), (pitch, conn)
            assert (body[:, w:] == 7).all() and (got[:off_out] == 7).all() and (got[off_out + h * pitch:] == 7).all()


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("h", [1e18, 9.3e18, 1e30, float("inf")])
def test_hmin_beyond_the_type(nsgb, oracle, dtype, h):
    """An h above every pixel, in and beyond 64 bits, is the largest h of the type."""
    img = np.random.default_rng(3).integers(0, 200, (40, 61)).astype(dtype)
    exp = oracle.imhmin(img, float(np.iinfo(dtype).max), 8)
    assert np.array_equal(nsgb.imhmin(torch.from_numpy(img).cuda(), h, 8).cpu().numpy(), exp)
