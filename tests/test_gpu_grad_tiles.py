"""Adjoint sums around the 32 x 32 tiles they are formed in: sources in the own tile, in a
neighbouring one and far away, one source for everything, marker and mask sources at one pixel,
tiny and zero gradients, pitched stacks; bit for bit against the oracle's exact sums."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 65), (65, 1), (31, 33), (32, 32), (33, 64), (64, 97), (100, 130)]


def _check(nsgb, oracle, g, prov):
    dm, dk = nsgb.recon_f32_backward(torch.from_numpy(g).cuda(), torch.from_numpy(prov).cuda())
    em, ek = oracle.recon_f32_grad(g, prov)
    for got, exp in ((dm, em), (dk, ek)):
        got, exp = got.cpu().numpy(), np.asarray(exp)
        assert np.array_equal(got.view(np.uint32), exp.reshape(got.shape).view(np.uint32))


def _gradients(rng, shape):
    g = rng.standard_normal(shape).astype(np.float32)
    yield g
    yield (g * np.float32(2.0) ** rng.integers(-100, 20, shape)).astype(np.float32)  # below the resolution too
    yield np.where(rng.random(shape) < 0.7, np.float32(0), -g * 0).astype(np.float32)  # +0 and -0
    big = np.where(rng.random(shape) < 0.5, np.float32(2.0 ** 18), np.float32(-2.0 ** 18))
    yield (big + g * np.float32(2.0 ** -20)).astype(np.float32)


@pytest.mark.parametrize("shape", SHAPES)
def test_sums_over_tiles(nsgb, oracle, shape):
    h, w = shape
    n = h * w
    rng = np.random.default_rng(n)
    y, x = np.mgrid[0:h, 0:w]
    q = (y * w + x).astype(np.int64)
    near = np.clip(y + rng.integers(-3, 4, shape), 0, h - 1) * w + np.clip(x + rng.integers(-3, 4, shape), 0, w - 1)
    sources = [q, near, rng.integers(0, n, shape), np.full(shape, n // 2), np.full(shape, n - 1)]
    for g in _gradients(rng, shape):
        for src in sources:
            kind = rng.random(shape)
            prov = np.where(kind < 0.45, src, ~src).astype(np.int32)      # both classes at one pixel
            prov[kind > 0.97] = np.iinfo(np.int32).min                     # the ring
            _check(nsgb, oracle, g, prov)


def test_stack_and_in_place(nsgb, oracle):
    """A stack of images, and gradients written over the incoming gradient (C ABI)."""
    from nsgb import _ffi

    rng = np.random.default_rng(5)
    b, h, w = 3, 45, 70
    g = rng.standard_normal((b, h, w)).astype(np.float32)
    prov = rng.integers(0, h * w, (b, h, w)).astype(np.int32)
    prov = np.where(rng.random((b, h, w)) < 0.5, prov, ~prov)
    _check(nsgb, oracle, g, prov)
    tg, tp = torch.from_numpy(g).cuda(), torch.from_numpy(prov).cuda()
    dk = torch.empty_like(tg)
    need = _ffi.lib.nsgb_recon_f32_workspace_size(b, h, w, 1)
    ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    st = _ffi.lib.nsgb_recon_f32_bwd(tg.data_ptr(), tp.data_ptr(), tg.data_ptr(), dk.data_ptr(), b, h, w, w * 4,
                                     h * w * 4, (ws.data_ptr() + 255) & ~255, need,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    assert st == 0
    em, ek = oracle.recon_f32_grad(g, prov)
    assert np.array_equal(tg.cpu().numpy(), em) and np.array_equal(dk.cpu().numpy(), ek)
