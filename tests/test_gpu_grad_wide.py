"""Adjoint sums of gradients at the limits of the common unit: spans of 29 and 30 binary orders, gradients
at and below the resolution of 2^-96 (ties included), tiles with as many sources of several gradients as
there can be, images on both sides of 2^18 pixels (where clearing the far accumulators changes); bit for
bit against the oracle's exact sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradients(rng, shape):
    one = np.float32(1)
    sign = np.where(rng.random(shape) < 0.5, -one, one)
    man = (1 + rng.integers(0, 1 << 23, shape) / 2.0 ** 23).astype(np.float32)

    def pow2(e):
        return np.ldexp(one, e).astype(np.float32)

    for lo, hi in ((-29, 0), (-30, 0), (-73, -44), (-74, -44), (-73, -43)):  # spans and ends of the unit
        e = rng.integers(lo, hi + 1, shape)
        e.reshape(-1)[:2] = lo, hi
        yield f"2^{lo} .. 2^{hi}", sign * man * pow2(e)
    yield "tiny", sign * man * pow2(rng.integers(-110, -73, shape))
    yield "ties", sign * pow2(np.full(shape, -97)) * rng.integers(1, 8, shape).astype(np.float32)
    yield "subnormal", sign * pow2(np.full(shape, -149)) * rng.integers(1, 1 << 20, shape).astype(np.float32)
    yield "all orders", sign * man * pow2(rng.integers(-140, 20, shape))
    few = sign * man * pow2(rng.integers(-3, 3, shape))
    few.reshape(-1)[rng.integers(0, few.size, 1 + few.size // 300)] *= np.float32(2.0 ** -60)
    yield "few small", few


def _sources(rng, h, w):
    y, x = np.mgrid[0:h, 0:w]
    q = (y * w + x).astype(np.int64)
    yield "own", q
    yield "pairs", y * w + (x & ~1)  # 512 sources of two gradients in a tile
    yield "tile", (y & ~31) * w + (x & ~31)
    yield "far", rng.integers(0, h * w, (h, w))
    yield "one", np.full((h, w), h * w // 2)


def _check(nsgb, oracle, g, prov, what):
    dm, dk = nsgb.recon_f32_backward(torch.from_numpy(g).cuda(), torch.from_numpy(prov).cuda())
    em, ek = oracle.recon_f32_grad(g, prov)
    for got, exp in ((dm, em), (dk, ek)):
        got, exp = got.cpu().numpy(), np.asarray(exp, np.float32)
        assert np.array_equal(got.view(np.uint32), exp.reshape(got.shape).view(np.uint32)), what


@pytest.mark.parametrize("shape", [(32, 32), (40, 70), (64, 33)])
def test_units_and_wide_tiles(nsgb, oracle, shape):
    rng = np.random.default_rng(shape[0])
    for name, src in _sources(rng, *shape):
        for kind, g in _gradients(rng, shape):
            prov = np.where(rng.random(shape) < 0.5, src, ~src).astype(np.int32)
            _check(nsgb, oracle, np.ascontiguousarray(g, np.float32), prov, (name, kind))


@pytest.mark.parametrize("shape", [(512, 512), (512, 513), (1027, 259)])
def test_far_sources_around_the_small_image_limit(nsgb, oracle, shape):
    rng = np.random.default_rng(shape[1])
    for name, src in _sources(rng, *shape):
        if name in ("far", "one", "own"):
            prov = np.where(rng.random(shape) < 0.5, src, ~src).astype(np.int32)
            prov[rng.random(shape) < 0.02] = np.iinfo(np.int32).min
            for g in (rng.standard_normal(shape).astype(np.float32),
                      np.ldexp(rng.standard_normal(shape), rng.integers(-50, 10, shape)).astype(np.float32)):
                _check(nsgb, oracle, g, prov, name)
