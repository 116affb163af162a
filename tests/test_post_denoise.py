"""The denoise pass' quotients by a fixed divisor (postprocess.cu, div_by) are
the correctly rounded ones, and the pass equals the oracle's bit for bit over
sigmas on both sides of the fast path, block edges, HDR and non-finite texels;
the blur passes at sizes smaller than their reach."""
import numpy as np
import pytest

import pyoracle as po

F, L = np.float32, np.longdouble


@pytest.mark.parametrize("divisor", [0.0025, 0.05, 0.3, 1.0, 1.9999999, 7.0 ** -20, 3.0e17, 1.1754944e-17])
def test_quotient_by_reciprocal_is_correctly_rounded(divisor):
    b = F(divisor)
    r = F(1) / b
    rng = np.random.default_rng(int(divisor * 1e6) % 1000)
    m = rng.integers(0, 1 << 23, 400_000)
    m[:5] = (0, 1, (1 << 23) - 1, (1 << 23) - 2, 1 << 22)
    for e in (-60, -3, 0, 20):
        x = np.ldexp((1.0 + m / 2.0 ** 23).astype(F), e).astype(F)
        q = (x * r).astype(F)
        for _ in range(2):  # 24-bit products are exact in 64 bits; one rounding to float32 at the end
            rem = (x.astype(L) - q.astype(L) * L(b)).astype(F)
            q = (q.astype(L) + rem.astype(L) * L(r)).astype(F)
        assert np.array_equal(q, x / b)


def _img(h, w, seed, hi):
    rng = np.random.default_rng(seed)
    return (rng.uniform(0.0, hi, (h, w, 4))).astype(np.float16).astype(F)


@pytest.mark.gpu
@pytest.mark.parametrize("h,w", [(1, 1), (7, 31), (8, 32), (9, 33), (41, 70)])
@pytest.mark.parametrize("spatial,sigma", [(10.0, 0.05), (0.7, 0.2), (3.0, -0.4), (10.0, 1e-3), (5.0, 2e-10), (10.0, 3e9),
                                           (1e-12, 50.0)])
def test_denoise_bit_exact(ctx, h, w, spatial, sigma):
    import torch

    from myrt_b200 import post

    img = _img(h, w, h * w, 1.2)  # some centres above 1: their weights underflow with a small sigma
    if h > 8:
        img[3, 5, :3] = (np.inf, 1.0, 0.2)
        img[6, 20, 1] = np.nan
        img[2, 12, :3] = 60000.0
        img[7, 9, :3] = F(3e20)
        img[5, 3, :3] = F(1e-30)
    p = (spatial, sigma, 0.0, 0.0)
    got = post.run(ctx, 0, torch.from_numpy(img).cuda(), p=p).cpu().numpy()
    with po.glsl_math(1):
        ref = po.post_pass(0, img, p=p)
    assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("h,w,step", [(1, 1, 1.25), (3, 40, 1.25), (40, 3, 1.25), (17, 16, 0.4), (33, 35, -2.5), (50, 21, 1.0),
                                      (20, 90, 0.0)])
def test_blur_bit_exact(ctx, direction, h, w, step):
    import torch

    from myrt_b200 import post

    img = _img(h, w, h + w, 3.0)
    got = post.blur(ctx, torch.from_numpy(img).cuda(), direction, step).cpu().numpy()
    assert np.array_equal(got, po.post_pass(1, img, i=(direction, 0, 0), p=(step, 0, 0, 0)))
