"""Training kernel at the edges of its tiles: fewer samples than one 128-row
tile, a ragged last tile, several tiles per CTA (more than one per SM), all
against the numpy restatement with the device's BF16 rounding points; and host
training calls of changing sizes, which share one device buffer."""
import numpy as np
import pytest

import pyguide as pg
from myrt_b200.scenes import guiding_box

pytestmark = pytest.mark.gpu


def _samples(n, seed):
    rng = np.random.default_rng(seed)

    def unit(a):
        return a / np.linalg.norm(a, axis=1, keepdims=True)

    s = np.zeros((n, 16), np.float32)
    s[:, 0:3] = rng.uniform(-1, 1, (n, 3))
    s[:, 3] = rng.exponential(1.0, n) / n
    s[rng.random(n) < 0.1, 3] = 0.0
    s[:, 4:7] = unit(rng.normal(size=(n, 3)))
    s[:, 8:11] = unit(rng.normal(size=(n, 3)))
    s[:, 12:15] = unit(rng.normal(size=(n, 3)) + (1.0, 0.5, 0.0))
    return s


@pytest.fixture(scope="module")
def box(ctx):
    scene, _ = guiding_box(slab_cells=4, seed=3)
    ctx.upload_scene(**scene)
    v = np.asarray(scene["vertices"], np.float32).reshape(-1, 3)
    ctx.guide_configure(seed=11)
    ctx.guide_reset()
    rng = np.random.default_rng(1)
    p = ctx.guide_params()
    p[-256:] = rng.uniform(-0.3, 0.3, 256).astype(np.float32)  # biases: every layer's gradient has something to do
    ctx.guide_set_params(p)
    return p, np.concatenate([v.min(0), v.max(0)])


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 148 * 128 + 5, 40000])
def test_gradients_at_tile_edges(ctx, box, n):
    params, bounds = box
    s = _samples(n, seed=n)
    g, loss = ctx.guide_gradients(s)
    rg, rl = pg.gradients(params, s, bounds)
    # BF16 activations flip one rounding in 2^8 where the float sums differ in their last bits; a flip moves one
    # sample's contribution by 2^-8, so a layer's relative error is of the order of 2^-8 times the share of flips
    for a in list(range(0, 16384, 4096)):
        assert np.linalg.norm(g[a:a + 4096] - rg[a:a + 4096]) <= 1e-2 * np.linalg.norm(rg[a:a + 4096])
    for a in range(16384, 16640, 64):
        assert np.linalg.norm(g[a:a + 64] - rg[a:a + 64]) <= 1e-2 * np.linalg.norm(rg[a:a + 64])
    assert abs(loss - rl) <= 1e-4 * abs(rl) + 1e-7


def test_host_training_calls_of_changing_sizes(ctx, box):
    params, bounds = box
    first = None
    for n, steps in ((5000, 3), (64, 2), (20000, 1), (5000, 3)):
        ctx.guide_reset()  # a fresh optimiser
        ctx.guide_set_params(params)
        loss = ctx.guide_train(_samples(n, seed=7), steps)
        assert loss.shape == (steps,) and np.isfinite(loss).all()
        _, rl = pg.gradients(params, _samples(n, seed=7)[: min(n, ctx.guide_config()["batch"])], bounds)
        assert abs(loss[0] - rl) <= 1e-4 * abs(rl)
        if n == 5000:
            now = (loss, ctx.guide_params())
            if first is not None:  # the same call again, after calls of other sizes
                assert np.allclose(now[0], first[0], rtol=1e-4) and np.allclose(now[1], first[1], atol=2e-3)
            first = now
    lobes = ctx.guide_eval(np.zeros((300, 12), np.float32) + 0.5)
    assert np.isfinite(lobes).all()
