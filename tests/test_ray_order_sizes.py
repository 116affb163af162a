"""The visiting order of ray batches (rayorder.cuh) over sizes around its tiles
of 32 and 1,024 rays, and over batches whose warps all stay whole, are all taken
apart, or mix: every ray is answered once, at its own index, bit for bit as in
input order. Consecutive batches reuse one scratch."""
import numpy as np
import pytest

import myrt_b200 as mb
from myrt_b200.scenes import heightfield_scene, pinhole_rays

pytestmark = pytest.mark.gpu


def _batch(kind, n, rng):
    cam = pinhole_rays(64, 64)
    coherent = cam[np.zeros(n, int)] if kind == "one ray" else cam[np.arange(n) % len(cam)]
    loose = coherent.copy()
    loose[:, :3] = rng.uniform(-1.5, 1.5, (n, 3))
    d = rng.normal(size=(n, 3))
    loose[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "odd":  # axis directions, far and non-finite origins, no direction at all
        loose[: n // 2, 4:7] = np.eye(3)[rng.integers(0, 3, n // 2)] * rng.choice([-1.0, 1.0], (n // 2, 1))
        loose[::7, :3] *= 1e6
        loose[::31, 0] = np.nan
        loose[::37, 1] = np.inf
        loose[::41, 4:7] = 0.0
    if kind == "mixed":  # warps of both sorts in every tile
        pick = (np.arange(n) // 32) % 3 == 1
        return np.where(pick[:, None], loose, coherent).astype(np.float32)
    return (loose if kind in ("loose", "odd") else coherent).astype(np.float32)


@pytest.mark.parametrize("kind", ["one ray", "camera", "loose", "mixed", "odd"])
def test_order_answers_every_ray_once(kind):
    import torch

    rng = np.random.default_rng(7)
    with mb.Context(0) as ctx:
        scene, _ = heightfield_scene(48, seed=3)
        ctx.upload_scene(**scene)
        for n in (1, 31, 32, 33, 257, 1023, 1024, 1025, 1056, 4097, 70_001, 33):
            rays = torch.from_numpy(_batch(kind, n, rng)).cuda()
            got = {}
            for order in (1, 2):
                ctx.set_tuning(trace_order=order)
                hits = torch.full((n, 4), -7.0, device="cuda")
                occ = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                ctx.trace_closest_device(rays, hits)
                ctx.trace_any_device(rays, occ)
                ctx.sync()
                got[order] = hits.cpu().numpy().view(np.uint32), occ.cpu().numpy()
            assert np.array_equal(got[1][0], got[2][0]) and np.array_equal(got[1][1], got[2][1]), n
            assert got[2][1].max() <= 1


def test_default_order_at_its_line():
    """Batches on both sides of 2^20 rays, where the default starts to order them."""
    import torch

    rng = np.random.default_rng(8)
    with mb.Context(0) as ctx:
        scene, _ = heightfield_scene(16, seed=3)
        ctx.upload_scene(**scene)
        full = torch.from_numpy(_batch("mixed", (1 << 20) + 33, rng)).cuda()
        for n in ((1 << 20) - 1, 1 << 20, (1 << 20) + 33):
            got = []
            for order in (1, 0):
                ctx.set_tuning(trace_order=order)
                hits = torch.full((n, 4), -7.0, device="cuda")
                torch.cuda.synchronize()
                ctx.trace_closest_device(full[:n], hits)
                ctx.sync()
                got.append(hits)
            assert torch.equal(got[0].view(torch.int32), got[1].view(torch.int32))
