"""Host-memory queries on both sides of the size where they stop using mapped
memory (16,384 rays): same answers as the device-memory entry points."""
import numpy as np
import pytest

import myrt_b200 as mb
from myrt_b200.scenes import heightfield_scene, pinhole_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 2])
@pytest.mark.parametrize("isect", [mb.ISECT_REFERENCE, mb.ISECT_WATERTIGHT])
def test_host_queries_equal_device_queries(isect, order):
    import torch

    rays = pinhole_rays(160, 128).astype(np.float32)
    rays[::5, 7] = 1.5  # some end before the surface
    with mb.Context(0) as ctx:
        scene, _ = heightfield_scene(32, seed=2)
        ctx.upload_scene(**scene)
        ctx.set_tuning(trace_order=order)
        hits = torch.empty((len(rays), 4), device="cuda")
        occ = torch.empty(len(rays), dtype=torch.uint8, device="cuda")
        d_rays = torch.from_numpy(rays).cuda()
        torch.cuda.synchronize()
        ctx.trace_closest_device(d_rays, hits, isect)
        ctx.trace_any_device(d_rays, occ, isect)
        ctx.sync()
        ref, blocked = hits.cpu().numpy().view(np.uint32), occ.cpu().numpy()
        assert 0 < blocked.sum() < len(rays)
        for n in (1, 2, 127, 16383, 16384, 16385, len(rays), 1):
            got = ctx.trace_closest(rays[-n:], intersector=isect)
            assert np.array_equal(got.view(np.uint32).reshape(n, 4), ref[-n:])
            assert np.array_equal(ctx.trace_any(rays[-n:], intersector=isect), blocked[-n:])
        assert ctx.trace_closest(rays[:0], intersector=isect).shape == (0,)
