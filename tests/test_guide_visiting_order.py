"""Guided waves read the lobes of a point from tiles in visiting order: the same
image in queue order, ordered by cell, and over several waves, at path counts
around the 128-point tile."""
import numpy as np
import pytest

import myrt_b200 as mb
from myrt_b200.camera import look_at
from myrt_b200.scenes import guiding_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (16, 8, 1), (43, 3, 1), (37, 29, 3)])
def test_guided_image_does_not_depend_on_the_order(width, height, spp):
    rng = np.random.default_rng(4)
    with mb.Context(0) as ctx:
        scene, lights = guiding_box(slab_cells=12, seed=1)
        ctx.upload_scene(**scene)
        ctx.set_area_lights(lights)
        ctx.guide_configure(fraction=0.5, train=0)
        ctx.guide_set_params((rng.normal(size=16640) * 0.15).astype(np.float32))
        iv, ip = look_at((0.0, 0.5, -2.5), (0.0, 0.0, 0.0), vfov_deg=60.0, aspect=width / height)
        out = []
        for order, wave in ((1, 0), (2, 0), (2, 1024)):  # waves of 1,024 paths at least
            ctx.set_tuning(trace_order=order, wave_paths=wave)
            ctx.reset_accumulation()
            ctx.render_physical(iv, ip, width, height, spp=spp, max_depth=5, rr_start=3, seed=3, guided=True)
            out.append(ctx.read_accumulation(width, height)[0])
    assert out[0][..., 3].min() == spp and np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
