"""Path waves past the size from which blocks walk their queue (16 times the
blocks the device holds: 2.4 M paths), and batches whose shadow rays run beside
the next vertex's extension: with lights, without, and mixed, in waves of
different sizes. Images do not depend on any of it."""
import numpy as np
import pytest

import myrt_b200 as mb
from myrt_b200.camera import look_at
from myrt_b200.scenes import guiding_box, icosphere_field_lit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guided", [False, True])
def test_waves_larger_than_their_grid(guided):
    import torch

    width, height, spp = 641, 479, 9  # 2,763,351 paths
    grid = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 16 * 128
    assert grid < width * height * spp < 2 * grid
    scene, lights = guiding_box(slab_cells=12, seed=1) if guided else icosphere_field_lit(n_spheres=32, seed=4)
    eye, target, vfov = ((0.0, 0.0, -0.95), (0.0, 0.0, 0.5), 90.0) if guided else ((0, 1, -4.5), (0, -0.3, 0), 50.0)
    iv, ip = look_at(eye, target, vfov_deg=vfov, aspect=width / height)
    out = []
    with mb.Context(0) as ctx:
        ctx.upload_scene(**scene)
        ctx.set_area_lights(lights)
        ctx.guide_configure(fraction=0.5, train=0)
        for order, wave in ((1, 1 << 20), (1, 0), (0, 0)):  # three waves; one; one, visited by cell
            ctx.set_tuning(trace_order=order, wave_paths=wave)
            ctx.reset_accumulation()
            ctx.render_physical(iv, ip, width, height, spp=spp, max_depth=5, rr_start=2, seed=3, guided=guided)
            out.append(ctx.read_accumulation(width, height)[0])
    assert out[0][..., 3].min() == spp and out[0][..., :3].max() > 0
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("lit", [(True, True), (False, False), (True, False), (False, True)])
def test_batches_with_and_without_lights(lit):
    ctxs, jobs = [], []
    for k, on in enumerate(lit):
        scene, lights = icosphere_field_lit(n_spheres=8 + 8 * k, subdiv=2, floor_cells=4, seed=3 + k)
        ctx = mb.Context(0)
        ctx.upload_scene(**scene)
        if on:
            ctx.set_area_lights(lights)
        ctxs.append(ctx)
        for depth, width, height, spp in ((1, 48, 32, 3), (6, 33, 57, 5)):
            iv, ip = look_at((0, 1, -4.5), (0, -0.3, 0), vfov_deg=50, aspect=width / height)
            jobs.append(dict(scene=k, inverse_view=iv, inverse_projection=ip, width=width, height=height, spp=spp,
                             seed=depth, max_depth=depth, rr_start=2, env=(0.2, 0.3, 0.4)))
    refs = []
    for j in jobs:
        ctx = ctxs[j["scene"]]
        ctx.reset_accumulation()
        for _ in range(2):
            ctx.render_physical(j["inverse_view"], j["inverse_projection"], j["width"], j["height"], spp=j["spp"],
                                max_depth=j["max_depth"], rr_start=j["rr_start"], seed=j["seed"], env=j["env"])
        refs.append(ctx.read_accumulation(j["width"], j["height"])[0])
    for wave in (2000, 1 << 20):  # several waves a frame, each ending with its own join; one
        batch = mb.Batch(ctxs, jobs)
        batch.set_tuning(wave_paths=wave, blocks_per_sm=8)
        for _ in range(2):
            batch.render()
        for k, ref in enumerate(refs):
            assert np.array_equal(batch.read(k), ref), (wave, k)
        batch.close()
    for ctx in ctxs:
        ctx.close()
