"""A path wave takes the visiting order's scratch last: on a device with room
for everything else it renders unordered instead of failing."""
import numpy as np
import pytest

import myrt_b200 as mb
from myrt_b200.camera import look_at
from myrt_b200.scenes import guiding_box

pytestmark = pytest.mark.gpu

SIDE, SPP, DEPTH = 512, 64, 4
ORDER = 12 * SIDE * SIDE * SPP + (32 << 20)


def _wave_bytes(paths, guided):
    queues = 4 * 48 + 16                  # two ray queues, hits, shadow rays; radiance
    guide = 48 + 256 + 96 * DEPTH         # points, lobes, records
    return paths * (queues + (guide if guided else 0)) + (64 * max(paths, 1 << 20) if guided else 0)  # samples


@pytest.mark.parametrize("guided", [False, True])
def test_wave_renders_where_only_the_order_has_no_room(guided):
    import torch

    def render(ctx, spp):
        iv, ip = look_at((0.0, 0.0, -0.95), (0.0, 0.0, 0.5), vfov_deg=90.0, aspect=1.0)
        ctx.reset_accumulation()
        ctx.render_physical(iv, ip, SIDE, SIDE, spp=spp, max_depth=DEPTH, rr_start=2, seed=3, guided=guided)
        return ctx.read_accumulation(SIDE, SIDE)[0]

    images = []
    scene, lights = guiding_box(slab_cells=12, seed=1)
    for full in (False, True):
        with mb.Context(0) as ctx:
            ctx.upload_scene(**scene)
            ctx.set_area_lights(lights)
            ctx.guide_configure(fraction=0.5, train=0)
            render(ctx, 1)  # images, the guide's own buffers, kernels and their local memory
            torch.cuda.synchronize()
            hold = None
            if full:
                # leaves the wave's buffers (the small render's go back first) and half of the order's scratch
                room = _wave_bytes(SIDE * SIDE * SPP, guided) - _wave_bytes(SIDE * SIDE, guided) + ORDER // 2
                torch.cuda.empty_cache()
                hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
            images.append(render(ctx, SPP))
            del hold
            torch.cuda.empty_cache()
    assert images[0][..., 3].min() == SPP
    assert np.array_equal(images[0], images[1])
