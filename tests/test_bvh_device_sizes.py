"""Device BVH build at the edges of its kernels: node boxes come from runs of
256 sorted leaves (sizes around multiples of 256, where nodes begin to reach
past a block), slots are assigned by 8 lanes a node (trees of one leaf slot, of
one node, and of coincident triangles, whose boxes tie)."""
import numpy as np
import pytest

import myrt_b200 as mb
import pyoracle as po
from test_bvh_device import _check_tree, _rand_rays

pytestmark = pytest.mark.gpu


def _triangles(kind, n):
    rng = np.random.default_rng(n)
    if kind == "coincident":  # few distinct triangles, many times over
        base = rng.uniform(-1, 1, (max(1, n // 40), 3, 3))
        return base[np.arange(n) % len(base)].astype(np.float32)
    centre = rng.uniform(-1, 1, (n, 1, 3))
    if kind == "line":  # an unbalanced radix tree: sizes and distances over 12 decades
        centre = np.sign(rng.normal(size=(n, 1, 1))) * 10.0 ** rng.uniform(-9, 0, (n, 1, 1)) * [[[1.0, 1e-3, 1e-3]]]
        return (centre + rng.normal(size=(n, 3, 3)) * np.abs(centre[..., :1]) * 0.1).astype(np.float32)
    return (centre + rng.normal(size=(n, 3, 3)) * 0.05).astype(np.float32)


@pytest.mark.parametrize("n", [2, 4, 5, 33, 255, 256, 257, 512, 513, 3000])
@pytest.mark.parametrize("kind", ["scattered", "line", "coincident"])
def test_device_build_sizes(ctx, kind, n):
    tris9 = _triangles(kind, n).reshape(-1, 9)
    rays = _rand_rays(3_000, seed=n)
    rays[: 1500, 4:7] = tris9[np.arange(1500) % n].reshape(-1, 3, 3).mean(1) - rays[: 1500, 0:3]  # toward triangles
    try:
        ctx.set_tuning(bvh_builder=1)
        info = ctx.upload_scene(np.arange(3 * n, dtype=np.uint32), tris9.reshape(-1, 3))
        nodes, tris = ctx.scene_bvh()
        assert info["triangles"] == n and info["leaf_slots"] >= -(-n // 4)
        _check_tree(nodes, tris, n)
        # the leaf-ordered copies are the prims' own corners
        prim = tris[:, 3].view(np.uint32)
        assert np.array_equal(tris[:, [0, 1, 2, 4, 5, 6, 8, 9, 10]], tris9[prim])
        walk, _, _ = po.bvh8_traverse(nodes, tris, rays)
        hits = ctx.trace_closest(rays)
        assert np.array_equal(hits, walk)
        if kind != "line":  # 1e-9-sized triangles: the float test itself accepts rays that pass their boxes by
            assert np.array_equal(hits, po.brute_closest(tris9, rays))
    finally:
        ctx.set_tuning()
