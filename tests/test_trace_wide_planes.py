"""The widened child-box planes of the ray queries (trace.cuh, wide_plane2):
they keep every box the exact planes keep (restated in numpy, CPU), and the
queries' hits equal brute force where the box test is at its limits (GPU)."""
import numpy as np
import pytest

F = np.float32
BIAS, FAR_SCALE = F(1 + 2.0 ** -21), F(1 + 6 * 2.0 ** -23)


def _wide_hits(p, e, lo, hi, o, d, tmin, tbest):
    """The device's box test in float32 (products of a fused multiply-add are exact in float64)."""
    with np.errstate(all="ignore"):
        den = np.where(np.abs(d) > F(1e-20), d, np.copysign(F(1e-20), d)).astype(F)
        inv = (F(1) / den).astype(F)
        S = (np.exp2(e.astype(np.float64)).astype(F) * (inv * F(32768)).astype(F)).astype(F)
        org = ((p - o).astype(F) * inv).astype(F)
        b = (org.astype(np.float64) - S.astype(np.float64) * np.float64(BIAS)).astype(F)

        def plane(q, f):
            v = 1.0 + (q + f / 256.0) / 32768.0
            assert np.array_equal(v.astype(F).astype(np.float64), v)
            return (v * S.astype(np.float64) + b.astype(np.float64)).astype(F)

        pl, ph = plane(lo.astype(np.float64), 0.0), plane(hi.astype(np.float64), 8.0)
        neg = inv < 0
        tn = np.fmax(np.fmax.reduce(np.where(neg, ph, pl), axis=1), tmin)
        tf = np.fmin(np.fmin.reduce(np.where(neg, pl, ph), axis=1), tbest)
        return tn <= (tf * FAR_SCALE).astype(F)


def _exact_hits(p, e, lo, hi, o, d, tmin, tbest):
    """Slab test over the exact quantised box, float64, with its own roundings against it."""
    p, o, d = p.astype(np.float64), o.astype(np.float64), d.astype(np.float64)
    s = np.exp2(e.astype(np.float64))
    a, b = p + lo * s, p + hi * s
    with np.errstate(all="ignore"):
        t0, t1 = (a - o) / d, (b - o) / d
    still = d == 0.0
    inside = (o >= a) & (o <= b)
    n = np.where(still, np.where(inside, -np.inf, np.inf), np.minimum(t0, t1)).max(1)
    f = np.where(still, np.where(inside, np.inf, -np.inf), np.maximum(t0, t1)).min(1)
    n, f = np.maximum(n, tmin), np.minimum(f, tbest)
    return (n <= f) & (f >= 0)


@pytest.mark.parametrize("scale_exp,far", [(-30, 1.0), (-9, 1.0), (-9, 1e4), (0, 10.0), (20, 1.0), (35, 3.0)])
@pytest.mark.parametrize("axis", ["any", "parallel", "tiny"])
def test_widened_planes_keep_every_exact_box(scale_exp, far, axis):
    rng = np.random.default_rng(abs(scale_exp) + int(far) + len(axis))
    n = 200_000
    e = rng.integers(scale_exp - 2, scale_exp + 3, (n, 3))
    s = np.exp2(e.astype(np.float64))
    p = (rng.normal(size=(n, 3)) * 100 * np.exp2(float(scale_exp)) * far).astype(F)
    lo = rng.integers(0, 256, (n, 3))
    hi = np.minimum(255, lo + rng.choice([0, 0, 1, 3, 40, 255], (n, 3)))  # flat boxes included
    # rays through a point of the box, often one of its corners, so that many just touch it
    at = np.where(rng.random((n, 3)) < 0.5, np.where(rng.random((n, 3)) < 0.5, lo, hi), rng.uniform(lo, hi))
    point = p.astype(np.float64) + at * s
    d = rng.normal(size=(n, 3))
    if axis == "parallel":
        d[np.arange(n), rng.integers(0, 3, n)] = 0.0
        d[rng.random(n) < 0.3, 0] = -0.0
    elif axis == "tiny":
        d[np.arange(n), rng.integers(0, 3, n)] *= 10.0 ** rng.uniform(-30, -5, n)
    d[np.abs(d).max(1) == 0.0] = (0.0, 1.0, 0.0)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    t = rng.uniform(0.0, 500.0, n) * np.exp2(float(scale_exp)) * far
    o = (point - t[:, None] * d.astype(np.float64)).astype(F)
    tmin = np.where(rng.random(n) < 0.5, 0.0, t * 0.5).astype(F)
    tbest = np.where(rng.random(n) < 0.5, np.inf, t * 1.5).astype(F)
    exact = _exact_hits(p, e, lo, hi, o, d, tmin, tbest)
    # a component the device replaces by 1e-20 moves the ray, where it is not zero, by its own definition
    exact &= ((d == 0) | (np.abs(d) > 1e-20)).all(1)
    assert exact.sum() > n // 50
    wide = _wide_hits(p, e, lo, hi, o, d, tmin, tbest)
    assert not (exact & ~wide).any()


@pytest.mark.gpu
@pytest.mark.parametrize("isect", [0, 1])
@pytest.mark.parametrize("size", [1e-3, 1.0, 30.0])
def test_hits_at_box_limits_equal_brute_force(size, isect):
    """Axis-parallel, grazing, far and vertex-aimed rays over scaled scenes, sorted and unsorted."""
    import pyoracle as po

    import myrt_b200 as mb
    from myrt_b200.scenes import heightfield

    rng = np.random.default_rng(5)
    idx, pts = heightfield(24, seed=3)
    pts = (pts * F(size)).astype(F)
    tris9 = pts[idx.reshape(-1, 3)].reshape(-1, 9)
    n = 4000
    goal = pts[rng.integers(0, len(pts), n)].astype(np.float64)      # vertices: corners of many boxes
    goal[n // 2:] += rng.normal(size=(n - n // 2, 3)) * 0.03 * size
    d = rng.normal(size=(n, 3))
    d[: n // 4, :] = np.eye(3)[rng.integers(0, 3, n // 4)] * rng.choice([-1.0, 1.0], (n // 4, 1))
    d[n // 4: n // 3, 1] = 0.0
    d[n // 3: n // 2, 1] *= 1e-6
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    rays = np.empty((n, 8), F)
    rays[:, :3] = goal - d.astype(np.float64) * rng.uniform(0.0, 5.0, (n, 1)) * size
    rays[:, 3] = np.where(rng.random(n) < 0.8, 0.0, 0.5 * size)
    rays[:, 4:7] = d
    rays[:, 7] = np.where(rng.random(n) < 0.8, np.inf, 3.0 * size)
    with mb.Context(0) as ctx:
        ctx.upload_scene(idx, pts)
        ref = po.brute_closest(tris9, rays, isect=isect)
        assert (ref["prim"] >= 0).sum() > n // 10
        for order in (1, 2):
            ctx.set_tuning(trace_order=order)
            assert np.array_equal(ctx.trace_closest(rays, intersector=isect), ref)
            assert np.array_equal(ctx.trace_any(rays, intersector=isect).astype(bool), ref["prim"] >= 0)
