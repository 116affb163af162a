"""The work a user of myrt_b200 has it do, as cases that can be prepared, run and timed.

A case is a dict of plain values. `listed()` names the standing ones, `draw(rng)`
gives one more of the same ranges, `prepare(case, seed)` makes what a program
holds before the call (scene uploaded, buffers and weights in place), and
`run(state)` is one pass through the public entry points. Kinds:

  pick     scene::pick: a handful of rays from host memory, answered on the host
  query    closest-hit / any-hit queries on device memory (batches of rays)
  view     the reference's own frames (reference shading)
  path     physical path tracing, plain or with a learned guide
  train    Adam steps of the guide on host samples
  preview  the raster preview, optionally after moving every instance
  post     the per-frame post-processing chain and the denoiser

Scenes, cameras and sizes are the ones of this repository's tests and benchmark;
the seed changes every scene, ray, image and weight.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import myrt_b200 as mb
from myrt_b200 import _abi, post, scenes
from myrt_b200 import sdf as sdfs
from myrt_b200.camera import look_at, view_projection

FAR = 100.0  # tmax of the query rays: past every scene here
EYE, TARGET, VFOV = scenes.ICOSPHERE_EYE, scenes.ICOSPHERE_TARGET, scenes.ICOSPHERE_VFOV
HF_EYE, HF_TARGET, HF_VFOV = (0.0, 2.0, -3.0), (0.0, 0.0, 0.0), 60.0


def listed():
    return [
        # one click in the editor: the object under the cursor of the 655,872-triangle scene
        dict(name="pick_ray", kind="pick", scene="ico", size=512, rays=1),
        # a 1024 x 1024 visibility pass over the small height field, any intersection order the library picks
        dict(name="closest_field_1m", kind="query", scene="hf", size=128, rays=1 << 20, bounce=0.0, any=False,
             watertight=False, instanced=False),
        # the benchmark's batch: 512 x 512 x 64 spp camera rays and the first diffuse bounce of those that hit
        dict(name="closest_ico_28m", kind="query", scene="ico", size=512, rays=27_900_000, bounce=0.4, any=False,
             watertight=False, instanced=False),
        # a ragged batch of shadow rays from visible points to an area light, watertight
        dict(name="shadow_ico_3m", kind="query", scene="ico", size=512, rays=3_000_017, bounce=1.0, any=True,
             watertight=True, instanced=False),
        # an accumulating offline render in the reference's shading: 64 frames a call
        dict(name="view_64_frames", kind="view", scene="ico", size=512, width=512, height=512, bounces=8, frames=64,
             extras=False),
        # the interactive viewport: one frame a call, the default 10 bounces, textures, cube map and depth of field
        dict(name="view_720p_frame", kind="view", scene="hf", size=256, width=1280, height=720, bounces=10, frames=1,
             extras=True),
        # plain path tracing, 512 x 512, 64 spp, depth 8, FP32 accumulation
        dict(name="path_64_spp", kind="path", scene="ico", size=512, width=512, height=512, spp=64, depth=8, sdf=0,
             guided=False, fp64=False),
        # a guided frame with a finished guide (inference only) of the indirect-lit box
        dict(name="path_guided", kind="path", scene="box", size=160, width=512, height=512, spp=16, depth=8, sdf=0,
             guided=True, fp64=False),
        # meshes and a 256-primitive smooth union in one frame, FP64 accumulation
        dict(name="path_sdf", kind="path", scene="ico", size=64, width=512, height=512, spp=8, depth=8, sdf=256,
             guided=False, fp64=True),
        # the guide's online training: 16 Adam steps of 16,384 samples
        dict(name="train_guide", kind="train", samples=65536, steps=16, batch=16384),
        # dragging objects in the preview: every instance moves, then a 1920 x 1080 frame with its shadow map
        dict(name="preview_moving", kind="preview", scene="ico", size=512, width=1920, height=1080, shadow=2048,
             move=True),
        # the frame chain (bloom, tonemap, FXAA) and the denoiser on a 2048 x 2048 image
        dict(name="post_2048", kind="post", width=2048, height=2048, super_sampling=1.0, denoise=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng):
    scene = rng.choice(["hf", "ico"])
    return scene, _log(rng, 16, 512) if scene == "hf" else _log(rng, 4, 512)


def draw(rng):
    kind = rng.choice(["pick", "query", "query", "query", "view", "view", "path", "path", "train", "preview", "post"])
    if kind == "pick":
        scene, size = _mesh(rng)
        return dict(kind=kind, scene=scene, size=size, rays=_log(rng, 1, 1000))
    if kind == "query":
        scene, size = _mesh(rng)
        return dict(kind=kind, scene=scene, size=size, rays=_log(rng, 1000, 20_000_000),
                    bounce=rng.choice([0.0, 0.4, 1.0]), any=rng.random() < 0.4, watertight=rng.random() < 0.4,
                    instanced=scene == "ico" and rng.random() < 0.25)
    if kind == "view":
        scene, size = _mesh(rng)
        w, h = _log(rng, 65, 1400), _log(rng, 65, 1400)
        extras = scene == "hf" and rng.random() < 0.5
        return dict(kind=kind, scene=scene, size=size, width=w, height=h, bounces=rng.randint(2, 10),
                    frames=max(1, min(_log(rng, 1, 64), (10 << 20) // (w * h))), extras=extras)
    if kind == "path":
        scene, size = _mesh(rng)
        sdf = rng.choice([0, 0, 0, _log(rng, 16, 256)])
        guided = sdf == 0 and rng.random() < 0.35
        if guided:
            scene, size = "box", _log(rng, 16, 200)
        w, h = _log(rng, 65, 700), _log(rng, 65, 700)
        paths = 1 << 20 if sdf else (3 << 20 if guided else 10 << 20)
        return dict(kind=kind, scene=scene, size=size, width=w, height=h,
                    spp=max(1, min(_log(rng, 1, 64), paths // (w * h))), depth=rng.randint(3, 8), sdf=sdf,
                    guided=guided, fp64=rng.random() < 0.3)
    if kind == "train":
        batch = 128 * _log(rng, 8, 128)
        return dict(kind=kind, samples=_log(rng, 1000, 100_000), steps=rng.randint(4, 16), batch=batch)
    if kind == "preview":
        return dict(kind=kind, scene="ico", size=_log(rng, 4, 512), width=_log(rng, 320, 1920),
                    height=_log(rng, 200, 1200), shadow=rng.choice([512, 1024, 2048]), move=rng.random() < 0.5)
    return dict(kind=kind, width=_log(rng, 65, 2048), height=_log(rng, 65, 2048),
                super_sampling=rng.choice([1.0, 1.0, 2.0]), denoise=rng.random() < 0.5)


# ---- scenes -----------------------------------------------------------------------------------

def _scene(case, seed):
    """(upload_scene arguments, area lights) of a case's mesh scene."""
    size = case["size"]
    if case["scene"] == "hf":  # 2 size^2 triangles
        return scenes.heightfield_scene(size, seed=seed)
    if case["scene"] == "box":
        return scenes.guiding_box(slab_cells=size, seed=seed)
    return scenes.icosphere_field_lit(n_spheres=size, seed=seed)  # 1,280 size + 512 triangles


def _camera(case):
    """Eye, target and field of view of a case's scene."""
    if case["scene"] == "hf":
        return HF_EYE, HF_TARGET, HF_VFOV
    if case["scene"] == "box":
        return (0.0, 0.0, -0.95), (0.0, 0.0, 0.5), 90.0
    return EYE, TARGET, VFOV


def _triangles(case):
    size = case["size"]
    return {"hf": 2 * size * size, "ico": 1280 * size + 512, "box": 4 * size * size + 770}[case["scene"]]


def _world(scene):
    """World triangles float64 [T, 3, 3] of an upload_scene dict, in the library's prim order."""
    idx, v = scene["indices"].astype(np.int64), np.asarray(scene["vertices"], np.float64)[:, :3]
    if scene.get("drawables") is None:
        return v[idx].reshape(-1, 3, 3)
    out = []
    for d in scene["drawables"]:
        m = np.array(d.transformation[:], np.float64).reshape(4, 4).T
        p = v[idx[d.indices_base_index: d.indices_base_index + d.index_count] + d.points_base_index]
        out.append(p @ m[:3, :3].T + m[:3, 3])
    return np.concatenate(out).reshape(-1, 3, 3)


def _context(case, scene, lights):
    ctx = mb.Context(torch.cuda.current_device())
    if case.get("instanced"):
        ctx.set_tuning(instancing=1)
    ctx.upload_scene(**scene)
    if lights is not None:
        ctx.set_area_lights(lights)
    return ctx


def _stream():
    return torch.cuda.current_stream().cuda_stream or 1  # 1: the legacy default stream's own handle


class _Memory:
    """A device image of the library, for torch.as_tensor (no copy). The tensor keeps this object, and this object the
    context that owns the image."""

    def __init__(self, ctx, ptr, shape, kind):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def _tensor(ctx, ptr, shape, kind):
    return torch.as_tensor(_Memory(ctx, ptr, shape, kind), device="cuda")


# ---- rays -------------------------------------------------------------------------------------

def _camera_rays(case, n, seed):
    """float32 [n, 8] jittered rays of the case's view on the GPU, in rows of pixels, sample after sample."""
    eye, target, vfov = (np.asarray(a, np.float64) for a in _camera(case))
    side = max(1, min(1024, int(round(math.sqrt(n))))) if case["scene"] == "hf" else max(1, min(512, int(math.sqrt(n))))
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = (target - eye) / np.linalg.norm(target - eye)
    r = np.cross(f, (0.0, 1.0, 0.0))
    r /= np.linalg.norm(r)
    u = np.cross(r, f)
    f, r, u = (torch.tensor(a, device="cuda", dtype=torch.float32) for a in (f, r, u))
    t = math.tan(math.radians(float(vfov)) / 2)
    i = torch.arange(n, device="cuda") % (side * side)
    if n < 1024:  # a few rays: anywhere in the image
        i = torch.randint(0, 1 << 20, (n,), generator=g, device="cuda")
        side = 1024
    sx = (2 * ((i % side) + torch.rand(n, generator=g, device="cuda")) / side - 1) * t
    sy = (1 - 2 * ((i // side) + torch.rand(n, generator=g, device="cuda")) / side) * t
    d = torch.nn.functional.normalize(f + sx[:, None] * r + sy[:, None] * u, dim=1)
    rays = torch.empty((n, 8), device="cuda")
    rays[:, :3] = torch.tensor(eye, device="cuda", dtype=torch.float32)
    rays[:, 3] = 0.0
    rays[:, 4:7] = d
    rays[:, 7] = FAR
    return rays


def _secondary_rays(case, ctx, scene, camera, n, seed, light):
    """n rays from what the camera rays hit: diffuse bounces, or shadow rays to the area light `light`."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    hits = torch.empty((camera.shape[0], 4), device="cuda")
    ctx.trace_closest_device(camera, hits, stream=_stream())
    ctx.sync()
    torch.cuda.synchronize()
    prim = hits.view(torch.int32)[:, 0]
    at = torch.nonzero(prim >= 0)[:, 0]
    at = at[torch.arange(n, device="cuda") % at.shape[0]]
    tri = torch.from_numpy(_world(scene).astype(np.float32)).cuda()[prim[at].long()]
    nrm = torch.nn.functional.normalize(torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]), dim=1)
    d = camera[at, 4:7]
    nrm = torch.where((nrm * d).sum(1, keepdim=True) > 0, -nrm, nrm)
    p = camera[at, :3] + hits[at, 1:2] * d + 1e-4 * nrm
    rays = torch.empty((n, 8), device="cuda")
    rays[:, :3] = p
    rays[:, 3] = 0.0
    if light is None:
        w = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1) + nrm
        rays[:, 4:7] = torch.nn.functional.normalize(w, dim=1)
        rays[:, 7] = FAR
    else:
        row = torch.from_numpy(light).cuda()
        a = torch.rand((n, 2), generator=g, device="cuda")
        to = row[0:3] + a[:, :1] * row[3:6] + a[:, 1:] * row[6:9] - p
        dist = to.norm(dim=1, keepdim=True)
        rays[:, 4:7] = to / dist
        rays[:, 7:] = dist * 0.999
    return rays


# ---- prepare ----------------------------------------------------------------------------------

def prepare(case, seed):
    return {"pick": _prepare_pick, "query": _prepare_query, "view": _prepare_view, "path": _prepare_path,
            "train": _prepare_train, "preview": _prepare_preview, "post": _prepare_post}[case["kind"]](case, seed)


def _prepare_pick(case, seed):
    scene, _ = _scene(case, seed)
    rays = _camera_rays(case, case["rays"], seed).cpu().numpy()
    return dict(case=case, ctx=_context(case, scene, None), rays=rays, scene=scene)


def _prepare_query(case, seed):
    scene, lights = _scene(case, seed)
    ctx = _context(case, scene, None)
    n = case["rays"]
    second = int(n * case["bounce"])
    camera = _camera_rays(case, max(n - second, 1024 if second else 0), seed)
    rays = camera[: n - second]
    if second:
        more = _secondary_rays(case, ctx, scene, camera, second, seed, lights[0] if case["any"] else None)
        rays = torch.cat([rays, more]).contiguous()
    if case["any"]:
        out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    else:
        out = torch.zeros((n, 4), device="cuda")
    isect = mb.ISECT_WATERTIGHT if case["watertight"] else mb.ISECT_REFERENCE
    return dict(case=case, ctx=ctx, rays=rays.contiguous(), out=out, isect=isect)


def _textured(case, seed):
    """The height field with uvs, a textured material, a cube map and a bokeh mask."""
    rng = np.random.default_rng(seed)
    n = case["size"]
    scene, lights = _scene(case, seed)
    g = np.linspace(0.0, 4.0, n + 1, dtype=np.float32)
    u, v = np.meshgrid(g, g, indexing="xy")
    scene["uvs"] = np.stack([u.ravel(), v.ravel()], 1)
    data = np.asarray(scene["material_data"], np.float32).copy()
    data[5:6] = np.array([1], np.uint32).view(np.float32)  # albedo texture handle: slot 0 + 1
    scene["material_data"] = data
    albedo = rng.uniform(0.2, 1.0, (64, 64, 4)).astype(np.float32)
    y, x = np.mgrid[0:32, 0:32]
    mask = np.repeat((((x - 15.5) ** 2 + (y - 15.5) ** 2) < 225)[..., None], 4, 2).astype(np.float32)
    cube = np.ones((6, 64, 64, 4), np.float32)
    cube[..., :3] = rng.uniform(0.2, 1.2, (6, 1, 1, 3)) * np.linspace(0.6, 1.0, 64)[None, :, None, None]
    return scene, lights, albedo, mask, cube


def _prepare_view(case, seed):
    more = {}
    if case["extras"]:
        scene, _, albedo, mask, cube = _textured(case, seed)
    else:
        scene, _ = _scene(case, seed)
    ctx = _context(case, scene, None)
    if case["extras"]:
        ctx.upload_texture(0, albedo)
        ctx.upload_texture(1, mask)
        ctx.upload_cubemap(cube)
        more = dict(dof=True, lens_size=(0.1, 0.08), focus=3.2, bokeh_slot=1)
    eye, target, vfov = _camera(case)
    iv, ip = look_at(eye, target, vfov_deg=vfov, aspect=case["width"] / case["height"])
    return dict(case=case, ctx=ctx, iv=iv, ip=ip, more=more, seed=seed)


def _guide_weights(seed):
    """Parameters of a guide of plausible sharpness: Glorot layers, an output layer that spreads its lobes."""
    rng = np.random.default_rng(seed)
    w = rng.uniform(-1.0, 1.0, (4, 64, 64)) * math.sqrt(6.0 / 128.0)
    b = rng.uniform(-0.2, 0.2, (4, 64))
    b[3, 1:40:5] += 2.0  # kappa of the lobes
    b[3, 2:40:5] += rng.uniform(-1.0, 1.0, 8)
    b[3, 3:40:5] += rng.uniform(-1.0, 1.0, 8)
    b[3, 4:40:5] += rng.uniform(-1.0, 1.0, 8)
    return np.concatenate([w.ravel(), b.ravel()]).astype(np.float32)


def _prepare_path(case, seed):
    scene, lights = _scene(case, seed)
    ctx = _context(case, scene, lights)
    if case["sdf"]:
        lib = sdfs.SdfLibrary()
        lib.add(sdfs.random_sdf_field(case["sdf"], k=0.1, seed=seed, extent=0.8, chain=True))
        move = np.eye(4)
        move[:3, 3] = (0.0, -0.2, 0.3)
        ctx.upload_sdf(lib.instrs, lib.programs, lib.params, sdfs.sdf_drawables([move], [0]))
    if case["guided"]:
        ctx.guide_configure(fraction=0.5, train=0)
        ctx.guide_set_params(_guide_weights(seed))
    eye, target, vfov = _camera(case)
    iv, ip = look_at(eye, target, vfov_deg=vfov, aspect=case["width"] / case["height"])
    return dict(case=case, ctx=ctx, iv=iv, ip=ip, seed=seed)


def _prepare_train(case, seed):
    rng = np.random.default_rng(seed)
    n = case["samples"]
    scene, _ = scenes.guiding_box(slab_cells=8, seed=seed)
    ctx = _context(case, scene, None)
    ctx.guide_configure(batch=case["batch"], learning_rate=1e-3, train=1)
    ctx.guide_set_params(_guide_weights(seed))

    def unit(a):
        return a / np.linalg.norm(a, axis=1, keepdims=True)

    # radiance samples of the box: points, normals, views, and directions that lean towards the slots
    s = np.zeros((n, 16), np.float32)
    p = rng.uniform(-1.0, 1.0, (n, 3))
    nrm = unit(rng.normal(size=(n, 3)))
    s[:, 0:3] = p
    s[:, 3] = rng.exponential(1.0, n) / n
    s[:, 4:7] = nrm
    s[:, 8:11] = unit(nrm + 0.9 * unit(rng.normal(size=(n, 3))))
    goal = np.where((p[:, 1] > 0.0)[:, None], (0.9, 0.3, 0.0), (-0.9, -0.3, 0.0))
    s[:, 12:15] = unit(unit(goal - p) + 0.7 * unit(rng.normal(size=(n, 3))))
    return dict(case=case, ctx=ctx, samples=s)


def _prepare_preview(case, seed):
    rng = np.random.default_rng(seed)
    scene, _ = _scene(case, seed)
    ctx = _context(case, scene, None)
    poses = []
    for _ in range(2):
        moved = (_abi.myrt_drawable * len(scene["drawables"]))()
        for k, d in enumerate(scene["drawables"]):
            ctypes.memmove(ctypes.byref(moved[k]), ctypes.byref(d), ctypes.sizeof(d))
            if k + 1 == len(scene["drawables"]):
                break  # the floor stays
            m = np.array(d.transformation[:], np.float64).reshape(4, 4)
            m[3, :3] += rng.uniform(-0.1, 0.1, 3)
            moved[k].transformation[:] = m.astype(np.float32).ravel().tolist()
            moved[k].inverse_transformation[:] = np.linalg.inv(m).astype(np.float32).ravel().tolist()
        poses.append(moved)
    view, proj = view_projection(EYE, TARGET, vfov_deg=VFOV, aspect=case["width"] / case["height"], near=0.05,
                                 far=50.0)
    return dict(case=case, ctx=ctx, poses=poses, passes=0, view=view, proj=proj, seed=seed)


def _prepare_post(case, seed):
    scene, _ = scenes.heightfield_scene(4, seed=seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["height"], case["width"]
    # an HDR image: smooth shading, texture noise and a few bright lights
    y = torch.linspace(0.0, 1.0, h, device="cuda")[:, None, None]
    x = torch.linspace(0.0, 1.0, w, device="cuda")[None, :, None]
    c = torch.rand((2, 4), generator=g, device="cuda")
    img = 0.2 + 0.6 * c[0] * (0.5 + 0.5 * torch.sin(9 * x + 5 * y)) + 0.3 * c[1] * y
    img = img + 0.1 * torch.rand((h, w, 4), generator=g, device="cuda")
    img = torch.where(torch.rand((h, w, 1), generator=g, device="cuda") < 0.01, img * 6.0, img)
    return dict(case=case, ctx=_context(dict(case), scene, None), img=img.half().float().contiguous())


# ---- run --------------------------------------------------------------------------------------

def run(state):
    return {"pick": _run_pick, "query": _run_query, "view": _run_view, "path": _run_path, "train": _run_train,
            "preview": _run_preview, "post": _run_post}[state["case"]["kind"]](state)


def _run_pick(s):
    h = s["ctx"].trace_closest(s["rays"])
    return dict(prim=h.view(np.int32).reshape(-1, 4)[:, 0], tuv=h.view(np.float32).reshape(-1, 4)[:, 1:])


def _run_query(s):
    if s["case"]["any"]:
        s["ctx"].trace_any_device(s["rays"], s["out"], s["isect"], stream=_stream())
        return dict(occluded=s["out"])
    s["ctx"].trace_closest_device(s["rays"], s["out"], s["isect"], stream=_stream())
    return dict(prim=s["out"].view(torch.int32)[:, 0], tuv=s["out"][:, 1:])


def _images(ctx, width, height):
    """The context's device images (myrt_render_buffers): accumulation and display."""
    a, d = ctypes.c_void_p(), ctypes.c_void_p()
    ctx._check(_abi.lib().myrt_render_buffers(ctx._h, ctypes.byref(a), ctypes.byref(d)), "myrt_render_buffers")
    shape = (height, width, 4)
    return _tensor(ctx, a.value, shape, "<f4"), _tensor(ctx, d.value, shape, "<f4")


def _run_view(s):
    c, ctx = s["case"], s["ctx"]
    ctx.set_seed(s["seed"])
    ctx.reset_accumulation()
    ctx.render(s["iv"], s["ip"], c["width"], c["height"], num_bounces=c["bounces"], frames=c["frames"], **s["more"])
    accum, display = _images(ctx, c["width"], c["height"])
    return dict(accum=accum, display=display)


def _run_path(s):
    c, ctx = s["case"], s["ctx"]
    ctx.reset_accumulation()
    ctx.render_physical(s["iv"], s["ip"], c["width"], c["height"], spp=c["spp"], max_depth=c["depth"], rr_start=3,
                        seed=s["seed"], fp64=c["fp64"], guided=c["guided"], sdf_marching_steps=256,
                        sdf_marching_epsilon=1e-4)
    accum, display = _images(ctx, c["width"], c["height"])
    if c["fp64"]:
        accum = _tensor(ctx, ctx.render_buffer_f64(), (c["height"], c["width"], 4), "<f8")
    return dict(accum=accum, display=display)


def _run_train(s):
    loss = s["ctx"].guide_train(s["samples"], s["case"]["steps"])
    return dict(loss=loss, params=s["ctx"].guide_params())


def _run_preview(s):
    c, ctx = s["case"], s["ctx"]
    if c["move"]:
        ctx.set_transforms(s["poses"][s["passes"] & 1])
        s["passes"] += 1
    w, h, n = c["width"], c["height"], c["shadow"]
    ctx.forward_render(s["view"], s["proj"], w, h, random_seed=s["seed"] & 0xFFFF, shadow_size=n)
    b = ctx.forward_buffers()
    return dict(result=_tensor(ctx, b["result"], (h, w, 4), "<f2"),
                gbuffer=_tensor(ctx, b["gbuffer"], (3, h, w, 4), "<f2"),
                shadow_map=_tensor(ctx, b["shadow_map"], (n, n, 4), "<f4"),
                visibility=_tensor(ctx, b["visibility"], (h, w), "<i8"))


def _run_post(s):
    c = s["case"]
    frame = post.frame(s["ctx"], s["img"], super_sampling=c["super_sampling"])
    return dict(frame=frame, denoised=post.denoise(s["ctx"], frame)) if c["denoise"] else dict(frame=frame)


# ---- work -------------------------------------------------------------------------------------

def _levels(case):
    return max(1, math.ceil(math.log(_triangles(case), 8)))


def _scene_bytes(case, rays=1 << 40):
    """The triangles' corners once, or what `rays` rays reach of them: a node a level and a triangle each."""
    return min(_triangles(case) * 36, rays * (_levels(case) * 64 + 36))


def _ray_flops(case):
    """Least work of one ray: one eight-box node a level of an 8-wide tree, one triangle."""
    return _levels(case) * 8 * 15 + 45


def work(case):
    kind = case["kind"]
    if kind in ("pick", "query"):
        n, hit = case["rays"], 1 if case.get("any") else 16
        return {"bytes": n * (32 + hit) + _scene_bytes(case, n), "flops": n * _ray_flops(case)}
    if kind == "view":
        px = case["width"] * case["height"]
        # the camera ray and its shadow ray of each sample; images written once
        return {"bytes": px * 32 + _scene_bytes(case), "flops": px * case["frames"] * 2 * _ray_flops(case)}
    if kind == "path":
        px = case["width"] * case["height"]
        flops = 2 * _ray_flops(case) + (2 * 4 * 64 * 64 if case["guided"] else 0) + case["sdf"] * 10
        return {"bytes": px * (48 if case["fp64"] else 32) + _scene_bytes(case), "flops": px * case["spp"] * flops}
    if kind == "train":
        n = min(case["samples"], case["batch"])
        return {"bytes": case["samples"] * 64 + 2 * 16640 * 4, "flops": case["steps"] * n * 3 * 2 * 4 * 64 * 64}
    if kind == "preview":
        px, sp, t = case["width"] * case["height"], case["shadow"] ** 2, _triangles(case)
        return {"bytes": t * 72 + px * (8 + 24 + 8) + sp * 16, "flops": t * 2 * 100 + (px + sp) * 50}
    px = case["width"] * case["height"]
    out = px / case["super_sampling"] ** 2
    return {"bytes": 16 * (px + out * (3 if case["denoise"] else 1)),
            "flops": out * (0.5 * 31 * 8 + 200) + (out * 81 * 20 if case["denoise"] else 0)}


# ---- exact ------------------------------------------------------------------------------------

def exact(case, seed):
    """run()'s answer for a fresh state in 64-bit torch / numpy, where that is a matter of seconds."""
    kind = case["kind"]
    if kind in ("pick", "query"):
        if case.get("any") or case.get("bounce") or case["rays"] * _triangles(case) > 5e10:
            return None
        return _exact_closest(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "post":
        return _exact_post(case, seed)
    return None  # random walks and rasterised coverage have no plain 64-bit counterpart


def _exact_closest(case, seed):
    """Moller-Trumbore of every ray with every triangle: the four determinants are bilinear in the ray's
    (direction, moment, origin, 1) and the triangle's edge products."""
    scene, _ = _scene(case, seed)
    tri = torch.from_numpy(_world(scene)).cuda()
    v1, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = torch.linalg.cross
    z3, z1 = torch.zeros_like(v1), torch.zeros_like(v1[:, :1])
    n = cross(e1, e2)
    cols = [torch.cat(c, 1).T.contiguous() for c in (
        (-n, z3, z3, z1),                                               # det
        (-cross(e2, v1), e2, z3, z1),                                   # u det
        (cross(e1, v1), -e1, z3, z1),                                   # v det
        (z3, z3, n, -(v1 * n).sum(1, keepdim=True)))]                   # t det
    rays = _camera_rays(case, case["rays"], seed).double()
    o, d, tmax = rays[:, :3], rays[:, 4:7], rays[:, 7:]
    feat = torch.cat([d, cross(o, d), o, torch.ones_like(tmax)], 1)
    out = torch.empty((rays.shape[0], 3), dtype=torch.float64, device="cuda")
    step = max(1, int(1.5e8) // tri.shape[0])
    for a in range(0, rays.shape[0], step):
        f = feat[a:a + step]
        inv = 1.0 / (f @ cols[0])
        u = (f @ cols[1]).mul_(inv)
        v = (f @ cols[2]).mul_(inv)
        t = (f @ cols[3]).mul_(inv)
        ok = (u >= -1e-6) & (v >= -1e-6) & (u + v <= 1 + 1e-6) & (t > 0) & (t < tmax[a:a + step])
        best, at = torch.where(ok, t, math.inf).min(1)
        hit = torch.isfinite(best)
        pick = at[:, None]
        out[a:a + step, 0] = torch.where(hit, best, tmax[a:a + step, 0])
        out[a:a + step, 1] = torch.where(hit, u.gather(1, pick)[:, 0], 0.0)
        out[a:a + step, 2] = torch.where(hit, v.gather(1, pick)[:, 0], 0.0)
    return dict(prim=None, tuv=out)


def _exact_train(case, seed):
    """The same Adam steps through autograd in 64 bits."""
    s = _prepare_train(case, seed)["samples"]
    scene, _ = scenes.guiding_box(slab_cells=8, seed=seed)
    lo, hi = _world(scene).reshape(-1, 3).min(0), _world(scene).reshape(-1, 3).max(0)
    s = torch.from_numpy(s).cuda().double()
    lo, hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    p = ((s[:, :3] - 0.5 * (lo + hi)) / (0.5 * (hi - lo))).clamp(-1, 1)
    f = [p]
    for k in range(6):
        for a in range(3):
            f += [torch.sin(math.pi * p[:, a:a + 1] * 2 ** k), torch.cos(math.pi * p[:, a:a + 1] * 2 ** k)]
    x = torch.cat(f + [s[:, 4:7], s[:, 8:11], torch.ones_like(p[:, :1]), torch.zeros((s.shape[0], 18), device="cuda")],
                  1)
    w, d = s[:, 3], s[:, 12:15]
    prm = torch.from_numpy(_guide_weights(seed)).cuda().double().requires_grad_()
    m, v = torch.zeros_like(prm), torch.zeros_like(prm)
    losses, n = [], s.shape[0]
    batch = min(n, case["batch"])
    for step in range(case["steps"]):
        a = (step * batch) % (n - batch + 1) if n > batch else 0
        h = x[a:a + batch]
        for k in range(4):
            h = h @ prm[k * 4096:(k + 1) * 4096].view(64, 64).T + prm[16384 + 64 * k:16448 + 64 * k]
            h = torch.relu(h) if k < 3 else h
        o = h[:, :40].view(-1, 8, 5)
        kap = (torch.nn.functional.softplus(o[:, :, 1]) + 0.01).clamp(max=1000.0)
        mu = torch.nn.functional.normalize(o[:, :, 2:], dim=2)
        c = (mu * d[a:a + batch, None]).sum(2)
        q = (torch.softmax(o[:, :, 0], 1) * kap / (-2 * math.pi * torch.expm1(-2 * kap)) * torch.exp(kap * (c - 1)))
        loss = -(w[a:a + batch] * torch.log(q.sum(1))).sum()
        g, = torch.autograd.grad(loss, prm)
        losses.append(loss.detach())
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.99 * v + 0.01 * g * g
            mh, vh = m / (1 - 0.9 ** (step + 1)), v / (1 - 0.99 ** (step + 1))
            prm = (prm - 1e-3 * mh / (vh.sqrt() + 1e-8)).requires_grad_()
    return dict(loss=torch.stack(losses), params=prm.detach())


def _taps(img, x, y, mirrored=True):
    """Bilinear samples at texel coordinates x [W'] by y [H'] of img [H, W, 4]."""
    h, w = img.shape[:2]

    def wrap(i, n):
        if not mirrored:
            return i.clamp(0, n - 1)
        m = i.remainder(2 * n)
        return torch.where(m < n, m, 2 * n - 1 - m)

    fx, fy = torch.floor(x), torch.floor(y)
    a, b = (x - fx)[None, :, None], (y - fy)[:, None, None]
    x0, x1 = wrap(fx.long(), w), wrap(fx.long() + 1, w)
    y0, y1 = wrap(fy.long(), h), wrap(fy.long() + 1, h)
    rows = img[y0] * (1 - b) + img[y1] * b
    return rows[:, x0] * (1 - a) + rows[:, x1] * a


def _grid_taps(img, x, y):
    """Bilinear samples at texel coordinates x, y [H', W'] (mirrored)."""
    h, w = img.shape[:2]

    def at(i, j):
        i, j = i.remainder(2 * w), j.remainder(2 * h)
        i, j = torch.where(i < w, i, 2 * w - 1 - i), torch.where(j < h, j, 2 * h - 1 - j)
        return img[j, i]

    i, j = torch.floor(x).long(), torch.floor(y).long()
    a, b = (x - i)[..., None], (y - j)[..., None]
    return (at(i, j) * (1 - a) + at(i + 1, j) * a) * (1 - b) + (at(i, j + 1) * (1 - a) + at(i + 1, j + 1) * a) * b


def _exact_post(case, seed):
    """The frame chain and the denoiser as plain 64-bit images (no rounding to half between passes)."""
    img = _prepare_post(case, seed)["img"].double()

    def axis(n):
        return torch.arange(n, device="cuda", dtype=torch.float64)

    def scale(im, factor):
        h, w = post.scaled_size(im.shape[0], im.shape[1], factor)
        return _taps(im, (axis(w) + 0.5) / w * im.shape[1] - 0.5, (axis(h) + 0.5) / h * im.shape[0] - 0.5, False)

    weights = [0.08756118061424645, 0.08547984344465417, 0.07952880794840879, 0.0705164133185798, 0.05958841266910679,
               0.04798885898065629, 0.03683205838316095, 0.0269412473017388, 0.018780823225920923,
               0.012477173150624141, 0.007899915153736418, 0.004766876346593609, 0.0027412691146821303,
               0.001502371210393176, 0.0007847156649807812, 0.0003906237796399568]

    def blur(im, along_y):
        h, w = im.shape[:2]
        r = weights[0] * _taps(im, axis(w) - 0.5, axis(h) - 0.5)
        for i in range(1, 16):
            sx, sy = (0.0, 1.25 * i) if along_y else (1.25 * i, 0.0)
            r = r + weights[i] * (_taps(im, axis(w) + sx - 0.5, axis(h) + sy - 0.5) +
                                  _taps(im, axis(w) - sx - 0.5, axis(h) - sy - 0.5))
        return r

    im = scale(img, 1.0 / case["super_sampling"])
    r = scale(torch.where(im <= 1.0, 0.0, im), 0.5)
    r = scale(blur(blur(r, False), True), 2.0)
    h, w = im.shape[:2]
    im = im + 0.3 * _taps(r, axis(w) / w * r.shape[1] - 0.5, axis(h) / h * r.shape[0] - 0.5)
    x = (im[..., :3] - 0.004).clamp(min=0.0)
    x = ((x * (6.2 * x + 0.5)) / (x * (6.2 * x + 1.7) + 0.06)) ** 1.3
    im = torch.cat([x, torch.ones_like(x[..., :1])], 2)

    luma = torch.tensor([0.299, 0.587, 0.114, 0.0], device="cuda", dtype=torch.float64)
    gx, gy = axis(w)[None, :].expand(h, w) - 0.5, axis(h)[:, None].expand(h, w) - 0.5
    nw, ne, sw, se, mid = (_grid_taps(im, gx + i, gy + j) for i, j in ((-1, -1), (1, -1), (-1, 1), (1, 1), (0, 0)))
    lw, le, lo, lp, lm = (t @ luma for t in (nw, ne, sw, se, mid))
    every = torch.stack([lw, le, lo, lp, lm])
    low, high = every.min(0).values, every.max(0).values
    dx, dy = -((lw + le) - (lo + lp)), (lw + lo) - (le + lp)
    reduce = ((lw + le + lo + lp) * 0.03125).clamp(min=1.0 / 128.0)
    rcp = 1.0 / (torch.minimum(dx.abs(), dy.abs()) + reduce)
    dx, dy = (dx * rcp).clamp(-8, 8), (dy * rcp).clamp(-8, 8)

    def along(k):
        return _grid_taps(im, gx + dx * k, gy + dy * k)

    first = 0.5 * (along(1 / 3 - 0.5) + along(2 / 3 - 0.5))
    second = 0.5 * first + 0.25 * (along(-0.5) + along(0.5))
    lb = second @ luma
    frame = torch.where(((lb < low) | (lb > high))[..., None], first, second)
    frame[..., 3] = 1.0
    if not case["denoise"]:
        return dict(frame=frame)
    z = torch.zeros((h, w, 1), device="cuda", dtype=torch.float64)
    total = torch.zeros((h, w, 3), device="cuda", dtype=torch.float64)
    centre = frame[..., :3]
    for i in range(-4, 5):
        xs = (axis(w).long() + i).clamp(0, w - 1)
        for j in range(-4, 5):
            t = frame[(axis(h).long() + j).clamp(0, h - 1)][:, xs, :3].clamp(0, 1)
            k = torch.exp(-0.5 * ((t - centre) ** 2).sum(2, keepdim=True) / 0.05 ** 2)
            k = k * math.exp(-0.5 * (i * i + j * j) / 10.0 ** 2)
            z += k
            total += k * t
    return dict(frame=frame, denoised=torch.cat([total / z, torch.ones_like(z)], 2))
