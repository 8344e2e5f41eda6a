"""The work that this framework is measured on.

A case is one call, or one short fixed sequence of calls, that a user's program makes over and over:

* ``preview``   one interactive batch through ``render_sample_batch`` (a new host frame buffer per call);
* ``viewport``  a progressive viewport update: accumulation steps on the device, one resolved frame to the host;
* ``frame``     a final frame through ``render_batch`` into a page-locked frame buffer the program keeps;
* ``plain``     the same through the strict one-request entry point ``render``;
* ``views``     many requests of uneven size against one scene in one ``render_batch`` call;
* ``gradient``  steps of inverse rendering: forward and backward of ``autograd.render``, new parameters every step;
* ``animate``   deformed geometry: upload and preview of two frames of an animation;
* ``relight``   look development: upload and preview after an edit of lights, environment and materials;
* ``rays``      closest hits and occlusion of the caller's own rays (picking, baking).

Scenes are the repository's workloads (scenes.py): the sphere on a ground quad, the field of noise-displaced
icospheres, the sphere cut into one mesh per material, and a studio of glass, emitters, cut-outs and layered
materials (those of the golden frames).  Geometry, materials, environment and cameras all come from the seed.
Every state owns its backend, as every program does.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from shiro_gb300 import (DistantLight, DomeLight, FrameBuffer, GpuBackend, Material, Mesh, RenderRequest, RenderSettings,
                         Scene, lambert, scenes, standard_surface, usd_preview_surface)

# The arithmetic a path cannot do without, from the work counts of the estimator (closest and occlusion rays: eight
# boxes of about 14 operations per wide node visited, 45 per triangle tested; about 150 per BSDF value or pdf, 100
# per environment lookup, 40 per sample dimension): the field's path visits 25 nodes and tests 9.5 triangles, the
# sphere's about a third of that.
FLOPS_PER_PATH = {"field": 4200.0, "sphere": 2000.0, "parts": 2000.0, "studio": 3000.0}
FLOPS_PER_RAY = 1500.0
PIXEL_BYTES = 44  # beauty 4, albedo 3, normal 3, depth 1 floats


def listed():
    return [
        # the first refinement of an interactive view: launches and latency are all of it
        {"name": "preview 256x256x1 sphere", "kind": "preview", "scene": "sphere", "width": 256, "height": 256, "spp": 1,
         "depth": 3, "env": 512},
        # one display update of a progressive HD viewport with the accumulator's default (one-thread-per-path) form
        {"name": "viewport 1280x720x2 field", "kind": "viewport", "scene": "field", "width": 1280, "height": 720, "spp": 1,
         "steps": 2, "depth": 3, "instances": 256, "env": 2048, "wavefront": False},
        # the small reference configuration: 64x32-segment sphere, 256x256, 16 samples, depth 8
        {"name": "frame 256x256x16 sphere", "kind": "frame", "scene": "sphere", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "env": 512},
        # the headline: a 1.31 M triangle field at 1080p, 64 samples, depth 12
        {"name": "frame 1920x1080x64 field", "kind": "frame", "scene": "field", "width": 1920, "height": 1080, "spp": 64,
         "depth": 12, "instances": 256, "env": 2048},
        # the strict single-request entry point, at an odd size and sample count
        {"name": "plain 961x541x15 field", "kind": "plain", "scene": "field", "width": 961, "height": 541, "spp": 15,
         "depth": 12, "instances": 256, "env": 2048},
        # every lobe of the integrator: glass, a medium, a thin pane, emitters, cut-outs, coats, sheen, anisotropy
        {"name": "frame 640x480x32 studio", "kind": "frame", "scene": "studio", "width": 640, "height": 480, "spp": 32,
         "depth": 8, "env": 512},
        # a render service's queue: uneven requests packed into one call
        {"name": "views 24 uneven sphere", "kind": "views", "scene": "sphere", "requests": 24, "size": 640, "spp": 64,
         "depth": 12, "env": 512},
        # material and environment gradients of one 512x512 view, 32 samples, depth 6, 256 materials
        {"name": "gradient 512x512x32 parts", "kind": "gradient", "scene": "parts", "width": 512, "height": 512, "spp": 32,
         "depth": 6, "materials": 256, "env": 512, "steps": 2, "decorrelate": False},
        # one view of a multi-view inverse rendering of the field, gradients from an independent sample range
        {"name": "gradient 512x512x16 field", "kind": "gradient", "scene": "field", "width": 512, "height": 512, "spp": 16,
         "depth": 8, "instances": 256, "env": 1024, "steps": 2, "decorrelate": True},
        # two frames of deforming geometry, each uploaded whole and previewed
        {"name": "animate 64 blobs 960x540x4", "kind": "animate", "scene": "field", "width": 960, "height": 540, "spp": 4,
         "depth": 4, "instances": 64, "env": 1024},
        # look development: the geometry stays, lights, environment and materials change
        {"name": "relight 1279x719x4 field", "kind": "relight", "scene": "field", "width": 1279, "height": 719, "spp": 4,
         "depth": 4, "instances": 256, "env": 2048},
        # picking and baking rays against a small model
        {"name": "rays 200003 sphere", "kind": "rays", "scene": "sphere", "rays": 200003, "env": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: image sizes from thumbnails to 1080p (odd ones as they come), 1 to 64
    samples, depths 1 to 12, small to full scenes; at most half the headline's paths."""
    kind = rng.choice(["preview", "viewport", "frame", "frame", "frame", "plain", "views", "gradient", "gradient", "animate",
                       "relight", "rays"])
    if kind == "rays":
        return {"kind": kind, "scene": "sphere", "rays": _log(rng, 1000, 1000000), "env": 64}
    if kind == "views":
        return {"kind": kind, "scene": "sphere", "requests": rng.randint(2, 32), "size": _log(rng, 160, 640),
                "spp": rng.choice([4, 16, 64]), "depth": rng.choice([4, 8, 12]), "env": rng.choice([64, 512])}
    width = _log(rng, 64, 1920)
    height = max(33, int(width * rng.uniform(0.5, 1.0)))
    c = {"kind": kind, "width": width, "height": height, "env": rng.choice([256, 512, 1024, 2048])}
    if kind == "gradient":
        c["width"], c["height"] = min(width, 640), min(height, 512)
        c["scene"] = rng.choice(["parts", "field"])
        c["spp"], c["depth"] = _log(rng, 4, 32), rng.randint(2, 8)
        c["steps"], c["decorrelate"] = rng.randint(1, 2), rng.random() < 0.5
        c["env"] = min(c["env"], 1024)
        if c["scene"] == "parts":
            c["materials"] = _log(rng, 2, 256)
    elif kind in ("animate", "relight"):
        c["scene"], c["spp"], c["depth"] = "field", rng.randint(1, 8), rng.randint(2, 6)
    elif kind in ("preview", "viewport"):
        c["scene"], c["spp"], c["depth"] = rng.choice(["sphere", "field", "studio"]), rng.randint(1, 4), rng.randint(2, 5)
        if kind == "viewport":
            c["steps"], c["wavefront"] = rng.randint(1, 4), rng.random() < 0.5
    else:
        c["scene"], c["depth"] = rng.choice(["sphere", "field", "studio"]), rng.randint(3, 12)
        c["spp"] = max(1, min(_log(rng, 4, 64), (1 << 26 if kind == "frame" else 1 << 24) // (width * height)))
    if c["scene"] == "field":
        c["instances"] = _log(rng, 8, 256)
    return c


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=1)
def _blob():
    """The unit icosphere of the field (5 120 triangles) and, per vertex, the faces around it (six at most; the
    twelve of the icosahedron have five, their sixth entry points past the last face)."""
    unit, faces = scenes.icosphere(5)
    around = np.full((unit.shape[0], 6), faces.shape[0], np.int64)
    used = np.zeros(unit.shape[0], np.int64)
    for f, tri in enumerate(faces):
        for v in tri:
            around[v, used[v]] = f
            used[v] += 1
    return unit.astype(np.float32), faces, around


def _blobs(count, seed, phase=0.0):
    """`count` displaced icospheres at unit size with smooth normals, (count, vertices, 3) each."""
    unit, faces, around = _blob()
    rng = np.random.default_rng([seed, 11])
    freqs = rng.normal(0.0, 3.0, (count, 3, 3)).astype(np.float32)
    shift = rng.uniform(0, 2 * np.pi, (count, 3)).astype(np.float32) + np.float32(phase)
    amps = rng.uniform(0.03, 0.08, (count, 3)).astype(np.float32)
    disp = 1.0 + (amps[:, None, :] * np.sin(np.einsum("vk,cjk->cvj", unit, freqs) + shift[:, None, :])).sum(2)
    pos = torch.from_numpy(unit[None] * disp[:, :, None].astype(np.float32)).cuda()
    f = torch.from_numpy(faces).cuda()
    p0, p1, p2 = pos[:, f[:, 0]], pos[:, f[:, 1]], pos[:, f[:, 2]]
    fn = torch.cat([torch.linalg.cross(p1 - p0, p2 - p0), torch.zeros(count, 1, 3, device="cuda")], 1)
    nrm = torch.nn.functional.normalize(fn[:, torch.from_numpy(around).cuda()].sum(2), dim=2)
    return pos.cpu().numpy(), nrm.cpu().numpy()


def _hdri(width, seed):
    rng = np.random.default_rng([seed, 5])
    az, el = rng.uniform(0, 2 * np.pi), rng.uniform(0.4, 0.9)
    sun = (math.cos(el) * math.sin(az), math.sin(el), math.cos(el) * math.cos(az))
    return scenes.procedural_hdri(width, width // 2, seed, sun_dir=sun)


def _surfaces(count, rng):
    mats = []
    for _ in range(count):
        base = tuple(float(x) for x in rng.uniform(0.05, 0.95, 3))
        mats.append(standard_surface(base, float(rng.uniform(0.05, 1.0)), 1.0 if rng.random() < 0.3 else 0.0, 1.5))
    return mats


def _field(instances, env, seed, phase=0.0, plane=50.0):
    rng = np.random.default_rng([seed, 3])
    mats = _surfaces(64, rng) + [lambert((0.5, 0.5, 0.5))]
    pos, nrm = _blobs(instances, seed, phase)
    idx = _blob()[1].astype(np.uint32).reshape(-1)
    h = plane * 0.5 - 1.5
    meshes = []
    for k in range(instances):
        r = float(rng.uniform(0.4, 1.2))
        x, z = rng.uniform(-h, h, 2)
        at = np.array([x, r * 0.85, z], np.float32)
        meshes.append(Mesh(pos[k] * np.float32(r) + at, idx, nrm[k], int(rng.integers(0, 64))))
    meshes.append(Mesh(*_ground(plane), 64))
    return Scene(materials=mats, meshes=meshes, dome_lights=[DomeLight(env=_hdri(env, seed))],
                 distant_lights=[DistantLight(direction=(-0.3, -1.0, -0.4), radiance=(2.5, 2.4, 2.2))])


def _ground(size):
    p, n, i = scenes.ground_quad(size)
    return p, i, n


@functools.lru_cache(maxsize=4)
def _ball(segments, rings):
    return scenes.uv_sphere((0.0, 0.0, 0.0), 1.0, segments, rings)


def _sphere_at(center, radius, material, segments=64, rings=32):
    p, n, i = _ball(segments, rings)
    return Mesh(p * np.float32(radius) + np.asarray(center, np.float32), i, n, material)


def _sphere(env, seed):
    rng = np.random.default_rng([seed, 1])
    mats = [usd_preview_surface(diffuse_color=tuple(float(x) for x in rng.uniform(0.5, 0.9, 3)),
                                roughness=float(rng.uniform(0.2, 0.5))), lambert((0.5, 0.5, 0.5))]
    return Scene(materials=mats, meshes=[_sphere_at((0.0, 1.0, 0.0), 1.0, 0), Mesh(*_ground(10.0), 1)],
                 dome_lights=[DomeLight(env=_hdri(env, seed))])


def _parts(materials, env, seed):
    """The sphere scene cut into `materials` meshes with a material each (the ground is the last)."""
    rng = np.random.default_rng([seed, 4])
    p, n, i = _ball(64, 32)
    meshes, mats = [], []
    for k, tri in enumerate(np.array_split(i.reshape(-1, 3), max(1, materials - 1))):
        used, inv = np.unique(tri.reshape(-1), return_inverse=True)
        meshes.append(Mesh(p[used] + np.array([0, 1, 0], np.float32), inv.astype(np.uint32).reshape(-1), n[used], k))
    meshes.append(Mesh(*_ground(10.0), len(meshes)))
    for _ in meshes:
        mats.append(standard_surface(tuple(float(x) for x in rng.uniform(0.05, 0.95, 3)), float(rng.uniform(0.05, 1.0)),
                                     float(rng.uniform(0.0, 1.0)), 1.5))
    return Scene(materials=mats, meshes=meshes, dome_lights=[DomeLight(env=_hdri(env, seed))])


def _studio(env, seed):
    rng = np.random.default_rng([seed, 2])
    tint = lambda: tuple(float(x) for x in rng.uniform(0.2, 0.9, 3))  # noqa: E731
    mats = [
        standard_surface((1.0, 1.0, 1.0), 0.0, 0.0, 1.5, transmission=1.0),
        standard_surface((1.0, 1.0, 1.0), 0.25, 0.0, 1.45, transmission=0.9, transmission_extra_roughness=0.1),
        standard_surface((1.0, 1.0, 1.0), 0.0, 0.0, 1.33, transmission=1.0, transmission_color=(0.5, 0.8, 0.9),
                         transmission_depth=0.8, transmission_scatter=(0.3, 0.1, 0.05)),
        standard_surface((1.0, 1.0, 1.0), 0.1, 0.0, 1.5, transmission=0.8, thin_walled=True,
                         transmission_color=(0.9, 0.95, 1.0)),
        standard_surface(tint(), 0.3, 0.0, 1.5, coat_weight=1.0, coat_roughness=0.1, coat_affect_color=0.5),
        standard_surface(tint(), 0.4, 1.0, 1.5, specular_anisotropy=0.6, specular_rotation=0.2),
        standard_surface(tint(), 0.5, 0.0, 1.5, sheen=0.8, diffuse_roughness=0.5),
        standard_surface(tint(), 0.2, 0.0, 1.5, thin_film_thickness=450.0, subsurface=0.4),
        usd_preview_surface(tint(), 0.4, opacity=0.45),
        Material(emission_color=(1.0, 0.85, 0.6), emission_strength=6.0, base_color=(0.1, 0.1, 0.1)),
        lambert((0.55, 0.5, 0.45)),
    ]
    meshes = []
    for k in range(9):
        r = float(rng.uniform(0.45, 0.6))
        meshes.append(_sphere_at(((k % 3 - 1) * 1.4, r, (k // 3 - 1) * 1.4), r, k))
    lamp, n, i = scenes.ground_quad(1.5, 3.2)
    meshes.append(Mesh(lamp, i.reshape(-1, 3)[:, ::-1].copy().reshape(-1), -n, 9))  # faces down
    meshes.append(Mesh(*_ground(12.0), 10))
    return Scene(materials=mats, meshes=meshes, dome_lights=[DomeLight(env=_hdri(env, seed))],
                 distant_lights=[DistantLight(direction=(-0.4, -1.0, -0.3), radiance=(1.5, 1.4, 1.3))])


def _scene(case, seed, phase=0.0):
    if case["scene"] == "field":
        return _field(case["instances"], case["env"], seed, phase)
    if case["scene"] == "parts":
        return _parts(case["materials"], case["env"], seed)
    return (_studio if case["scene"] == "studio" else _sphere)(case["env"], seed)


def _camera(kind, seed, aspect):
    rng = np.random.default_rng([seed, 9])
    az = rng.uniform(0, 2 * np.pi)
    dist, high, look = {"field": (36.0, 14.0, (0.0, 0.0, 0.0)), "studio": (5.5, 2.4, (0.0, 0.5, 0.0))}.get(
        kind, (4.5, 1.6, (0.0, 0.9, 0.0)))
    dist, high = dist * rng.uniform(0.9, 1.1), high * rng.uniform(0.9, 1.1)
    return scenes.look_at((dist * math.sin(az), high, dist * math.cos(az)), look, 45.0, aspect)


def _settings(width, height, spp, depth):
    return RenderSettings(width=width, height=height, samples_per_pixel=spp, max_depth=depth, diffuse_depth=depth,
                          specular_depth=depth, dome_light_samples=1, background_visible=True, backend=1)


def _planes(fb):
    return {"beauty": fb.beauty, "albedo": fb.albedo, "normal": fb.normal, "depth": fb.depth}


# ---------------------------------------------------------------------------
# a case's inputs and one pass
# ---------------------------------------------------------------------------

def _view_requests(case, seed):
    """Square views of log-uniform size up to `size`, samples and depth up to the case's, orbiting cameras.  The sizes
    belong to the case (the same for every seed), so that a pass costs the same whatever the inputs."""
    sizes = np.random.default_rng([case["requests"], case["size"], 6])
    out = []
    for k in range(case["requests"]):
        s = int(round(math.exp(sizes.uniform(math.log(96), math.log(case["size"])))))
        spp = int(sizes.choice([x for x in (4, 16, 64) if x <= case["spp"]]))
        depth = int(sizes.choice([x for x in (4, 8, 12) if x <= case["depth"]]))
        out.append((_camera("sphere", 1000 * seed + k, 1.0), _settings(s, s, spp, depth)))
    return out


def _frames_in_one(settings):
    """Frame buffers of all views inside four page-locked planes, as a service that ships whole batches keeps them."""
    total = sum(s.width * s.height for s in settings)
    planes = {k: torch.empty((total, n), dtype=torch.float32, pin_memory=True).numpy()
              for k, n in (("beauty", 4), ("albedo", 3), ("normal", 3), ("depth", 1))}
    frames, at = [], 0
    for s in settings:
        f = FrameBuffer(0, 0)
        f.width, f.height = s.width, s.height
        for k, p in planes.items():
            view = p[at:at + s.width * s.height]
            setattr(f, k, view[:, 0] if k == "depth" else view)
        at += s.width * s.height
        frames.append(f)
    return planes, frames


def _parameters(scene, seed, steps):
    """`steps` parameter sets around the scene's own, as successive optimiser steps give them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    base = torch.tensor([m.base_color for m in scene.materials], dtype=torch.float32, device="cuda")
    rough = torch.tensor([m.roughness for m in scene.materials], dtype=torch.float32, device="cuda")
    metal = torch.tensor([m.metallic for m in scene.materials], dtype=torch.float32, device="cuda")
    env = torch.from_numpy(scene.dome_lights[0].env).cuda()
    out = []
    for _ in range(steps):
        r = lambda t: 0.05 * (torch.rand(t.shape, generator=g, device="cuda") - 0.5)  # noqa: E731
        p = [(base + r(base)).clamp(0.02, 0.98), (rough + r(rough)).clamp(0.05, 1.0), (metal + r(metal)).clamp(0.0, 1.0),
             env * (1.0 + r(env))]
        out.append([t.contiguous().requires_grad_() for t in p])
    return out


def _edited(scene, seed, k):
    """The scene with other materials, lights and environment exposure; the meshes are the same arrays."""
    rng = np.random.default_rng([seed, 21, k])
    s = float(rng.uniform(0.5, 1.5))
    sun = tuple(float(x) for x in rng.uniform(1.0, 3.0, 3))
    return Scene(materials=_surfaces(64, rng) + [scene.materials[-1]], meshes=scene.meshes,
                 dome_lights=[DomeLight(env=scene.dome_lights[0].env * np.float32(s))],
                 distant_lights=[DistantLight(direction=(-0.3, -1.0, float(rng.uniform(-0.6, 0.6))), radiance=sun)])


def _rays(scene, count, seed):
    """Rays from around the model to points inside its triangles, with reaches on both sides of the hit."""
    rng = np.random.default_rng([seed, 8])
    tri = np.concatenate([m.positions[m.indices.reshape(-1, 3)] for m in scene.meshes]).astype(np.float64)
    b = rng.dirichlet((4.0, 4.0, 4.0), count)
    target = (tri[rng.integers(0, tri.shape[0], count)] * b[:, :, None]).sum(1)
    az, el = rng.uniform(0, 2 * np.pi, count), rng.uniform(0.1, 1.3, count)
    o = 6.0 * np.stack([np.cos(el) * np.sin(az), np.sin(el), np.cos(el) * np.cos(az)], 1)
    d = target - o
    dist = np.linalg.norm(d, axis=1, keepdims=True)
    reach = (dist[:, 0] * rng.uniform(0.5, 1.5, count)).astype(np.float32)
    return o.astype(np.float32), (d / dist).astype(np.float32), reach


def prepare(case, seed):
    kind, gpu = case["kind"], GpuBackend(0)
    st = {"case": case, "gpu": gpu}
    scene = st["scene"] = _scene(case, seed)
    if kind == "rays":
        st["rays"] = _rays(scene, case["rays"], seed)
    elif kind == "views":
        st["requests"] = _view_requests(case, seed)
        st["planes"], st["frames"] = _frames_in_one([s for _, s in st["requests"]])
    else:
        st["settings"] = _settings(case["width"], case["height"], case["spp"], case["depth"])
        st["camera"] = _camera(case["scene"], seed, case["width"] / case["height"])
        if kind in ("frame", "animate", "relight", "viewport"):
            count = 2 if kind in ("animate", "relight") else 1
            st["frames"] = [FrameBuffer(case["width"], case["height"], pinned=True) for _ in range(count)]
        if kind == "viewport":
            st["accumulator"] = gpu.accumulator()
        if kind == "gradient":
            st["parameters"] = _parameters(scene, seed, case["steps"])
            g = torch.Generator(device="cuda").manual_seed(seed + 1)
            st["target"] = torch.rand((case["height"], case["width"], 3), generator=g, device="cuda")
        if kind == "animate":
            st["scenes"] = [scene, _scene(case, seed, 0.3)]
        if kind == "relight":
            st["scenes"] = [_edited(scene, seed, k) for k in range(2)]
    gpu.upload_scene(scene)
    return st


def run(state):
    case, gpu, kind = state["case"], state["gpu"], state["case"]["kind"]
    scene = state["scene"]
    if kind == "rays":
        prim, t, occluded = gpu.trace_rays(scene, *state["rays"])
        return {"prim": prim, "t": t, "occluded": occluded}
    if kind == "views":
        gpu.render_batch(scene, state["requests"], outs_fb=state["frames"])
        return state["planes"]
    camera, settings = state["camera"], state["settings"]
    if kind == "preview":
        return _planes(gpu.render_sample_batch(RenderRequest(scene, camera, settings, 0, case["spp"])))
    if kind == "viewport":
        acc = state["accumulator"]
        for k in range(case["steps"]):
            acc.render_step(scene, camera, settings, k * case["spp"], case["spp"], wavefront=case["wavefront"])
        return _planes(acc.resolve(state["frames"][0]))
    if kind == "frame":
        (fb,) = gpu.render_batch(scene, [(camera, settings)], outs_fb=state["frames"])
        return _planes(fb)
    if kind == "plain":
        return _planes(gpu.render(scene, camera, settings))
    if kind == "gradient":
        from shiro_gb300.autograd import render

        out = []
        for p in state["parameters"]:
            img = render(gpu, camera, settings, *p, adjoint_sample_start=case["spp"] if case["decorrelate"] else None)
            loss = (img[..., :3] - state["target"]).square().mean()
            out.append([img.detach(), *torch.autograd.grad(loss, p)])
        return out
    out = []
    for s, fb in zip(state["scenes"], state["frames"]):  # animate, relight
        gpu.render_batch(s, [(camera, settings)], outs_fb=[fb])
        out.append(_planes(fb))
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it should return
# ---------------------------------------------------------------------------

def _scene_bytes(case):
    tri = {"field": 5120 * case.get("instances", 0) + 2, "studio": 9 * 3968 + 4}.get(case["scene"], 3970)
    # positions and normals (24 bytes a vertex, half a vertex a triangle), indices; environment texels
    return tri * (12 + 12) + case["env"] * (case["env"] // 2) * 12


def work(case):
    kind, scene = case["kind"], _scene_bytes(case)
    if kind == "rays":
        return {"bytes": scene + case["rays"] * 40.0, "flops": case["rays"] * FLOPS_PER_RAY}
    per = FLOPS_PER_PATH[case["scene"]]
    if kind == "views":
        rs = [s for _, s in _view_requests(case, 0)]
        return {"bytes": scene + float(sum(s.width * s.height for s in rs)) * PIXEL_BYTES,
                "flops": float(sum(s.width * s.height * s.samples_per_pixel for s in rs)) * per}
    px = float(case["width"] * case["height"])
    if kind == "gradient":
        # forward paths (the replayed range too when it is another one) and their replay with derivatives
        forward = 2 if case["decorrelate"] else 1
        params = 12.0 * case["env"] * (case["env"] // 2)
        return {"bytes": case["steps"] * (scene + 2 * px * 16 + 2 * params),
                "flops": case["steps"] * px * case["spp"] * (forward + 1.0) * per}
    frames = 2 if kind in ("animate", "relight") else 1
    steps = case.get("steps", 1)
    return {"bytes": frames * (scene + px * PIXEL_BYTES), "flops": frames * steps * px * case["spp"] * per}


def exact(case, seed):
    """Hit distances of the caller's rays, by testing every triangle in 64 bits.  The other cases have no such value
    within seconds: a frame is a Monte Carlo estimate whose paths branch on the last bits of 32-bit arithmetic, and
    which path is taken is part of what they return."""
    if case["kind"] != "rays":
        return None
    scene = _scene(case, seed)
    o, d, _ = _rays(scene, case["rays"], seed)
    tri = torch.from_numpy(np.concatenate([m.positions[m.indices.reshape(-1, 3)] for m in scene.meshes])).double().cuda()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    best = []
    for a in range(0, case["rays"], 4096):
        ro, rd = (torch.from_numpy(x[a:a + 4096]).double().cuda()[:, None] for x in (o, d))
        pv = torch.linalg.cross(rd.expand(-1, e2.shape[0], -1), e2[None].expand(rd.shape[0], -1, -1))
        det = (e1 * pv).sum(2)
        tv = ro - p0
        u = (tv * pv).sum(2) / det
        qv = torch.linalg.cross(tv, e1[None].expand(rd.shape[0], -1, -1))
        v = (rd * qv).sum(2) / det
        t = (e2 * qv).sum(2) / det
        ok = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= 1e-4)
        best.append(torch.where(ok, t, float(np.finfo(np.float32).max)).amin(1))
    return {"prim": None, "t": torch.cat(best), "occluded": None}
