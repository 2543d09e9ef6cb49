"""The calls that the library's performance is followed on: whole passes through its public Python API.

A pass is one call as a user's program makes it, on scenes made from a seed:

  render    one image into device buffers (`DeviceScene.render_device`), scene resident;
  batch     many images through one wavefront (`Context.render_batch`);
  serve     a burst of requests to a render server, waited for in order (`RenderServer`);
  closest   closest hits of a host array of rays (`DeviceScene.trace_closest`);
  launch    the reference's launchGPU pattern: world built, image rendered to host buffers, world dropped.

`listed()` are the calls followed by name; `draw()` gives others from the same ranges: images of 64 to
1,920 pixels a side, odd sizes among them, 1 to 64 samples, depths of 4 to 50, scenes of 20 primitives to
1.3 million triangles, both modes and draw orders, both node layouts, sample groups, environment sampling.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cortexraytracercuda_b200 import configs
from cortexraytracercuda_b200.renderer import Context, DeviceScene, Job, RenderServer
from cortexraytracercuda_b200.scene import (BVH_DEVICE, BVH_SAH, DRAW_ORDER_DEVICE, DRAW_ORDER_HOST,
                                            FLAG_ENV_SAMPLING, FLAG_SAMPLE_GROUPS, FLAG_WIDE_BVH, MODE_CLEAN,
                                            MODE_COMPAT, RenderParams)

# a path's mean number of rays and the primitives of each scene, for work()
_SCENES = {
    #            rays a path, primitives (of mesh level l: a function)
    "cornell":   (4.0, lambda l: 30),
    "spheres":   (3.8, lambda l: 489),
    "meshes":    (2.6, lambda l: 4 * 20 * 4 ** l + 2),
    "textured":  (2.6, lambda l: 6),
    "icosphere": (2.6, lambda l: 3 * 20 * 4 ** l + 2),
    "lights":    (2.6, lambda l: 328),
    "uvmesh":    (2.4, lambda l: 3842),
    "xforms":    (4.0, lambda l: 350),
    "batch":     (3.0, lambda l: 70000),
}


def _case(kind, scene, w=0, h=0, spp=0, depth=0, *, level=3, mode="compat", order="device", groups=False, env=False,
          wide=False, rgb8=False, bvh="sah", n=0, name=None):
    c = dict(kind=kind, scene=scene, width=w, height=h, spp=spp, depth=depth, level=level, mode=mode, order=order,
             groups=groups, env=env, wide=wide, rgb8=rgb8, bvh=bvh, n=n)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # a thumbnail / first preview of a small textured scene, with its 8-bit image: latency and launches
        _case("render", "textured", 64, 48, 4, 10, rgb8=True, name="preview"),
        # the Cornell box at the size the reference's own example renders it
        _case("render", "cornell", 256, 256, 16, 8, name="cornell"),
        # the flagship frame: 489 spheres with defocus, glass chains up to 50 bounces
        _case("render", "spheres", 1280, 720, 64, 50, name="spheres"),
        # the same scene in clean mode with sample groups, as an interactive viewer renders it
        _case("render", "spheres", 960, 540, 16, 16, mode="clean", groups=True, name="spheres_clean"),
        # every light type at an odd size, the g++ build's draw order and arithmetic
        _case("render", "lights", 641, 479, 16, 10, order="host", name="lights_host"),
        # transformed boxes, spheres and meshes (the second BVH), clean mode, ragged size
        _case("render", "xforms", 333, 251, 32, 8, mode="clean", name="transforms"),
        # a large triangle scene at full HD: 1.31 M triangles, environment map, textures
        _case("render", "meshes", 1920, 1080, 16, 16, level=7, name="meshes"),
        # a mid-size triangle scene with importance-sampled sky and the 8-wide nodes
        _case("render", "meshes", 1280, 720, 8, 12, level=5, mode="clean", env=True, wide=True, name="meshes_env"),
        # a batch of different scenes, cameras and sizes, as an offline queue submits it
        _case("batch", "batch", 320, 240, 16, 20, n=16, name="batch"),
        # a burst of requests to a running server
        _case("serve", "batch", 320, 240, 8, 12, mode="clean", groups=True, n=12, name="serve"),
        # ray queries (picking, visibility, collision) against a resident mesh, host arrays in and out
        _case("closest", "icosphere", level=5, n=200_003, name="closest"),
        # a launchGPU call: build the world on the device, render, read the image back, drop it
        _case("launch", "icosphere", 300, 200, 16, 12, level=6, bvh="device", rgb8=True, name="launch"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["render"] * 6 + ["batch", "serve", "closest", "launch"])
        mode = rng.choice(["compat", "compat", "clean"])
        order = rng.choice(["device", "device", "device", "host"]) if mode == "compat" else "device"
        groups = mode == "clean" and rng.random() < 0.5
        w = _log(rng, 64, 1920)
        h = max(36, int(w * rng.uniform(0.5, 1.0)))
        spp, depth = _log(rng, 1, 64), _log(rng, 4, 50)
        rgb8 = rng.random() < 0.3
        if kind == "render":
            scene = rng.choice(["cornell", "spheres", "spheres", "meshes", "meshes", "textured", "icosphere", "lights",
                                "uvmesh", "xforms"])
            level = rng.randint(4, 7) if scene == "meshes" else rng.randint(2, 6)
            c = _case(kind, scene, w, h, spp, depth, level=level, mode=mode, order=order, groups=groups,
                      env=mode == "clean" and scene == "meshes" and rng.random() < 0.5, wide=rng.random() < 0.2, rgb8=rgb8)
            # one slot per work unit, so that the image does not depend on which slot took which pixel
            if w * h * (min(8, spp) if groups else 1) > 1 << 22:
                continue
        elif kind == "batch":
            n = rng.randint(3, 24)
            w, h = min(w, 512), min(h, 384)
            if n * w * h > 1 << 21:
                continue
            c = _case(kind, "batch", w, h, spp, depth, mode=mode, order=order, n=n)
        elif kind == "serve":
            c = _case(kind, "batch", min(w, 512), min(h, 384), min(spp, 16), depth, mode=mode, order=order, groups=groups,
                      n=rng.randint(2, 20))
        elif kind == "closest":
            c = _case(kind, rng.choice(["spheres", "icosphere", "lights", "uvmesh"]), level=rng.randint(2, 5),
                      wide=rng.random() < 0.3, n=_log(rng, 500, 400_000))
        else:
            c = _case(kind, rng.choice(["cornell", "spheres", "textured", "icosphere", "lights"]), min(w, 640), min(h, 480),
                      min(spp, 16), min(depth, 16), level=rng.randint(3, 6), mode=mode, order=order, rgb8=rgb8,
                      bvh=rng.choice(["sah", "device"]))
        if _cost(c) <= top:
            return c


# ---- what a program has in hand ------------------------------------------------------------------

_CTX = None
_SERVERS = {}
_RESIDENT = {}


def _ctx():
    """One context per process, as a program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = Context(0)
    return _CTX


def _resident(k):
    """Scene k of the batched workload, resident on the device for as long as the program runs."""
    if k not in _RESIDENT:
        s, _ = configs.batch_scene(k)
        _RESIDENT[k] = (DeviceScene(_ctx(), s), s.camera)
    return _RESIDENT[k]


def _server(mode, order, flags, n):
    """A running server and the ids of its first n scenes."""
    if (mode, order, flags) not in _SERVERS:
        _SERVERS[mode, order, flags] = (RenderServer(0, mode=mode, draw_order=order, flags=flags, hbm_budget_bytes=8 << 30), [])
    server, ids = _SERVERS[mode, order, flags]
    while len(ids) < n:
        s, _ = configs.batch_scene(len(ids))
        ids.append((server.add_scene(s), s.camera))
    return server, ids


def _scene(case, seed):
    """The case's scene; geometry, materials, light or view differ from seed to seed."""
    rng = np.random.default_rng([7, int(seed)])
    name, level = case["scene"], case["level"]
    if name == "cornell":
        s = configs.cornell(light_intensity=float(rng.uniform(0.8, 1.2)))
        center = (278.0, 278.0, 0.0)
    elif name == "meshes":
        s = configs.meshes(level, seed=int(seed), env_size=(1024, 512))
        center = (0.0, 0.9, 0.0)
    elif name == "icosphere":
        s = configs.icosphere_scene(level, seed=int(seed))
        center = (0.0, 1.0, 0.0)
    elif name == "xforms":
        s = configs.transforms_scene(seed=int(seed))
        center = (278.0, 278.0, 0.0)
    else:
        make = {"spheres": configs.spheres, "textured": configs.textured, "lights": configs.lights_scene,
                "uvmesh": configs.uv_mesh_scene}[name]
        s = make(seed=int(seed))
        center = s.camera.look_at
    s.camera = configs.orbit_camera(s.camera, float(rng.uniform(-0.1, 0.1)), center)
    if case["width"]:
        s.camera.aspect = case["width"] / case["height"]
    return s


def _params(case, seed, w=None, h=None):
    flags = ((FLAG_SAMPLE_GROUPS if case["groups"] else 0) | (FLAG_ENV_SAMPLING if case["env"] else 0) |
             (FLAG_WIDE_BVH if case["wide"] else 0))
    return RenderParams(width=w or case["width"], height=h or case["height"], spp=case["spp"], max_depth=case["depth"],
                        seed=int(seed) * 7919 % 1_000_003 + 11,
                        mode=MODE_CLEAN if case["mode"] == "clean" else MODE_COMPAT,
                        draw_order=DRAW_ORDER_HOST if case["order"] == "host" else DRAW_ORDER_DEVICE, flags=flags)


def _bvh(case):
    return BVH_DEVICE if case["bvh"] == "device" else BVH_SAH


def _views(case, seed, cameras):
    """Cameras and parameters of a batch or a burst: every other image is the case's size, the others
    are smaller and ragged; each is seen from an angle of its own."""
    rng = np.random.default_rng([11, int(seed)])
    out = []
    for k, (cam, (w, h)) in enumerate(zip(cameras, _sizes(case))):
        cam = configs.orbit_camera(cam, float(rng.uniform(0.0, 2.0 * math.pi)))
        cam.aspect = w / h
        out.append((cam, _params(case, int(seed) + 31 * k, w, h)))
    return out


def _sizes(case):
    rng = np.random.default_rng(case["n"])   # the sizes are the same for every seed
    f = [1.0 if k % 2 == 0 else float(rng.uniform(0.4, 1.0)) for k in range(case["n"])]
    return [(max(16, int(case["width"] * x)), max(16, int(case["height"] * x))) for x in f]


def _rays(case, scene, seed):
    """Rays from around the scene towards it, and bounce-like rays from inside it."""
    rng = np.random.default_rng([13, int(seed)])
    n, cam = case["n"], scene.camera
    eye, at = np.asarray(cam.look_from, np.float64), np.asarray(cam.look_at, np.float64)
    dist = np.linalg.norm(eye - at)
    o = np.where(rng.random((n, 1)) < 0.5, eye + rng.normal(size=(n, 3)) * 0.02 * dist,
                 at + rng.uniform(-0.4, 0.4, (n, 3)) * dist)
    d = at + rng.normal(size=(n, 3)) * 0.15 * dist - o
    r = np.empty((n, 8), np.float32)
    r[:, 0:3], r[:, 3] = o, 1e-4
    r[:, 4:7], r[:, 7] = d / np.linalg.norm(d, axis=1, keepdims=True), 3e38
    return r


def prepare(case, seed):
    kind = case["kind"]
    if kind == "render":
        st = dict(case=case, scene=DeviceScene(_ctx(), _scene(case, seed), _bvh(case)), params=_params(case, seed))
        st["out"] = torch.empty(case["height"], case["width"], 4, device="cuda")
        st["rgb"] = torch.empty(case["height"], case["width"], 3, dtype=torch.uint8, device="cuda") if case["rgb8"] else None
        return st
    if kind == "batch":
        jobs, outs = [], []
        scenes = [_resident(k) for k in range(case["n"])]
        for (scene, _), (cam, p) in zip(scenes, _views(case, seed, [c for _, c in scenes])):
            outs.append(torch.empty(p.height, p.width, 4, device="cuda"))
            jobs.append(Job(scene, p, outs[-1].data_ptr(), cam))
        return dict(case=case, jobs=jobs, outs=outs)
    if kind == "serve":
        p = _params(case, seed)
        server, ids = _server(p.mode, p.draw_order, p.flags, case["n"])
        views = _views(case, seed, [c for _, c in ids[:case["n"]]])
        return dict(case=case, server=server,
                    reqs=[(sid, p, cam, np.empty((p.height, p.width, 4), np.float32))
                          for (sid, _), (cam, p) in zip(ids, views)])
    if kind == "closest":
        s = _scene(case, seed)
        return dict(case=case, scene=DeviceScene(_ctx(), s), rays=_rays(case, s, seed))
    return dict(case=case, world=_scene(case, seed), params=_params(case, seed))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "render":
        st["scene"].render_device(st["params"], st["out"].data_ptr(), st["rgb"].data_ptr() if case["rgb8"] else None)
        return [st["out"], st["rgb"]] if case["rgb8"] else [st["out"]]
    if kind == "batch":
        _ctx().render_batch(st["jobs"])
        return st["outs"]
    if kind == "serve":
        tickets = [st["server"].submit(sid, p, cam, out)[0] for sid, p, cam, out in st["reqs"]]
        return [st["server"].wait(t)[0] for t in tickets]
    if kind == "closest":
        prim, t = st["scene"].trace_closest(st["rays"], flags=FLAG_WIDE_BVH if case["wide"] else 0)
        return [prim, t]
    ds = DeviceScene(_ctx(), st["world"], _bvh(case))
    try:
        rad, rgb = ds.render(st["params"], want_rgb8=case["rgb8"])
    finally:
        ds.close()
    return [rad, rgb] if case["rgb8"] else [rad]


# ---- what a pass cannot do without ---------------------------------------------------------------

def _pixels(case):
    if case["kind"] in ("batch", "serve"):
        return sum(w * h for w, h in _sizes(case))
    return case["width"] * case["height"]


def _ray_count(case):
    if case["kind"] == "closest":
        return float(case["n"])
    spp = case["spp"] if case["mode"] == "clean" else math.isqrt(case["spp"]) ** 2
    return _pixels(case) * spp * min(_SCENES[case["scene"]][0], float(case["depth"]))


def work(case):
    """Scene read once, images (or rays and hits) moved once; per ray the box tests of a walk down a
    balanced binary tree and back into one sibling path (24 operations a node), two primitive tests and
    one bounce of shading."""
    prims = _SCENES[case["scene"]][1](case["level"])
    images = case["n"] if case["kind"] in ("batch", "serve") else 1
    per_ray = 24 * 2 * max(1.0, math.log2(prims)) + 2 * 30 + (0 if case["kind"] == "closest" else 150)
    moved = 40 * case["n"] if case["kind"] == "closest" else _pixels(case) * (19 if case["rgb8"] else 16)
    return {"bytes": float(moved + images * prims * 48), "flops": float(_ray_count(case) * per_ray)}


def _cost(case):
    w = work(case)
    return w["flops"] + 4.0 * w["bytes"]


# ---- what the outputs are in 64 bits -------------------------------------------------------------

def exact(case, seed):
    """Hit distances of `closest`: every ray against every primitive in double precision.  (A rendered
    image has no such value: its random walk is decided by float roundings, sample by sample.)"""
    if case["kind"] != "closest":
        return None
    s = _scene(case, seed)
    tris = _triangles(s)
    rays = _rays(case, s, seed)
    if case["n"] * (len(tris) + 1) > 4e10:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    R = torch.from_numpy(rays.astype(np.float64)).to(dev)
    T = torch.full((len(rays),), math.inf, dtype=torch.float64, device=dev)
    tri = torch.from_numpy(tris).to(dev)
    sph = torch.tensor(_spheres(s), dtype=torch.float64, device=dev).reshape(-1, 4)
    par = _parallelograms(s, dev)
    step = max(1, int(4e7 // max(1, len(tris) + len(sph) + len(par))))
    for a in range(0, len(rays), step):
        r = R[a:a + step]
        o, d, lo = r[:, None, 0:3], r[:, None, 4:7], r[:, None, 3]
        best = torch.full((len(r),), math.inf, dtype=torch.float64, device=dev)
        if len(sph):
            oc = o - sph[None, :, 0:3]
            A, B = (d * d).sum(-1), (oc * d).sum(-1)
            disc = B * B - A * ((oc * oc).sum(-1) - sph[None, :, 3] ** 2)
            q = disc.clamp_min(0).sqrt()
            t0, t1 = (-B - q) / A, (-B + q) / A
            t = torch.where(t0 > lo, t0, torch.where(t1 > lo, t1, math.inf))
            best = torch.minimum(best, torch.where(disc >= 0, t, math.inf).amin(1))
        for g, inside in ((tri, "triangle"), (par, "parallelogram")):
            if len(g):
                best = torch.minimum(best, _planar(o, d, lo, g[None], inside))
        T[a:a + step] = best
    return [None, T]


def _planar(o, d, lo, g, inside):
    """Least t over triangles or parallelograms g = (corner, edge 1, edge 2)."""
    v0, e1, e2 = g[..., 0:3], g[..., 3:6], g[..., 6:9]
    n = torch.linalg.cross(e1, e2)
    den = (n * d).sum(-1)
    t = (n * (v0 - o)).sum(-1) / den
    p = o + t[..., None] * d - v0
    nn = (n * n).sum(-1)
    u = (torch.linalg.cross(p, e2.expand_as(p)) * n).sum(-1) / nn
    v = (torch.linalg.cross(e1.expand_as(p), p) * n).sum(-1) / nn
    ok = (den != 0) & (t >= lo) & (u >= 0) & (v >= 0)
    ok &= (u + v <= 1) if inside == "triangle" else (u <= 1) & (v <= 1)
    return torch.where(ok, t, math.inf).amin(1)


def _triangles(s):
    out = [np.zeros((0, 9))]
    for m in s.meshes:
        v, f = np.asarray(m["vertices"], np.float64), np.asarray(m["indices"])
        a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
        out.append(np.concatenate([a, b - a, c - a], axis=1))
    return np.concatenate(out)


def _spheres(s):
    return ([(*c, r) for c, r, _ in s.spheres] + [(*l[0], l[1]) for l in s.omni_lights] +
            [(*l[0], l[5]) for l in s.spot_lights])


def _parallelograms(s, dev):
    g = [(*q, *u, *v) for q, u, v, _ in s.quads]
    for l in s.dir_lights:   # a light's position is its centre
        p, u, v = (np.asarray(x, np.float64) for x in l[0:3])
        g.append((*(p - 0.5 * u - 0.5 * v), *u, *v))
    return torch.tensor(g, dtype=torch.float64, device=dev).reshape(-1, 9)
