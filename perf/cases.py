"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict of plain values; prepare() makes what a program holds before the call (a
context with its scene, device or page-locked buffers, a tuned ray-query variant, a radiance
cache, a batch), run() is one pass through the public entry points, work() what a pass cannot
do without. Contexts hold a scene and its path buffers for as long as a program renders it, so
they are made once per scene and shared by the states of a case; rays, films and seeds are each
state's own.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "ray-based-rendering_b200"))

from rbr_b200 import Batch, Context, abi, render_params, scenes  # noqa: E402

# Primitives of each scene, for work(): triangles, spheres, quads, planes.
PRIMITIVES = {"world": 261, "cornell": 18, "fog": 18, "ico6": 81920, "ico8": 1310720, "ggx100": 20259,
              "ggx1000": 2000259}


def listed():
    return [
        # One short query batch of an interactive tool (picking, collision probes): latency of a launch.
        dict(name="closest_small", kind="rays", scene="world", rays="test", n=1001, any_hit=False, tuned=False),
        # Primary visibility of a full-HD frame (depth, normal and AO passes): coherent camera rays,
        # on a context as it is created.
        dict(name="closest_camera", kind="rays", scene="ggx1000", rays="camera", n=1920 * 1080, any_hit=False,
             tuned=False),
        # The benchmark's ray queries: incoherent rays through a large mesh, variant tuned on the rays.
        dict(name="closest_uniform", kind="rays", scene="ico8", rays="uniform", n=1 << 22, any_hit=False, tuned=True),
        # Visibility segments towards the area lights (light baking, occlusion), an odd number of them.
        dict(name="any_shadow", kind="rays", scene="ggx1000", rays="shadow", n=1500001, any_hit=True, tuned=True),
        # A batch of rays kept in host memory, as the C++ accelerator adapter passes them.
        dict(name="closest_host", kind="host_rays", scene="ico8", rays="uniform", n=1 << 21, any_hit=False, tuned=True),
        # An interactive preview frame: the smallest render, launches and gaps.
        dict(name="render_preview", kind="render", scene="cornell", width=64, height=48, spp=1, depth=5, nee=True,
             mis=True, moments=False),
        # The Cornell box configuration of the benchmark.
        dict(name="render_cornell", kind="render", scene="cornell", width=256, height=256, spp=16, depth=8, nee=True,
             mis=True, moments=False),
        # The material scene of the benchmark: 2M triangles, 256 spheres, full HD, the longest call.
        dict(name="render_ggx", kind="render", scene="ggx1000", width=1920, height=1080, spp=64, depth=16, nee=True,
             mis=True, moments=False),
        # The volumetric integrator: the Cornell box in fog.
        dict(name="render_fog", kind="render", scene="fog", width=256, height=256, spp=16, depth=8, nee=True,
             mis=True, moments=False),
        # Frames of the radiance cache with online training (forward, backward, optimiser).
        dict(name="cache_frames", kind="cache", scene="ggx1000", width=1920, height=1080, spp=1, depth=16, frames=4,
             train=True),
        # The batched request loop: a render service's queue of mixed requests.
        dict(name="batch_requests", kind="batch", requests=16, max_size=512, max_spp=32),
        # Tone-mapped 8-bit export of a full-HD film.
        dict(name="film_export", kind="film", width=1920, height=1080, tonemap=True, gamma=2.2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "host_rays", "render", "render", "render", "cache", "batch", "film"])
    if kind in ("rays", "host_rays"):
        scene = rng.choice(["world", "ico6", "ico8", "ggx100", "ggx1000"])
        rays = "test" if scene == "world" else "uniform" if scene.startswith("ico") else rng.choice(["camera", "shadow"])
        return dict(kind=kind, scene=scene, rays=rays, n=_log(rng, 1, 1 << 22 if kind == "rays" else 1 << 21),
                    any_hit=rays == "shadow" or rng.random() < 0.25, tuned=rng.random() < 0.5)
    if kind == "render":
        scene = rng.choice(["cornell", "fog", "ggx100", "ggx1000"])
        width = _log(rng, 16, 1280)
        height = max(9, int(width * rng.uniform(0.5, 1.0)))
        spp = min(_log(rng, 1, 64), max(1, (1 << 24) // (width * height)))
        return dict(kind="render", scene=scene, width=width, height=height, spp=spp, depth=rng.randint(2, 16),
                    nee=rng.random() < 0.9, mis=rng.random() < 0.8, moments=rng.random() < 0.25)
    if kind == "cache":
        width = _log(rng, 160, 1920)
        return dict(kind="cache", scene=rng.choice(["ggx100", "ggx1000"]), width=width, height=max(9, width * 9 // 16),
                    spp=rng.randint(1, 2), depth=rng.randint(4, 16), frames=rng.randint(1, 3), train=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind="batch", requests=rng.randint(2, 16), max_size=rng.choice([128, 256, 512]),
                    max_spp=rng.randint(1, 32))
    return dict(kind="film", width=_log(rng, 16, 3840), height=_log(rng, 16, 2160), tonemap=rng.random() < 0.5,
                gamma=rng.choice([1.0, 2.2, 2.4]))


# ------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _scene(name):
    if name == "world":
        return scenes.random_world(40, 200, with_plane=True, seed=7)
    if name == "cornell":
        return scenes.cornell_box()
    if name == "fog":
        return scenes.foggy_cornell_box()
    if name.startswith("ico"):
        return scenes.ray_query_scene(level=int(name[3:]))
    return scenes.ggx_scene(mesh_n=int(name[3:]))


@functools.lru_cache(maxsize=None)
def _context(name, use):
    """A context with the scene resident, one for each use of it."""
    ctx = Context(0)
    ctx.upload(_scene(name))
    return ctx


@functools.lru_cache(maxsize=None)
def _tuned(name, rays, any_hit):
    """A context whose ray-query variant was tuned once on a sample of the program's rays."""
    ctx = Context(0)
    ctx.upload(_scene(name))
    sample = _rays(name, rays, 1 << 21, 12345)
    ctx.autotune_trace(sample.data_ptr(), sample.shape[0], any_hit)
    return ctx


def _camera(name, width, height):
    if name == "cornell" or name == "fog":
        return (scenes.cornell_box if name == "cornell" else scenes.foggy_cornell_box)(width, height).camera
    return scenes.look_at_camera(width, height, (0.0, 3.0, 14.0), (0.0, 0.8, 0.0), (0.0, 1.0, 0.0), 40.0,
                                 lens_radius=0.05, focal_distance=14.173)


def _rays(name, rays, n, seed):
    """[n, 8] float32 on the GPU: origin, tmax, unit direction, padding (rbr_ray)."""
    if rays == "test":
        r = scenes.random_test_rays(2 * n + 8, seed)[:n]
        return torch.from_numpy(r.view(np.float32).reshape(-1, 8).copy()).cuda()
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(n, 6, device="cuda", generator=g)
    out = torch.zeros(n, 8, device="cuda")
    out[:, 3] = math.inf
    if rays == "uniform":  # origins uniform in the scene box, directions uniform on the sphere
        lo, hi = scenes.scene_bounds(_scene(name))
        lo, hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
        out[:, 0:3] = lo + u[:, 0:3] * (hi - lo)
        z = 1.0 - 2.0 * u[:, 3]
        r = (1.0 - z * z).clamp_min(0.0).sqrt()
        phi = 2.0 * math.pi * u[:, 4]
        d = torch.stack([r * phi.cos(), r * phi.sin(), z], 1)
    elif rays == "camera":  # one jittered ray per pixel of a 16:9 image, in scanline order
        w = max(1, int(round(math.sqrt(n * 16.0 / 9.0))))
        h = (n + w - 1) // w
        cam = _camera(name, w, h)
        k = torch.arange(n, device="cuda")
        x = ((k % w) + u[:, 0] - cam.cx) / cam.fx
        y = (cam.cy - (k // w) - u[:, 1]) / cam.fy
        f, rt, up = (torch.tensor(list(v), device="cuda") for v in (cam.forward, cam.right, cam.up))
        out[:, 0:3] = torch.tensor(list(cam.position), device="cuda")
        d = f + x[:, None] * rt + y[:, None] * up
    else:  # shadow: points near the ground and the mound towards points on the first area light
        o = torch.stack([u[:, 0] * 18 - 9, u[:, 1] * u[:, 1] * 3 + 0.01, u[:, 2] * 18 - 9], 1)
        t = torch.stack([u[:, 3] * 2 - 4, torch.full_like(u[:, 3], 6.99), u[:, 4] * 2 + 1], 1)
        out[:, 0:3] = o
        d = t - o
        out[:, 3] = d.norm(dim=1) - 1e-4
    out[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return out


def _requests(case, seed):
    """The batch's requests: (scene or "fog", camera, spp, depth, flags), sizes from the case alone."""
    rng = np.random.default_rng(5)
    reqs = []
    for i in range(case["requests"]):
        size = int(rng.choice([s for s in (64, 128, 256, 512) if s <= case["max_size"]]))
        spp = int(rng.integers(1, case["max_spp"] + 1))
        if i % 8 == 7:
            reqs.append((3, _camera("fog", size, size), spp, 8, abi.RBR_RENDER_VOLUMETRIC))
        else:
            reqs.append((int(rng.integers(0, 3)), _camera("ggx100", size, size), spp, 16, 0))
    return reqs


@functools.lru_cache(maxsize=None)
def _batch():
    """A batch with three material variants of one geometry and the foggy box."""
    ctx = Context(0)
    base = _scene("ggx100")
    b = Batch(ctx)
    ids = [b.add_scene(base)]
    ids += [b.add_scene_variant(ids[0], scenes.ggx_variant(base, v)) for v in (1, 2)]
    return b, ids + [b.add_scene(_scene("fog"))]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("rays", "host_rays"):
        ctx = (_tuned(case["scene"], case["rays"], case["any_hit"]) if case["tuned"] else _context(case["scene"], "rays"))
        rays = _rays(case["scene"], case["rays"], case["n"], seed)
        n = rays.shape[0]
        if kind == "rays":
            out = torch.zeros(n if case["any_hit"] else n * 2, dtype=torch.uint8 if case["any_hit"] else torch.int32,
                              device="cuda")
            return dict(kind=kind, ctx=ctx, rays=rays, n=n, any_hit=case["any_hit"], out=out)
        host = rays.cpu().pin_memory()
        out = torch.zeros(n * (1 if case["any_hit"] else 8), dtype=torch.uint8).pin_memory()
        return dict(kind=kind, ctx=ctx, keep=host, rays=host.numpy().reshape(-1).view(abi.RAY_DTYPE), any_hit=case["any_hit"],
                    out=out.numpy() if case["any_hit"] else out.numpy().view(abi.HIT_DTYPE), keep_out=out)
    if kind == "film":
        g = torch.Generator(device="cuda").manual_seed(seed)
        npix = case["width"] * case["height"]
        film = torch.rand(npix * 3, device="cuda", generator=g).neg().add_(1.0).log_().neg_()  # radiance, mean 1
        return dict(kind=kind, ctx=_context("cornell", "film"), film=film, case=dict(case),
                    out=torch.zeros(npix * 3, dtype=torch.uint8, device="cuda"))
    if kind == "batch":
        b, ids = _batch()
        reqs = _requests(case, seed)
        return dict(kind=kind, batch=b, ids=ids, reqs=reqs, seed=seed % 1000003,
                    films=[torch.zeros(c.height, c.width, 3, device="cuda") for _, c, _, _, _ in reqs])
    npix = case["width"] * case["height"]
    film = torch.zeros(npix * 3, device="cuda")
    cam = _camera(case["scene"], case["width"], case["height"])
    flags = abi.RBR_RENDER_VOLUMETRIC if case["scene"] == "fog" else 0
    if kind == "cache":
        ctx = _context(case["scene"], "cache")
        ctx.cache_create(seed=seed % 1000, learning_rate=1e-3)
        return dict(kind=kind, ctx=ctx, cam=cam, film=film, frames=case["frames"], train=case["train"],
                    params=render_params(spp=case["spp"], max_depth=case["depth"], seed=seed))
    moments = film.clone() if case["moments"] else None
    return dict(kind=kind, ctx=_context(case["scene"], "render"), cam=cam, film=film, moments=moments,
                params=render_params(spp=case["spp"], max_depth=case["depth"], use_nee=case["nee"], use_mis=case["mis"],
                                     seed=seed, flags=flags | (abi.RBR_RENDER_SECOND_MOMENT if case["moments"] else 0)))


def run(s):
    kind = s["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "rays":
        if s["any_hit"]:
            s["ctx"].trace_any_dev(s["rays"].data_ptr(), s["n"], s["out"].data_ptr(), stream)
            return s["out"]
        s["ctx"].trace_closest_dev(s["rays"].data_ptr(), s["n"], s["out"].data_ptr(), stream)
        hits = s["out"].view(-1, 2)
        return {"prim": hits[:, 0], "t": hits[:, 1].view(torch.float32)}
    if kind == "host_rays":
        s["ctx"].trace_host(s["rays"], any_hit=s["any_hit"], out=s["out"])
        return s["out"] if s["any_hit"] else {"prim": s["out"]["prim"].view(np.int32), "t": s["out"]["t"]}
    if kind == "film":
        c = s["case"]
        st = s["ctx"].lib.rbr_film_to_rgb8(s["ctx"].h, C.c_void_p(s["film"].data_ptr()), c["width"], c["height"], 1.0,
                                           c["gamma"], int(c["tonemap"]), C.c_void_p(s["out"].data_ptr()),
                                           C.c_void_p(stream))
        if st != abi.RBR_OK:
            raise RuntimeError(s["ctx"].last_error())
        return s["out"]
    if kind == "batch":
        for i, ((sid, cam, spp, depth, flags), film) in enumerate(zip(s["reqs"], s["films"])):
            s["batch"].submit(s["ids"][sid], cam, render_params(spp=spp, max_depth=depth, seed=s["seed"] + i, flags=flags),
                              film.data_ptr())
        s["batch"].run(stream)
        return s["films"]
    if kind == "cache":
        s["ctx"].cache_render_dev(s["cam"], s["params"], s["frames"], s["film"].data_ptr(), 0, s["train"], stream)
        if not s["train"]:
            return s["film"]
        w = s["ctx"].cache_get_params()  # the network after the frames' optimiser steps
        return {"film": s["film"], "weights": (w.astype(np.uint32) << 16).view(np.float32)}
    m2 = s["moments"]
    s["ctx"].render_dev(s["cam"], s["params"], s["film"].data_ptr(), 0 if m2 is None else m2.data_ptr(), stream)
    return s["film"] if m2 is None else {"film": s["film"], "moments": m2}


# ------------------------------------------------------------------------------------------
def _ray_flops(prims):
    """Least arithmetic of one ray against a hierarchy of 8 children a node: per level eight boxes of
    six planes (multiply and add), then one triangle test."""
    return max(1, math.ceil(math.log(max(2, prims), 8))) * 8 * 6 * 2 + 50


def work(case):
    kind = case["kind"]
    if kind == "film":
        npix = case["width"] * case["height"]
        return {"bytes": npix * 15, "flops": npix * 12}
    if kind == "batch":
        paths = sum(c.width * c.height * spp for _, c, spp, _, _ in _requests(case, 0))
        pixels = sum(c.width * c.height for _, c, _, _, _ in _requests(case, 0))
        return {"bytes": pixels * 12 + 36 * PRIMITIVES["ggx100"], "flops": paths * 2 * _ray_flops(PRIMITIVES["ggx100"])}
    prims = PRIMITIVES[case["scene"]]
    if kind in ("rays", "host_rays"):
        return {"bytes": case["n"] * (33 if case["any_hit"] else 40) + min(prims, case["n"]) * 36,
                "flops": case["n"] * _ray_flops(prims)}
    npix = case["width"] * case["height"]
    frames = case.get("frames", 1)
    paths = npix * case["spp"] * frames
    flops = paths * 2 * _ray_flops(prims)  # at least a camera ray and one light sample per path
    if kind == "cache":
        flops += paths * 2 * (4 * 64 * 64 + 64 * 16)  # one network query per path
        if case["train"]:
            flops += frames * 4 * 16384 * 6 * (4 * 64 * 64 + 64 * 16)
    return {"bytes": npix * (24 if case.get("moments") else 12) + min(prims, paths) * 36, "flops": flops}


def exact(case, seed):
    """Hit distances of small query batches by brute force in 64 bits (render and cache results have no
    closed value)."""
    if case["kind"] != "rays" or case["scene"] != "world" or case["any_hit"] or case["n"] > 20000:
        return None
    s = _scene("world")
    r = _rays("world", "test", case["n"], seed).cpu().numpy().astype(np.float64)
    o, tmax, d = r[:, 0:3], r[:, 3], r[:, 4:7]
    eps = 1e-4
    best = np.full(len(r), np.inf)

    def keep(t, ok):
        nonlocal best
        t = np.where(ok & (t >= eps) & (t <= tmax), t, np.inf)
        best = np.minimum(best, t)

    with np.errstate(all="ignore"):
        for tri in s.triangles.astype(np.float64):
            v0, e1, e2 = tri[0:3], tri[3:6] - tri[0:3], tri[6:9] - tri[0:3]
            h = np.cross(d, e2)
            a = h @ e1
            sv = o - v0
            q = np.cross(sv, e1)
            u, v = (sv * h).sum(1) / a, (d * q).sum(1) / a
            keep((q @ e2) / a, (np.abs(a) >= eps) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1))
        for c in s.spheres.astype(np.float64):
            oc = o - c[0:3]
            a, hb, cc = (d * d).sum(1), (oc * d).sum(1), (oc * oc).sum(1) - c[3] * c[3]
            disc = hb * hb - a * cc
            sq = np.sqrt(disc)
            near, far = (-hb - sq) / a, (-hb + sq) / a
            keep(np.where((near < eps) | (near > tmax), far, near), disc >= 0)
        for pl in s.planes.astype(np.float64):
            den = d @ pl[0:3]
            keep(-(o @ pl[0:3] + pl[3]) / den, np.abs(den) >= eps)
    return {"prim": None, "t": np.where(np.isfinite(best), best, 0.0)}
