"""Workloads of the render path, timed through the package's public entry points.

A case is a dict of plain values.  Its "kind" names the call:

  frame  one eos_render call (plain or wavefront), the per-frame call of an interactive
         program; "host" copies the image to host memory as DeviceRenderer's callers do
  batch  one eos_render_batch call over several views and scenes
  train  one eos_render_batch with path records and one eos_render_backward: a step of
         inverse shading (image, then gradients of materials and lights)
  build  a scene built from device arrays and one frame of it: a step of an animation
  query  eos_trace_closest and eos_trace_any on rays in device memory: picking, visibility

and "scene" / "size" the seeded generator (eos_b200/scenes.py) and its size.  Scenes,
cameras, rays and image gradients all come from the seed.
"""
from __future__ import annotations

import copy
import ctypes
import math
import os

import numpy as np
import torch

from eos_b200 import _lib, api, autotune, scenes

TABLE = os.path.join(os.path.dirname(os.path.abspath(api.__file__)), "tuning_b200.json")

# triangles of one unit of "size", per generator
SPHERE_TRIS = 20482
SPREAD_SPHERE, SPREAD_FIELD = 5120, 2 * 128 * 128
CLUSTER, FOLIAGE_FIELD = 5000, 2 * 512 * 512


def _case(name, kind, scene, size, width, height, views=1, depth=1, spp=1, grid=False, mode="plain", host=False,
          rays=0):
    c = {"kind": kind, "scene": scene, "size": size, "width": width, "height": height, "views": views,
         "depth": depth, "spp": spp, "grid": grid, "mode": mode, "host": host, "rays": rays}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a thumbnail or a picking preview: the smallest call, latency and launches count
        _case("thumbnail", "frame", "sphere", 0, 64, 64),
        # the drop-in facade's frame with the 2 x 2 anti-aliasing grid, RGBA8 into host memory
        _case("facade_aa", "frame", "sphere", 0, 512, 512, spp=4, grid=True, mode="wavefront", host=True),
        # an interactive 1080p frame of an ordinary scene, one megakernel launch
        _case("frame_1080p", "frame", "mixed", 200_000, 1920, 1080, depth=2),
        # glass and mirrors: ray trees, an odd image size
        _case("glass", "frame", "glass", 24, 961, 541, depth=4),
        # the benchmark's batch: 1.06M triangles, four 1080p views, four lights
        _case("views_1m", "batch", "spread", 200, 1920, 1080, views=4, depth=2),
        # many jobs of many sizes on several scenes, as a render service gets them
        _case("mixed_jobs", "batch", "jobs", 6, 0, 0, views=30, depth=2),
        # the stress view: 4.5M triangles of thin foliage, 4K, two samples, eight lights
        _case("stress_4k", "batch", "foliage", 800, 3840, 2160, depth=3, spp=2),
        # the same world as placements of one stored cluster
        _case("instanced", "batch", "instanced", 800, 1920, 1080, depth=2),
        # a step of inverse shading: eight views and their gradients
        _case("train_views", "train", "materials", 0, 256, 256, views=8),
        # animation: a small scene rebuilt for each frame
        _case("rebuild_small", "build", "mixed", 20_000, 320, 200),
        # animation: the million-triangle scene rebuilt
        _case("rebuild_1m", "build", "spread", 200, 960, 540),
        # incoherent rays against an ordinary scene, an odd count
        _case("queries", "query", "mixed", 60_000, 0, 0, rays=300_007),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "batch", "train", "build", "query"])
    if kind == "frame":
        scene = rng.choice(["sphere", "mixed", "mixed", "glass", "instanced"])
        size = {"sphere": 0, "mixed": _log(rng, 10_000, 500_000), "glass": rng.randint(4, 32),
                "instanced": _log(rng, 10, 800)}[scene]
        grid = scene != "instanced" and rng.random() < 0.3
        w, h = _log(rng, 48, 1920), _log(rng, 48, 1080)
        return _case(None, kind, scene, size, w, h, depth=rng.randint(0, 3), spp=4 if grid else 1, grid=grid,
                     mode=rng.choice(["plain", "wavefront"]), host=rng.random() < 0.3)
    if kind == "batch":
        scene = rng.choice(["spread", "jobs", "foliage", "instanced"])
        if scene == "jobs":
            return _case(None, kind, scene, rng.randint(2, 6), 0, 0, views=rng.randint(3, 30), depth=rng.randint(1, 3))
        size = {"spread": _log(rng, 4, 200), "foliage": _log(rng, 20, 400), "instanced": _log(rng, 20, 800)}[scene]
        return _case(None, kind, scene, size, _log(rng, 97, 1920), _log(rng, 97, 1080), views=rng.randint(1, 3),
                     depth=rng.randint(0, 3), spp=1 if scene == "instanced" else rng.choice([1, 2]))
    if kind == "train":
        return _case(None, kind, "materials", 0, _log(rng, 33, 384), _log(rng, 33, 384), views=rng.randint(1, 10),
                     depth=rng.randint(0, 2), spp=rng.choice([1, 1, 2]))
    if kind == "build":
        scene = rng.choice(["mixed", "spread", "glass"])
        size = {"mixed": _log(rng, 10_000, 500_000), "spread": _log(rng, 8, 200), "glass": rng.randint(4, 32)}[scene]
        return _case(None, kind, scene, size, _log(rng, 120, 960), _log(rng, 90, 540))
    scene = rng.choice(["mixed", "sphere"])
    return _case(None, kind, scene, _log(rng, 10_000, 300_000) if scene == "mixed" else 0, 0, 0,
                 rays=_log(rng, 100, 1_000_000))


# ----------------------------------------------------------------------------- inputs
def _scene(case, seed):
    kind, size = case["scene"], case["size"]
    if kind == "sphere":
        return scenes.config1_scene()
    if kind == "mixed":
        return scenes.mixed_scene(scenes.rng_for(seed), size)
    if kind == "spread":
        return scenes.config2_scene(seed, n_spheres=size)
    if kind == "foliage":
        return scenes.config5_scene(seed, instances=size)
    if kind == "instanced":
        return scenes.config5_instanced(seed, instances=size)
    if kind == "materials":
        return scenes.config4_scene(seed)
    return scenes.small_random_scene(seed, n_spheres=size, level=3, lights=2, transparent=size // 4, both=size // 3)


#: distance and height of the camera's orbit, and the point it looks at, per generator
ORBIT = {"sphere": (4.0, 1.5, 0.0), "mixed": (60.0, 25.0, 0.0), "spread": (160.0, 60.0, 0.0),
         "foliage": (260.0, 90.0, 10.0), "instanced": (260.0, 90.0, 10.0), "materials": (30.0, 18.0, -2.0),
         "glass": (7.0, 3.0, -0.5)}


def _cameras(case, seed, views):
    rng = scenes.rng_for(seed + 17)
    dist, high, aim = ORBIT[case["scene"]]
    a0 = rng.uniform(0.05, 0.8)
    return [scenes.look_at((dist * math.sin(a0 + 2 * math.pi * v / max(8, views)), high,
                            dist * math.cos(a0 + 2 * math.pi * v / max(8, views))), (0, aim, 0), 60.0,
                           case["width"], case["height"]) for v in range(views)]


def _service_jobs(case, seed):
    """(scene index, camera) of a render service's batch: one view in two shows the sphere,
    the others the mixed scenes, at the benchmark's resolutions and odd ones."""
    rng = scenes.rng_for(seed + 29)
    n = case["size"]
    data = [scenes.config1_scene()]
    for _ in range(n - 1):
        data.append(scenes.mixed_scene(rng, int(math.exp(rng.uniform(math.log(10_000), math.log(500_000))))))
    sizes = [(256, 256), (512, 512), (1280, 720), (1920, 1080), (333, 251), (1023, 577)]
    jobs = []
    for v in range(case["views"]):
        k = 0 if v % 2 == 0 else 1 + (v // 2) % (n - 1)
        w, h = sizes[(v * 5 + v // 2) % len(sizes)]
        a = rng.uniform(0, 2 * math.pi)
        dist, high, aim = ORBIT["sphere" if k == 0 else "mixed"]
        jobs.append((k, scenes.look_at((dist * math.sin(a), high, dist * math.cos(a)), (0, aim, 0), 60.0, w, h)))
    return data, jobs


def _rays(case, sc, seed):
    """Origins in the scene's bounds, every second ray aimed at a triangle's centre."""
    rng = scenes.rng_for(seed + 43)
    n = case["rays"]
    lo, hi = sc.verts.min(0), sc.verts.max(0)
    pad = 0.1 * (hi - lo)
    o = rng.uniform(lo - pad, hi + pad, size=(n, 3))
    d = rng.normal(size=(n, 3))
    aimed = rng.integers(sc.n_tris, size=(n + 1) // 2)
    d[::2] = sc.verts[sc.tris[aimed]].mean(1) - o[::2]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _resident(sc):
    """The scene with its arrays in device memory (an animation's vertices live there)."""
    r = copy.copy(sc)
    for k in ("verts", "normals"):
        setattr(r, k, torch.from_numpy(getattr(sc, k)).cuda())
    for k in ("tris", "tri_obj"):
        setattr(r, k, torch.from_numpy(getattr(sc, k).view(np.int32)).cuda())
    return r


def _context():
    ctx = api.Context(0)
    autotune.apply_table(ctx, autotune.load_table(TABLE))
    return ctx


def _image_gradient(case, seed):
    n = case["width"] * case["height"] * case["views"]
    return scenes.rng_for(seed + 71).normal(size=(n, 3)).astype(np.float32)


def prepare(case, seed):
    ctx = _context()
    s = {"case": case, "ctx": ctx}
    if case["scene"] == "jobs":
        data, jobs = _service_jobs(case, seed)
        s["scenes"] = [api.DeviceScene(ctx, d) for d in data]
        s["jobs"] = [api.BatchJob(s["scenes"][k], cam, case["depth"], 0.5) for k, cam in jobs]
        s["outs"] = api.make_batch_outputs(s["jobs"], ("rgba8",))
        return s
    sc = _scene(case, seed)
    if case["kind"] == "query":
        s["scene"] = api.DeviceScene(ctx, sc)
        s["rays"] = torch.from_numpy(_rays(case, sc, seed)).cuda()
        n = case["rays"]
        s["ids"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["t"] = torch.empty(n, dtype=torch.float32, device="cuda")
        s["occluded"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        return s
    s["cams"] = _cameras(case, seed, case["views"])
    if case["kind"] == "build":
        s["data"] = _resident(sc)
    elif case["scene"] == "instanced":
        meshes = [api.DeviceScene(ctx, m) for m in sc.meshes]
        s["scene"] = api.InstancedScene(ctx, meshes, sc.instances, sc.materials, sc.lights)
    else:
        s["scene"] = api.DeviceScene(ctx, sc)
    npx = case["width"] * case["height"]
    if case["kind"] in ("frame", "build"):
        if case["host"]:
            s["out"] = {"rgba8": torch.empty((case["height"], case["width"], 4), dtype=torch.uint8,
                                             pin_memory=True).numpy()}
        else:
            s["out"] = {"rgb": torch.empty((npx, 3), device="cuda"),
                        "rgba8": torch.empty((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")}
            if case["kind"] == "build":
                s["out"]["hit"] = torch.empty(npx * case["spp"], dtype=torch.int32, device="cuda")
        return s
    s["jobs"] = [api.BatchJob(s["scene"], c, case["depth"], 0.5, case["spp"], 7) for c in s["cams"]]
    if case["kind"] == "batch":
        s["outs"] = api.make_batch_outputs(s["jobs"], ("rgb", "rgba8") if case["views"] == 1 else ("rgba8",))
    else:
        # one array of path records over all views, each view's job writing its part
        s["paths"] = torch.empty((case["views"] * npx * case["spp"], 16), dtype=torch.int32, device="cuda")
        s["rgb"] = torch.empty((case["views"], npx, 3), device="cuda")
        s["outs"] = [{"rgb": s["rgb"][v], "paths": s["paths"][v * npx * case["spp"]:(v + 1) * npx * case["spp"]]}
                     for v in range(case["views"])]
        s["grad"] = torch.from_numpy(_image_gradient(case, seed)).cuda()
    return s


# ----------------------------------------------------------------------------- one pass
def _render(s, scene):
    c = s["case"]
    api.render(s["ctx"], scene, s["cams"][0], c["depth"], pixel_offset=0.5, spp=c["spp"], mode=c["mode"],
               outputs=tuple(s["out"]), out=s["out"], device=not c["host"], aa_grid=c["grid"])
    return dict(s["out"])


def run(state):
    s, c = state, state["case"]
    ctx = s["ctx"]
    if c["kind"] == "frame":
        return _render(s, s["scene"])
    if c["kind"] == "build":
        scene = api.DeviceScene(ctx, s["data"])
        out = _render(s, scene)
        scene.close()
        return out
    if c["kind"] == "batch":
        api.render_batch(ctx, s["jobs"], s["outs"])
        return [dict(o) for o in s["outs"]]
    if c["kind"] == "train":
        api.render_batch(ctx, s["jobs"], s["outs"])
        gm, gl = api.render_backward(ctx, s["scene"], s["cams"], c["depth"], s["paths"], s["grad"], pixel_offset=0.5,
                                     spp=c["spp"], jitter_seed=7)
        return {"rgb": s["rgb"], "grad_materials": gm, "grad_lights": gl}
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    h, n = s["scene"].h, c["rays"]
    _lib.check(ctx.lib.eos_trace_closest(ctx.h, h, ptr(s["rays"]), n, ptr(s["ids"]), ptr(s["t"])), "eos_trace_closest")
    _lib.check(ctx.lib.eos_trace_any(ctx.h, h, ptr(s["rays"]), n, ptr(s["occluded"])), "eos_trace_any")
    return {"ids": s["ids"], "t": s["t"], "occluded": s["occluded"]}


# ----------------------------------------------------------------------------- work
def _tris_lights(case):
    size = case["size"]
    return {"sphere": (SPHERE_TRIS, 1), "mixed": (size, 2), "spread": (SPREAD_FIELD + SPREAD_SPHERE * size, 4),
            "foliage": (FOLIAGE_FIELD + CLUSTER * size, 8), "instanced": (FOLIAGE_FIELD + CLUSTER, 8),
            "materials": (64002, 3), "glass": (1280 * size + 2, 2), "jobs": (SPHERE_TRIS + 70_000 * (size - 1), 2)}[
                case["scene"]]


def work(case):
    """Bytes: the scene's triangles (positions, normals, ids: 36 + 36 + 4 B) read once, the
    outputs written once (and records and image gradients read once by the adjoint).
    Operations: half of the primary rays hit and shade (one shadow ray per light each); a
    ray meets one four-box node per level of a four-wide tree (4 x 14 operations) and two
    triangles (2 x 50); a shaded light costs 60.  Secondary rays are left out."""
    tris, lights = _tris_lights(case)
    ray = 56.0 * max(1.0, math.log(max(tris, 4), 4)) + 100.0
    read = 76.0 * tris
    if case["kind"] == "query":
        n = case["rays"]
        return {"bytes": read + n * (24 + 24 + 4 + 4 + 1), "flops": 2 * n * ray}
    if case["scene"] == "jobs":
        px = case["views"] * 600_000
    else:
        px = case["views"] * case["width"] * case["height"]
    paths = px * case["spp"]
    flops = paths * (ray + 0.5 * lights * (ray + 60.0))
    out = 4.0 * px
    if case["kind"] in ("frame", "build") and not case["host"] or case["kind"] == "batch" and case["views"] == 1:
        out += 12.0 * px
    if case["kind"] == "train":
        out = 12.0 * px + 64.0 * paths + 64.0 * paths + 12.0 * px
        flops += paths * 0.5 * lights * 150.0
    if case["kind"] == "build":
        flops += tris * 32 * 12.0  # neighbour search of one clustering round
        read += 128.0 * tris / 4 + 96.0 * tris
    return {"bytes": read + out, "flops": flops}


# ----------------------------------------------------------------------------- 64-bit results
class _Exact:
    """The renderer in 64 bits without an acceleration structure: every ray against every
    triangle as matrix products.  With T = o - v1, m = o x d and n = e1 x e2 the
    Moller-Trumbore numerators are linear in the ray:
      det = -d.n   u det = e2.m - d.(e2 x v1)   v det = -e1.m - d.(v1 x e1)   t det = o.n - v1.n
    """

    def __init__(self, sc, dev):
        f = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        tri = sc.tris.astype(np.int64)
        p, n = f(sc.verts[tri]), f(sc.normals[tri])
        self.obj = torch.as_tensor(sc.tri_obj.astype(np.int64), device=dev)
        v1 = p[:, 0]
        e1 = f((sc.verts[tri[:, 1]] - sc.verts[tri[:, 0]]))
        e2 = f((sc.verts[tri[:, 2]] - sc.verts[tri[:, 0]]))
        nn = torch.linalg.cross(e1, e2)
        self.det = -nn.T
        self.u = torch.cat([e2, -torch.linalg.cross(e2, v1)], 1).T.contiguous()
        self.v = torch.cat([-e1, -torch.linalg.cross(v1, e1)], 1).T.contiguous()
        self.t = torch.cat([nn, -(v1 * nn).sum(1, keepdim=True)], 1).T.contiguous()
        self.normals = n
        self.mats, self.lights = f(sc.materials), f(sc.lights)
        self.ambient = float(sc.ambient_index)
        self.dev = dev
        self.chunk = max(64, int(6e7 // max(1, len(v1))))

    def _chunks(self, o, d):
        one = torch.ones(1, dtype=torch.float64, device=self.dev)
        for a in range(0, len(o), self.chunk):
            oo, dd = o[a:a + self.chunk], d[a:a + self.chunk]
            md = torch.cat([torch.linalg.cross(oo, dd), dd], 1)
            det = dd @ self.det
            inv = torch.where(det.abs() < 1e-5, math.nan, 1.0 / det)
            u, v = (md @ self.u).mul_(inv), (md @ self.v).mul_(inv)
            t = (torch.cat([oo, one.expand(len(oo), 1)], 1) @ self.t).mul_(inv)
            yield a, u, v, t, (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)

    def closest(self, o, d):
        n = len(o)
        tri = torch.full((n,), -1, dtype=torch.int64, device=self.dev)
        t, u, v = (torch.full((n,), math.inf, dtype=torch.float64, device=self.dev) for _ in range(3))
        for a, cu, cv, ct, ok in self._chunks(o, d):
            best, k = torch.where(ok, ct, math.inf).min(1)
            at = slice(a, a + len(k))
            hit = torch.isfinite(best)
            tri[at] = torch.where(hit, k, -1)
            t[at] = best
            u[at], v[at] = cu.gather(1, k[:, None])[:, 0], cv.gather(1, k[:, None])[:, 0]
        return tri, t, u, v

    def blocked(self, o, d):
        return torch.cat([ok.any(1) for _, _, _, _, ok in self._chunks(o, d)]) if len(o) else \
            torch.zeros(0, dtype=torch.bool, device=self.dev)

    def colour(self, o, d, eye, depth, mats, lights):
        """Colours of rays (o, d); mats / lights may require gradients (visibility frozen)."""
        unit = lambda x: x / x.norm(dim=1, keepdim=True)  # noqa: E731
        out = torch.zeros((len(o), 3), dtype=torch.float64, device=self.dev)
        tri, t, u, v = self.closest(o, d)
        idx = torch.nonzero(tri >= 0)[:, 0]
        if not len(idx):
            return out
        tri, t, u, v, o, d = tri[idx], t[idx, None], u[idx, None], v[idx, None], o[idx], d[idx]
        P = o + t * d
        n = self.normals[tri]
        N = unit(n[:, 0] * (1 - u - v) + n[:, 1] * u + n[:, 2] * v)
        m = mats[self.obj[tri]]
        raw = self.mats[self.obj[tri]]
        V = unit(eye - P)
        c = torch.zeros_like(P)
        for l, frozen in zip(lights, self.lights):
            S = unit(frozen[:3] - P)
            lit = ~self.blocked(P + 1e-3 * S, S)
            L = unit(l[:3] - P)
            ndl = (N * L).sum(1, keepdim=True)
            vr = (V * unit(2 * ndl * N - L)).sum(1, keepdim=True)
            spec = torch.where(vr > 0, vr.clamp(min=1e-300) ** m[:, 6:7], 0.0)
            c = c + lit[:, None] * (ndl.clamp(min=0) * m[:, :3] * l[3:] + spec * l[3:] * m[:, 3:6])
        if depth > 0:
            mirror = raw[:, 7] > 0
            k = torch.nonzero(mirror)[:, 0]
            if len(k):
                R = unit(d[k] - 2 * N[k] * (N[k] * d[k]).sum(1, keepdim=True))
                c = c.index_add(0, k, raw[k, 7:8] * self.colour(P[k] + 1e-3 * R, R, eye, depth - 1, mats, lights))
            k = torch.nonzero(raw[:, 8] > 0)[:, 0]
            if len(k):  # both Fresnel terms take the one traced ray: K c + (1 - K) c = c
                I = unit(d[k])
                side = torch.where((I * N[k]).sum(1, keepdim=True) < 0, 1.0, -1.0) * N[k]
                R = unit(d[k] - 2 * side * (side * d[k]).sum(1, keepdim=True))
                c = c.index_add(0, k, self.colour(P[k] + 1e-3 * side, R, eye, depth - 1, mats, lights))
        return out.index_add(0, idx, c)

    def image(self, cam, depth, spp, mats, lights):
        """RGB [H * W, 3]: pixel centres, or the reference's n x n grid for spp = n * n."""
        g = int(round(math.sqrt(spp)))
        f = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=self.dev)  # noqa: E731
        right, up, view, eye = f(cam.right), f(cam.up), f(cam.view), f(cam.position)
        y, x = torch.meshgrid(torch.arange(cam.height, device=self.dev, dtype=torch.float64),
                              torch.arange(cam.width, device=self.dev, dtype=torch.float64), indexing="ij")
        total = 0.0
        for q in range(spp):
            ox, oy = (0.5, 0.5) if spp == 1 else (q % g / g, q // g / g)
            a = ((x + ox) / (cam.width / 2) - 1).reshape(-1, 1)
            b = ((y + oy) / (cam.height / 2) - 1).reshape(-1, 1)
            d = a * right + b * up + view
            d = d / d.norm(dim=1, keepdim=True)
            total = total + self.colour(eye.expand(len(d), 3), d, eye, depth, mats, lights)
        return total / spp


def _exact_tests(case):
    """Ray-triangle tests of a brute-force pass, at its most."""
    tris, lights = _tris_lights(case)
    rays = case["views"] * case["width"] * case["height"] * case["spp"]
    grow = {"glass": 1.5, "materials": 0.0}.get(case["scene"], 0.5)
    return rays * tris * (1 + lights) * sum(grow ** k for k in range(case["depth"] + 1))


def exact(case, seed):
    jittered = case["spp"] > 1 and not case["grid"]
    if case["kind"] == "query":
        return None  # a ray through an edge hits or misses by its last bit, and a miss is infinite
    if (case["scene"] in ("jobs", "instanced") or case["host"] or jittered or not torch.cuda.is_available()
            or case["kind"] == "batch" and case["views"] > 1 or _exact_tests(case) > 7e11):
        return None
    sc = _scene(case, seed)
    with torch.no_grad():
        e = _Exact(sc, "cuda")
        cams = _cameras(case, seed, case["views"])
        if case["kind"] != "train":
            out = {"rgb": e.image(cams[0], case["depth"], case["spp"], e.mats, e.lights), "rgba8": None}
            if case["kind"] == "build":
                out["hit"] = None
            return [out] if case["kind"] == "batch" else out
    # gradients: material columns kd, ks, log shininess and all light columns
    log_mats = torch.cat([e.mats[:, :6], e.mats[:, 6:7].log()], 1).requires_grad_()
    lights = e.lights.clone().requires_grad_()
    grad = torch.from_numpy(_image_gradient(case, seed)).cuda().double().reshape(case["views"], -1, 3)
    rgb, gm, gl = [], 0.0, 0.0
    for cam, g in zip(cams, grad):
        mats = torch.cat([log_mats[:, :6], log_mats[:, 6:7].exp()], 1)
        img = e.image(cam, case["depth"], 1, mats, lights)
        dm, dl = torch.autograd.grad((img * g).sum(), (log_mats, lights))
        rgb.append(img.detach())
        gm, gl = gm + dm, gl + dl
    gl = torch.cat([gl[:, 3:], gl[:, :3]], 1)  # colour, then position, as eos_grads has them
    return {"rgb": torch.stack(rgb), "grad_materials": gm, "grad_lights": gl}
