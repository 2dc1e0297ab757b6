"""Measured cases of the renderer: the work that its users have it do, through its public entry
points, from one picking call to the full benchmark frame.

A case is a dict of plain values; `kind` selects the entry points:

  closest / any   ray queries on device buffers (trace_closest, trace_any)
  frame           one image of one scene: clear, render, read the FP64 means
  passes          progressive refinement: two sample ranges, raw film and error estimate
  tracer          the PathTracer host object (Milton's PropertyMap keys), render() and output()
  tonemap         a filtered image (reconstruction filter) through the Reinhard tone map
  batch           requests of different scenes and sizes in shared waves, every image read
  noalloc         a frame over the library's fixed device scratch

Scenes (`scene`, `tris`): `plain` (the 36-triangle box), `random` (spheres and boxes of about
`tris` triangles with 1-4 quad lights), `mid` (1,000,010 triangles), `terrain` (fBm terrain with
glossy and glass spheres, 16 lights, a deep tree), `textured` (image maps, a bump map and a
constant background), `balls` (analytic spheres in the box).  Everything is made from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from milton_gb300 import pathtracer as pt
from milton_gb300 import scenegen
from milton_gb300.scene import SceneBuilder, camera, dielectric, phong


def _case(name, kind, scene, **kw):
    c = dict(kind=kind, scene=scene, tris=0, width=0, height=0, spp=1, depth=8, rr=3, nds=1, rays=0, scenes=0,
             filter="none")
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a pick or an autofocus in an editor: a few rays, one launch, pure latency
        _case("pick_33_rays", "closest", "random", tris=20_000, rays=33),
        # ray queries of a baking or collision tool: half camera rays, half uniform rays, one odd count
        _case("closest_1m", "closest", "random", tris=300_000, rays=1_000_003),
        # visibility segments between random points (ambient occlusion, line of sight)
        _case("visibility_777k", "any", "random", tris=50_000, rays=777_777),
        # thumbnail: image sides off the 8x8 tiles, few paths, launches count
        _case("thumbnail_37x23", "frame", "random", tris=2_000, width=37, height=23, spp=4, depth=5),
        # the plain configuration of the benchmark
        _case("plain_256", "frame", "plain", width=256, height=256, spp=16, depth=5),
        # the headline frame of the benchmark
        _case("mid_frame", "frame", "mid", tris=1_000_010, width=1024, height=1024, spp=64),
        # interactive refinement: two calls of two passes each on a 300k-triangle scene, then the
        # error estimate and the raw film
        _case("refine_2x2spp", "passes", "random", tris=300_000, width=801, height=603, spp=4),
        # big geometry, many lights, long paths: tree beyond the L2, 16 shadow rays per vertex
        _case("terrain_2m", "frame", "terrain", tris=2_052_032, width=640, height=640, spp=8, depth=16),
        # requests of uneven size that share waves (the batched configuration, fewer scenes)
        _case("batch_10_scenes", "batch", "random", tris=30_000, width=512, height=512, spp=16, scenes=10),
        # image maps, bump map, background, 4 light samples, Mitchell filter, 8-bit output
        _case("textured_tonemap", "tonemap", "textured", width=333, height=250, spp=16, depth=5, nds=4,
              filter="mitchell"),
        # Milton's own defaults (no depth cap, roulette from 2) on analytic spheres with a thin lens
        _case("lens_spheres", "tracer", "balls", width=400, height=300, spp=9, depth=0, rr=2),
        # a host that forbids device allocation while it renders
        _case("noalloc_200x152", "noalloc", "random", tris=10_000, width=200, height=152, spp=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "any", "frame", "frame", "passes", "batch", "tonemap", "tracer", "noalloc"])
    tris = _log(rng, 500, 500_000)
    if kind in ("closest", "any"):
        # (a few segments would give the same bytes whatever the scene)
        return _case(None, kind, "random", tris=tris, rays=_log(rng, 1 if kind == "closest" else 1000, 3_000_000))
    w, h = _log(rng, 16, 1024), _log(rng, 16, 1024)
    spp = rng.choice([1, 2, 4, 7, 16, 25, 64])
    depth, rr, nds = rng.choice([1, 3, 5, 8, 16]), rng.choice([2, 3, 5]), rng.choice([1, 1, 1, 2, 4])
    kw = dict(width=w, height=h, spp=spp, depth=depth, rr=rr, nds=nds)
    if kind == "frame":
        scene = rng.choice(["plain", "random", "random", "textured", "terrain", "balls"])
        if scene == "terrain":
            kw.update(spp=min(spp, 4), nds=1)
            tris = _log(rng, 20_000, 500_000)
        return _case(None, kind, scene, tris=tris, **kw)
    if kind == "passes":
        kw["spp"] = 2 * max(1, min(spp, 16) // 2)
        return _case(None, kind, rng.choice(["plain", "random"]), tris=tris, **kw)
    if kind == "batch":
        kw.update(width=min(w, 512), height=min(h, 512), spp=min(spp, 16), depth=max(depth, 3))
        return _case(None, kind, "random", tris=min(tris, 60_000), scenes=rng.choice([2, 3, 5, 9, 16]), **kw)
    if kind == "tonemap":
        return _case(None, kind, rng.choice(["textured", "plain"]),
                     filter=rng.choice(["none", "box", "triangle", "gaussian", "mitchell", "lanczosSinc"]), **kw)
    if kind == "tracer":
        kw.update(spp=min(spp, 16), depth=rng.choice([0, 0, 5, 8]))
        return _case(None, kind, rng.choice(["balls", "plain", "random"]), tris=min(tris, 50_000), **kw)
    kw.update(width=min(w, 400), height=min(h, 400), spp=min(spp, 4))
    return _case(None, "noalloc", rng.choice(["plain", "random"]), tris=min(tris, 50_000), **kw)


# ------------------------------------------------------------------------------------------
# scenes

def _balls(seed):
    """Analytic spheres (glass, dispersive glass, Phong, one emitting) in the plain box."""
    rng = np.random.default_rng(seed)
    s0 = scenegen.plain(seed)
    b = SceneBuilder()
    for name, first, count in s0.shapes:
        if name in ("tallBox", "shortBox"):
            continue
        m = b.material(s0.materials[s0.tri_mat[first]])
        if name == "light":
            b.add_quad_light(name, (0.0, 1.999, 0.0), (0.5, 0.0, 0.0), (0.0, 0.0, -0.5), 15.0, m)
        else:
            b.add(name, s0.tri_v[first:first + count], s0.tri_n[first:first + count], m)
    glass, ph = b.material(dielectric(1.5)), b.material(phong(0.3, 0.4, 40.0))
    prism = b.material(dielectric([1.45, 1.55, 1.7]))
    for k, (x, z) in enumerate(((-0.5, -0.5), (0.5, -0.4), (-0.4, 0.4), (0.45, 0.45))):
        r = float(rng.uniform(0.18, 0.32))
        b.add_sphere((x, r, z), r, (glass, ph, prism, ph)[k])
    b.add_sphere((0.0, 1.3, 0.0), 0.1, b.material(s0.materials[0]), radiance=[12.0, 11.0, 9.0])
    c = s0.camera
    return b.build(camera(eye=c[0:3], look=c[3:6], up=c[6:9], height_angle=float(c[9]), aspect=float(c[10])))


def _scene(name, tris, seed):
    """The scene, and its kd-tree settings."""
    if name == "plain":
        return scenegen.plain(seed), pt.KdSettings()
    if name == "mid":
        return scenegen.mid(seed), pt.KdSettings()
    if name == "textured":
        s = scenegen.textured(seed, filters=("gaussian", 3.0, {"sigma": 0.9}))
        s.background_le = np.array([0.2, 0.25, 0.35], np.float32)
        return s, pt.KdSettings()
    if name == "balls":
        return _balls(seed), pt.KdSettings()
    if name == "terrain":
        # 79 % of the triangles in the terrain, the rest in spheres of 2,160 triangles
        objects = max(4, round(0.21 * tris / 2160))
        cells = max(16, int(math.sqrt(max(512, tris - 2160 * objects) / 2)))
        return scenegen.large(seed, cells=cells, n_objects=objects), pt.KdSettings(max_depth=32)
    return scenegen.random_scene(seed, tris), pt.KdSettings()


def _rays(case, scene, seed):
    """Half camera rays, half uniform rays through the scene box (closest); segments between
    points of the box (any).  Directions are unit, as a tracer's are."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rays"]
    lo = torch.tensor(scene.tri_v.reshape(-1, 3).min(0), device="cuda")
    hi = torch.tensor(scene.tri_v.reshape(-1, 3).max(0), device="cuda")
    rays = torch.zeros((n, 8), device="cuda")
    p = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    rays[:, 0:3] = p
    if case["kind"] == "any":
        q = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
        d = q - p
        rays[:, 7] = d.norm(dim=1) * 0.999
    else:
        d = torch.randn((n, 3), generator=g, device="cuda")
        rays[:, 7] = math.inf
        c = scene.camera
        look, up = torch.tensor(c[3:6], device="cuda"), torch.tensor(c[6:9], device="cuda")
        u = torch.linalg.cross(look, up)
        u = u / u.norm()
        v = torch.linalg.cross(u, look)
        k = n // 2
        xy = (2 * torch.rand((k, 2), generator=g, device="cuda") - 1) * math.tan(math.radians(float(c[9])) / 2)
        d[:k] = look + u * xy[:, 0:1] * float(c[10]) + v * xy[:, 1:2]
        rays[:k, 0:3] = torch.tensor(c[0:3], device="cuda")
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return rays


def _settings(case, seed, **kw):
    args = dict(width=case["width"], height=case["height"], spp=case["spp"], no_direct_samples=case["nds"],
                max_depth=case["depth"], rr_start_depth=case["rr"], seed=seed)
    args.update(kw)
    return pt.RenderSettings(**args)


def _requests(case, seed):
    """The requests of a batch: sides log-spread from an eighth of the case's to the whole (the
    sizes belong to the case; golden-ratio steps, so that neighbours differ), triangle counts
    log-uniform from a thirtieth, scenes from the seed, one sample count."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["scenes"]):
        f = 8.0 ** -((k * 0.6180339887) % 1.0)
        t = float(np.exp(rng.uniform(np.log(1 / 30), 0.0)))
        out.append((max(8, int(case["width"] * f)), max(8, int(case["height"] * f)), max(500, int(case["tris"] * t)),
                    int(rng.integers(1 << 30))))
    return out


# ------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        batch, films = pt.Batch(), []
        for w, h, tris, s in _requests(case, seed):
            scene, kd = _scene(case["scene"], tris, s)
            film = pt.Film(w, h)
            batch.add(pt.DeviceScene(scene, pt.Accel(scene, kd)), _settings(case, s, width=w, height=h), film)
            films.append(film)
        return dict(kind=kind, batch=batch, films=films)
    scene, kd = _scene(case["scene"], case["tris"], seed)
    if kind == "tracer":
        c = scene.camera.copy()
        c[11], c[12], c[13], c[14], c[15] = 0.05, 0.6, -1.0, 0.5, 0.5  # thin lens, autofocus at the centre
        scene.camera = c
        t = pt.PathTracer(dict(noSuperSamples=case["spp"], noDirectSamples=case["nds"], maxDepth=case["depth"],
                               rrStartDepth=case["rr"], seed=seed))
        t.set_scene(scene)
        t.set_output(case["width"], case["height"])
        t.init()
        return dict(kind=kind, tracer=t)
    dscene = pt.DeviceScene(scene, pt.Accel(scene, kd))
    if kind in ("closest", "any"):
        return dict(kind=kind, dscene=dscene, rays=_rays(case, scene, seed))
    film = pt.Film(case["width"], case["height"])
    if case["filter"] != "none":
        film.set_filter(case["filter"], 3.0)
    state = dict(kind=kind, dscene=dscene, film=film, settings=_settings(case, seed))
    if kind == "passes":
        half = case["spp"] // 2
        state["settings"] = [_settings(case, seed, sample_begin=0, sample_count=half),
                             _settings(case, seed, sample_begin=half, sample_count=case["spp"] - half)]
    return state


def run(state):
    kind = state["kind"]
    if kind == "closest":
        hits = pt.trace_closest(state["dscene"], state["rays"])
        return dict(t=hits[:, 0], prim=hits.view(torch.int32)[:, 1], b=hits[:, 2:4])
    if kind == "any":
        return dict(occluded=pt.trace_any(state["dscene"], state["rays"]))
    if kind == "batch":
        for f in state["films"]:
            f.clear()
        state["batch"].render()
        return [f.mean() for f in state["films"]]
    if kind == "tracer":
        state["tracer"].render()
        return dict(image=state["tracer"].output())
    film, settings = state["film"], state["settings"]
    film.clear()
    if kind == "passes":
        for s in settings:
            pt.render(state["dscene"], s, film)
        return dict(error=pt.film_error([film]), raw=film.raw())
    if kind == "noalloc":
        pt.render_noalloc(state["dscene"], settings, film)
        return dict(image=film.mean())
    pt.render(state["dscene"], settings, film)
    if kind == "tonemap":
        return dict(rgba=film.tonemap(), image=film.mean())
    return dict(image=film.mean())


# ------------------------------------------------------------------------------------------

_LIGHTS = {"plain": 1, "mid": 4, "terrain": 16, "textured": 1, "balls": 2, "random": 2.5}
_TRIS = {"plain": 36, "mid": 1_000_010, "textured": 1164, "balls": 12}


def work(case):
    """Bytes: every triangle that the rays can reach once (vertices and normals, 72 B), the rays
    and results once, or the film once.  Operations: per ray one descent of a binary hierarchy
    (24 per level) and one triangle test (60); per path vertex 250 for the surface and BSDF
    sample and 150 for each light sample.  A path is taken to have 1.8 vertices (min(depth, 1.8)),
    the least that the scenes here show."""
    tris = _TRIS.get(case["scene"], case["tris"])
    ray = 24 * max(1.0, math.log2(max(tris, 2))) + 60
    n = case["rays"]
    if case["kind"] in ("closest", "any"):
        out = 16 if case["kind"] == "closest" else 1
        return {"bytes": n * (32 + out) + min(tris, n) * 36, "flops": n * ray}
    if case["kind"] == "batch":
        frac = (1 - 0.125 ** 2) / (2 * math.log(8))   # mean of f^2 for log-uniform f in [1/8, 1]
        paths = case["scenes"] * case["width"] * case["height"] * frac * case["spp"]
        pixels, tris = paths / case["spp"], case["scenes"] * case["tris"] * 0.28
    else:
        pixels = case["width"] * case["height"]
        paths = pixels * case["spp"]
    vertices = 1.8 if case["depth"] == 0 else min(case["depth"], 1.8)
    lights = _LIGHTS[case["scene"]] * max(1, math.isqrt(case["nds"])) ** 2
    flops = paths * vertices * (ray + 250 + lights * (ray + 150))
    return {"bytes": min(tris, paths) * 72 + pixels * 24, "flops": flops}


def exact(case, seed):
    """Closest hits by brute force over all triangles in 64 bits (Moeller-Trumbore), where that
    takes a few seconds.  A rendered image has no such value: Russian roulette, lobe choice and
    the hit of an edge are decided on rounded numbers, so a 64-bit restatement follows other
    paths."""
    if case["kind"] != "closest" or case["rays"] * case["tris"] > 4e9:
        return None
    scene, _ = _scene(case["scene"], case["tris"], seed)
    rays = _rays(case, scene, seed).double()
    v = torch.tensor(scene.tri_v, device="cuda").double()
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = rays.shape[0]
    best_t = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    best_b = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    step = max(1, 8_000_000 // v.shape[0])
    for k in range(0, n, step):
        o, d = rays[k:k + step, None, 0:3], rays[k:k + step, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, v.shape[0], -1), e2[None].expand(d.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        s = o - v0
        inv = 1.0 / det
        b1 = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1[None].expand(s.shape[0], -1, -1))
        b2 = (d * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        ok = (det != 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t > rays[k:k + step, 3:4]) & \
            (t < rays[k:k + step, 7:8])
        t = torch.where(ok, t, math.inf)
        m, at = t.min(1)
        rows = torch.arange(m.shape[0], device="cuda")
        best_t[k:k + step] = m
        hit = torch.isfinite(m)[:, None]
        best_b[k:k + step] = torch.where(hit, torch.stack([b1[rows, at], b2[rows, at]], 1), 0.0)
    return dict(t=best_t, prim=None, b=best_b)
