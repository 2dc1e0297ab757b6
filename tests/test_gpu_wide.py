"""The 8-wide hierarchy that rays traverse against the kd-tree, bit for bit: the counted ray query and
mgpu_tune_set("wide", 0) go through the kd-tree, everything else through the hierarchy."""
import numpy as np
import pytest

from gpu_util import gpu_any, gpu_trace
from milton_gb300 import pathtracer as pt
from milton_gb300 import scenegen
from milton_gb300.scene import SceneBuilder, camera, dielectric, diffuse
from raygen import camera_rays, sphere_rays

pytestmark = pytest.mark.gpu


def _soup(tris, culled=False):
    b = SceneBuilder()
    m = b.material(diffuse(0.5))
    b.add("t", np.asarray(tris, np.float32), np.broadcast_to(np.float32([0, 1, 0]), (len(tris), 3, 3)), m, culled=culled)
    return b.build(camera(eye=(0, 1, 3), look=(0, 0, -1), up=(0, 1, 0), height_angle=40.0, aspect=1.0))


def _random_tris(n, seed, size=0.2, scale=1.0, offset=(0, 0, 0)):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    return (c + rng.normal(size=(n, 3, 3)) * size) * scale + np.asarray(offset)


def _scene(kind):
    if kind.startswith("n"):  # sizes around the leaf, node and builder block limits
        return _soup(_random_tris(int(kind[1:]), 7, size=0.5 if int(kind[1:]) < 100 else 0.05))
    if kind == "culled":
        return _soup(_random_tris(500, 3), culled=True)
    if kind == "coincident":  # every triangle twice, and a stack of copies of one
        t = _random_tris(300, 5)
        return _soup(np.concatenate([t, t[::-1], np.repeat(t[:1], 40, 0)]))
    if kind == "flat":        # one plane, a grid of axis-aligned quads
        g = np.arange(40) / 20.0 - 1.0
        q = [scenegen.quad_tris((x, 0, z + .05), (x + .05, 0, z + .05), (x + .05, 0, z), (x, 0, z)) for x in g for z in g]
        return _soup(np.concatenate(q))
    if kind == "points":      # degenerate triangles among proper ones
        t = _random_tris(200, 6)
        t[::3] = t[::3, :1]
        t[1::6, 2] = t[1::6, 1]
        return _soup(t)
    if kind == "line":        # clusters each nearest to the one before (linearly growing gaps)
        x = np.cumsum(np.arange(5000) * 1e-6)[:, None, None]
        return _soup(np.concatenate([x + np.zeros((1, 3, 1)), np.zeros((5000, 3, 2))], -1) +
                     np.float32([[0, 0, 0], [0, 1e-2, 0], [0, 0, 1e-2]]))
    if kind == "far":         # small geometry far from the origin
        return _soup(_random_tris(2000, 8, size=0.05, scale=1.0, offset=(3000, -2000, 5000)))
    if kind == "scales":      # one huge quad and tiny detail
        return _soup(np.concatenate([scenegen.quad_tris((-1e4, -1, 1e4), (1e4, -1, 1e4), (1e4, -1, -1e4), (-1e4, -1, -1e4)),
                                     _random_tris(3000, 9, size=1e-3)]))
    if kind == "balls":       # analytic spheres beside triangles
        s = scenegen.plain(2)
        s.spheres = np.float32([[0.3, 0.9, 0.5, 0.2, 0, 0, 0, 1], [-0.5, 1.5, 0.0, 0.3, 0, 0, 0, 1]])
        s.sphere_mat = np.int32([0, 0])
        s.sphere_light = np.int32([-1, -1])
        return s
    return scenegen.plain(1) if kind == "plain" else scenegen.random_scene(9, 60_000)


def _rays(s, n, seed):
    v = s.tri_v.reshape(-1, 3)
    lo, hi = v.min(0) - 0.3, v.max(0) + 0.3
    if np.ptp(v, axis=0).max() > 1e3:  # the detail, not the huge quad
        lo, hi = np.full(3, -1.2), np.full(3, 1.2)
    r = np.concatenate([camera_rays(s.camera, n, seed), sphere_rays(lo, hi, n, seed + 1)])
    rng = np.random.default_rng(seed + 2)
    ax = sphere_rays(lo, hi, n, seed + 3)  # axis-parallel, -0 among the zeros, origins on vertex planes
    k = rng.integers(0, 3, n)
    ax[:, 4:7] = np.where(rng.random((n, 3)) < 0.5, -0.0, 0.0)
    ax[np.arange(n), 4 + k] = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    p = v[rng.integers(0, len(v), n)]
    on = rng.random((n, 3)) < 0.3
    ax[:, 0:3] = np.where(on, p, ax[:, 0:3])
    aimed = sphere_rays(lo, hi, n, seed + 4)  # at points of triangles: edges, vertices, interiors
    t = s.tri_v[rng.integers(0, s.ntri, n)].astype(np.float64)
    w = rng.dirichlet((1, 1, 1), n) * np.where(rng.random((n, 1)) < 0.5, 1.0, rng.integers(0, 2, (n, 3)))
    w /= np.maximum(w.sum(1, keepdims=True), 1e-9)
    d = (t * w[..., None]).sum(1) - aimed[:, 0:3]
    aimed[:, 4:7] = d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-9)
    short = sphere_rays(lo, hi, n, seed + 5)
    short[:, 3] = rng.uniform(0, 0.5, n)
    short[:, 7] = short[:, 3] + rng.uniform(0, 1.5, n)
    short[::2, 4:7] *= 3.7  # directions need not be unit
    return np.concatenate([r, ax, aimed, short]).astype(np.float32)


KINDS = ["n1", "n2", "n3", "n4", "n7", "n25", "n2047", "n2048", "n2049", "n4097", "culled", "coincident", "flat", "points",
         "line", "far", "scales", "balls", "plain", "random"]


@pytest.mark.parametrize("kind", KINDS)
def test_ray_queries_equal_the_kd_trees(cuda, kind):
    s = _scene(kind)
    ds = pt.DeviceScene(s, pt.Accel(s))
    for n in (20_000, 33):
        rays = _rays(s, n, 11)
        kd, _ = gpu_trace(cuda, ds, rays, counts=True)
        wide, _ = gpu_trace(cuda, ds, rays)
        same = np.all(kd.view(np.uint32) == wide.view(np.uint32), axis=1)
        assert same.all(), (kind, n, int((~same).sum()), rays[~same][:2], kd[~same][:2], wide[~same][:2])
        assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


@pytest.mark.parametrize("kind", ["plain", "random", "textured", "balls", "deep", "batch"])
def test_films_equal_the_kd_trees(cuda, kind):
    if kind == "textured":
        s = scenegen.textured(3)
    elif kind in ("balls", "deep"):
        s = _scene("balls" if kind == "balls" else "random")
        s.materials[s.tri_mat[0]] = dielectric(1.5)
    else:
        s = _scene("random" if kind == "batch" else kind)
    scenes = [pt.DeviceScene(s, pt.Accel(s))]
    if kind == "batch":
        p = scenegen.plain(5)
        scenes += [pt.DeviceScene(p, pt.Accel(p)), scenes[0]]
    depth = 0 if kind == "deep" else 6
    sizes = [(61, 43), (40, 24), (16, 9)]
    out = []
    assert pt.tune_get("wide") == 1
    try:
        for wide in (0, 1):
            pt.tune("wide", wide)
            films = [pt.Film(*wh) for wh in sizes[:len(scenes)]]
            b = pt.Batch()
            for k, (ds, f, wh) in enumerate(zip(scenes, films, sizes)):
                b.add(ds, pt.RenderSettings(*wh, 9, max_depth=depth, rr_start_depth=3, seed=31 + k), f)
            b.render()
            out.append([f.raw() for f in films])
    finally:
        pt.tune("wide", 1)
    for a, c in zip(*out):
        assert np.array_equal(a.view(np.uint32), c.view(np.uint32))


def test_negative_tmin_and_lines(cuda):
    # the hierarchy's box tests move the planes by an absolute amount, so t < 0 needs no special case:
    # lines (tmin = -inf) and rays that start behind the origin against a brute force in 64 bits
    s = scenegen.plain(1)
    ds = pt.DeviceScene(s, pt.Accel(s))
    r = sphere_rays((-1, 0, -1), (1, 2, 1), 3000, 5)
    r[::2, 3] = -np.inf
    r[1::2, 3] = -0.75
    h, _ = gpu_trace(cuda, ds, r)
    o, d = r[:, None, 0:3].astype(np.float64), r[:, None, 4:7].astype(np.float64)
    v = s.tri_v.astype(np.float64)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    with np.errstate(divide="ignore", invalid="ignore"):
        p = np.cross(d, e2)
        det = (e1 * p).sum(-1)
        q = np.cross(o - v[:, 0], e1)
        b1, b2 = ((o - v[:, 0]) * p).sum(-1) / det, (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        t = np.where((b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t > r[:, 3:4]), t, np.inf)
    best = t.min(1)
    # FP32 against FP64: a ray within rounding of an edge (about 1e-6 of the box) may decide otherwise
    ok = np.isclose(h[:, 0], best, rtol=1e-4, atol=1e-5) | (np.isinf(h[:, 0]) & np.isinf(best))
    assert ok.mean() >= 0.999, ok.mean()


@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (5, 3, 7, 1), (16, 16, 1, 2), (33, 8, 1, 5), (37, 23, 4, 6),
                                           (64, 64, 9, 0)])
@pytest.mark.parametrize("kind", ["random", "textured", "balls"])
def test_whole_paths_equal_the_waves(cuda, kind, w, h, spp, depth):
    # one launch per wave (blocks of 32 to 256 rays, remainders, a long tail) against one launch per kernel and bounce
    s = scenegen.textured(5) if kind == "textured" else _scene(kind)
    if kind != "textured":
        s.materials[s.tri_mat[0]] = dielectric(1.5)
    ds = pt.DeviceScene(s, pt.Accel(s))
    st = pt.RenderSettings(w, h, spp, no_direct_samples=4, max_depth=depth, rr_start_depth=3, seed=8)
    out, stats = [], []
    assert pt.tune_get("whole_paths") == -1
    try:
        for whole in (0, -1, 1 << 20):
            pt.tune("whole_paths", whole)
            f = pt.Film(w, h)
            pt.render(ds, st, f)
            out.append(f.raw())
            r = pt.render_stats()
            stats.append((r["extension_rays"], r["shadow_rays"], r["bounces"], r["paths"]))
    finally:
        pt.tune("whole_paths", -1)
    assert all(np.array_equal(out[0].view(np.uint32), o.view(np.uint32)) for o in out[1:])
    assert stats[0] == stats[1] == stats[2] or depth == 0 and stats[0][:2] == stats[1][:2] == stats[2][:2]


def test_a_triangle_outside_the_kd_trees_root_box(cuda):
    # flat quads from -1 to 1 do not widen the root box (Milton's fuzzy comparison), and are hit inside it only
    t = _random_tris(400, 12, size=0.05) * 0.5
    q = [scenegen.quad_tris((x, -1, 1), (x, 1, 1), (x, 1, -1), (x, -1, -1)) for x in (-0.9, 0.1, 0.9)]
    s = _soup(np.concatenate(q + [t]))
    a = pt.Accel(s)
    ds = pt.DeviceScene(s, a)
    rays = _rays(s, 5000, 13)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    assert (kd[:, 1].view(np.int32) >= 0).any()
    assert np.array_equal(kd.view(np.uint32), wide.view(np.uint32))
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


def _outside(kind):
    """Scenes with triangles that the kd-tree's root box leaves out: flat ones from -1 to 1, and points."""
    b = SceneBuilder()
    m = b.material(diffuse(0.6))
    t = (_random_tris(1500, 12, size=0.08) * 0.6).astype(np.float32)
    up = np.float32([0, 1, 0])
    b.add("t", t, np.broadcast_to(up, t.shape), m)
    y = float(t[..., 1].min())

    def quad(name, *c):
        v = scenegen.quad_tris(*c)
        b.add(name, np.asarray(v, np.float32), np.broadcast_to(up, (2, 3, 3)), m, culled=kind == "culled floor")

    if kind in ("floor", "culled floor"):
        quad("floor", (-1, y, 1), (1, y, 1), (1, y, -1), (-1, y, -1))
    if kind == "room":
        quad("floor", (-1, -1, 1), (1, -1, 1), (1, -1, -1), (-1, -1, -1))
        quad("top", (-1, 1, 1), (1, 1, 1), (1, 1, -1), (-1, 1, -1))
        quad("left", (-1, -1, 1), (-1, 1, 1), (-1, 1, -1), (-1, -1, -1))
        quad("right", (1, -1, 1), (1, 1, 1), (1, 1, -1), (1, -1, -1))
        quad("back", (-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1))
    if kind == "inside":
        quad("cut", (-1, 0.1, 1), (1, 0.1, 1), (1, 0.1, -1), (-1, 0.1, -1))
    if kind == "points":
        p = np.float32([[50, 0, 0], [-3e7, 1, 2], [0.1, 0.1, 0.1], [0, 1e30, 0]])
        b.add("points", np.repeat(p[:, None], 3, 1), np.broadcast_to(up, (4, 3, 3)), m)
    b.add_quad_light("light", (0.0, 0.45, 0.0), (0.1, 0.0, 0.0), (0.0, 0.0, 0.12), 15.0, m)
    return b.build(camera(eye=(0, 0.2, 1.7), look=(0, -0.1, -1), up=(0, 1, 0), height_angle=50.0, aspect=1.0))


@pytest.mark.parametrize("kind", ["floor", "culled floor", "room", "inside", "points"])
def test_triangles_that_the_root_box_leaves_out(cuda, kind):
    # the scene keeps its hierarchy; what such a triangle hides, and where it can be hit, is the kd-tree's answer
    s = _outside(kind)
    ds = pt.DeviceScene(s, pt.Accel(s))
    assert ds.hierarchy_nodes > 0
    box = _outside("none")
    for seed in (13, 14):
        rays = _rays(box, 6000, seed)
        out = sphere_rays(np.full(3, -1.3), np.full(3, 1.3), 20_000, seed + 10)
        rays = np.concatenate([rays, out]).astype(np.float32)
        kd, _ = gpu_trace(cuda, ds, rays, counts=True)
        wide, _ = gpu_trace(cuda, ds, rays)
        prim = kd[:, 1].view(np.int32)
        if kind != "points":
            assert (prim >= 1500).any()
        same = np.all(kd.view(np.uint32) == wide.view(np.uint32), axis=1)
        assert same.all(), (kind, int((~same).sum()), rays[~same][:2], kd[~same][:2], wide[~same][:2])
        assert np.array_equal(gpu_any(cuda, ds, rays) != 0, prim >= 0)
    films = []
    try:
        for wide, whole in ((1, -1), (1, 0), (0, 0)):
            pt.tune("wide", wide)
            pt.tune("whole_paths", whole)
            f = pt.Film(70, 50)
            pt.render(ds, pt.RenderSettings(70, 50, 9, max_depth=5, rr_start_depth=3, seed=7), f)
            films.append(np.array(f.raw()).view(np.uint32))
    finally:
        pt.tune("wide", 1)
        pt.tune("whole_paths", -1)
    assert all(np.array_equal(films[0], f) for f in films[1:])


@pytest.mark.parametrize("gap", [0.0, 1e-7, 1e-4, 0.05, -0.1])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_hits_on_triangles_that_the_root_box_leaves_out(cuda, gap, axis):
    # flat ones from -1 to 1 on both sides, on the root box's faces, beyond them and cutting through it: rays from
    # inside and outside that leave through the face before them, through another, or miss the box
    t = (_random_tris(1500, 21, size=0.08) * 0.6).astype(np.float32)
    box = t.reshape(-1, 3).min(0), t.reshape(-1, 3).max(0)
    q = []
    for v in (np.float32(box[0][axis] - gap), np.float32(box[1][axis] + gap)):
        f = np.asarray(scenegen.quad_tris((-1, v, 1), (1, v, 1), (1, v, -1), (-1, v, -1)), np.float32)
        q.append(np.roll(f, axis - 1, axis=-1))
    s = _soup(np.concatenate([q[0], t, q[1]]))
    ds = pt.DeviceScene(s, pt.Accel(s))
    assert ds.hierarchy_nodes > 0
    n = 20_000
    rng = np.random.default_rng(22)
    r = np.concatenate([sphere_rays(np.full(3, a), np.full(3, -a), n, 23 + k) for k, a in enumerate((-0.5, -1.1, -3.0))])
    r[::3, 4 + axis] *= 8.0           # steep
    r[1::3, 4 + axis] *= 0.05         # grazing
    r[::7, 4:7] = 0.0                 # along the axis
    r[::7, 4 + axis] = np.where(rng.random(len(r[::7])) < 0.5, -1.0, 1.0)
    r[::11, 0:3] = box[0] + (box[1] - box[0]) * rng.integers(0, 2, (len(r[::11]), 3))  # from the box's corners
    r[::5, 3] = rng.uniform(-0.5, 1.0, len(r[::5]))
    r[::10, 7] = r[::10, 3] + rng.uniform(0, 2.0, len(r[::10]))
    rays = r.astype(np.float32)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    prim = kd[:, 1].view(np.int32)
    assert ((prim >= 0) & (prim < 2)).any() and (prim >= s.ntri - 2).any()
    same = np.all(kd.view(np.uint32) == wide.view(np.uint32), axis=1)
    assert same.all(), (int((~same).sum()), rays[~same][:2], kd[~same][:2], wide[~same][:2])
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, prim >= 0)


@pytest.mark.parametrize("points", [1, 2, 3, 9, 40, 3000])
@pytest.mark.parametrize("floors", [0, 1, 3])
def test_scenes_of_which_the_root_box_leaves_out_everything(cuda, points, floors):
    # points, and flat triangles from -1 to 1: the root box is empty, and no bounds of it take part in the build
    rng = np.random.default_rng(points)
    t = [np.repeat(rng.uniform(-1, 1, (points, 1, 3)), 3, 1)]
    for y in np.linspace(-0.5, 0.5, floors):
        t.insert(rng.integers(len(t) + 1), scenegen.quad_tris((-1, y, 1), (1, y, 1), (1, y, -1), (-1, y, -1)))
    s = _soup(np.concatenate(t))
    ds = pt.DeviceScene(s, pt.Accel(s))
    rays = sphere_rays(np.full(3, -1.3), np.full(3, 1.3), 5000, points).astype(np.float32)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    assert np.array_equal(kd.view(np.uint32), gpu_trace(cuda, ds, rays)[0].view(np.uint32))
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


def test_which_scenes_have_the_hierarchy(cuda):
    for kind in KINDS + ["pile", "strip", "needles"]:
        if kind == "pile":       # one triangle many times: every area in the hierarchy is the same
            s = _soup(np.repeat(_random_tris(1, 3), 3000, 0))
        elif kind == "strip":    # copies of one in a row, a power of two apart
            t = np.float32([[0, 0, 0], [1, 0, 0], [0, 1, 0]])
            s = _soup(t + np.float32([1, 0, 0]) * 2.0 ** np.arange(-12, 12, 0.005)[:, None, None])
        elif kind == "needles":  # thin and long, side by side
            t = _random_tris(3000, 4, size=1e-4)
            t[:, 2, 0] += 3.0
            s = _soup(t)
        else:
            s = _scene(kind)
        n = pt.DeviceScene(s, pt.Accel(s)).hierarchy_nodes
        assert 0 < n <= 5 * s.ntri / 16 + 8, (kind, s.ntri, n)
    s = _overlaid("none")  # coordinates beyond what its nodes hold
    assert pt.DeviceScene(s, pt.Accel(s)).hierarchy_nodes == 0


@pytest.mark.parametrize("scale,nudge", [(1.0, 0), (1.0, 1), (1.0, -1), (1e9, 1), (1e-9, -1)])
def test_planes_at_the_roundings_of_16_bit_floats(cuda, scale, nudge):
    # axis-aligned quads on, just above and just below values that the nodes store exactly (eight leading
    # bits), on both sides of the centre: the rounding outward must not lose a quad, nor a sign
    x = np.concatenate([np.arange(128, 256, 8) / 256, 2.0 ** -np.arange(1, 9), [0.0]])
    x = np.unique(np.concatenate([x, -x])).astype(np.float32)
    for _ in range(abs(nudge)):
        x = np.nextafter(x, np.float32(np.inf * nudge))
    q = np.concatenate([scenegen.quad_tris((v, -1, 1), (v, 1, 1), (v, 1, -1), (v, -1, -1)) for v in x[::5]] +
                       [scenegen.quad_tris((-1, v, 1), (1, v, 1), (1, v, -1), (-1, v, -1)) for v in x[1::5]] +
                       [scenegen.quad_tris((a, b, c), (a + .02, b, c), (a + .02, b + .02, c), (a, b + .02, c))
                        for a in x[::4] for b in x[1::4] for c in x[2::4]])
    s = _soup(q.astype(np.float64) * scale)
    ds = pt.DeviceScene(s, pt.Accel(s))
    rays = _rays(_soup(q), 5000, 21)
    rays[:, 0:4] *= np.float32(scale)
    rays[:, 7] *= np.float32(scale)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    same = np.all(kd.view(np.uint32) == wide.view(np.uint32), axis=1)
    assert same.all(), (int((~same).sum()), rays[~same][:2], kd[~same][:2], wide[~same][:2])
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


@pytest.mark.parametrize("depth,bins,nds", [(2, False, 1), (3, False, 4), (0, False, 1), (7, True, 1)])
@pytest.mark.parametrize("kind", ["random", "balls", "batch"])
def test_traversals_that_share_a_launch_equal_separate_ones(cuda, kind, depth, bins, nds):
    # small waves trace a bounce's closest hits with the occlusion queries of the one before; per-kernel timing
    # keeps the launches apart
    scenes = [_scene("random"), scenegen.plain(4), _scene("n300")] if kind == "batch" else [_scene(kind)]
    ds = [pt.DeviceScene(s, pt.Accel(s)) for s in scenes]
    st = pt.RenderSettings(83, 61, 3, no_direct_samples=nds, max_depth=depth, rr_start_depth=2, seed=3)
    out, stats = [], []
    try:
        pt.tune("whole_paths", 0)
        if bins:
            pt.tune("bin_min_paths", 0)
        for timed in (False, True):
            films = [pt.Film(83, 61) for _ in ds]
            pt.profile_enable(timed)
            if kind == "batch":
                b = pt.Batch()
                for d, f in zip(ds, films):
                    b.add(d, st, f)
                b.render()
            else:
                pt.render(ds[0], st, films[0])
            r = pt.render_stats()
            out.append([f.raw() for f in films])
            stats.append((r["extension_rays"], r["shadow_rays"], r["bounces"], r["paths"]))
    finally:
        pt.profile_enable(False)
        pt.tune("whole_paths", -1)
        pt.tune("bin_min_paths", 1 << 25)
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(*out))
    assert stats[0] == stats[1]


@pytest.mark.parametrize("c", [1e-4, 1e-12, 2.0 ** -40, 1e-30, 1e-36, 1e-37, 1e-38, 3e-39, 2e-39, 1e-40, 1e-45])
@pytest.mark.parametrize("offset", [0.0, 1000.0])
def test_tiny_direction_components(cuda, c, offset):
    # the reciprocal of such a component is huge, its product with the origin beyond the largest float, or the
    # reciprocal itself infinite; origins on and off vertex planes, and far from the scene's centre
    s = _scene("random")
    ds = pt.DeviceScene(s, pt.Accel(s))
    rng = np.random.default_rng(17)
    n = 20_000
    v = s.tri_v.reshape(-1, 3)
    o = np.where(rng.random((n, 3)) < 0.4, v[rng.integers(0, len(v), n)], rng.uniform(v.min(0), v.max(0), (n, 3)))
    k = rng.integers(0, 3, n)
    side = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    o[np.arange(n), k] += offset * side
    d = np.where(rng.random((n, 3)) < 0.5, -c, c)
    one = rng.random(n) < 0.3  # one component tiny, the other not
    d[one, (k[one] + 1) % 3] = rng.uniform(-1, 1, one.sum())
    d[np.arange(n), k] = -side
    rays = np.concatenate([o, np.zeros((n, 1)), d, np.full((n, 1), np.inf)], 1).astype(np.float32)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    hit = kd[:, 1].view(np.int32) >= 0
    assert hit.any()
    assert np.array_equal(kd.view(np.uint32), wide.view(np.uint32))
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, hit)


@pytest.mark.parametrize("kind", ["flat", "plain", "random", "coincident", "points", "culled", "balls", "n7"])
@pytest.mark.parametrize("zeros", [1, 2])
def test_zero_components_in_vertex_planes(cuda, kind, zeros):
    # a ray in a split plane sees the cells on one side of it only: rays through vertices, along edges and beside
    # them, whose origin shares the vertex' coordinate along every axis that the direction does not have
    s = _scene(kind)
    ds = pt.DeviceScene(s, pt.Accel(s))
    rng = np.random.default_rng(23)
    n = 30_000
    v = s.tri_v.reshape(-1, 3)
    t = s.tri_v[rng.integers(0, s.ntri, n)].astype(np.float64)
    w = rng.dirichlet((1, 1, 1), n) * np.where(rng.random((n, 1)) < 0.2, 1.0, rng.integers(0, 2, (n, 3)))
    w /= np.maximum(w.sum(1, keepdims=True), 1e-9)
    at = (t * w[..., None]).sum(1).astype(np.float32)
    at = np.where(w.max(1, keepdims=True) == 1.0, t[np.arange(n), w.argmax(1)].astype(np.float32), at)
    o = rng.uniform(v.min(0) - 0.5, v.max(0) + 0.5, (n, 3)).astype(np.float32)
    zero = np.zeros((n, 3), bool)
    k = rng.integers(0, 3, n)
    zero[np.arange(n), k] = True
    if zeros == 2:
        zero[np.arange(n), (k + 1) % 3] = True
    o = np.where(zero, at, o)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = o
    rays[:, 4:7] = np.where(zero, np.where(rng.random((n, 3)) < 0.5, -0.0, 0.0), at - o)
    rays[:, 7] = np.where(rng.random(n) < 0.5, np.inf, rng.uniform(0.5, 1.5, n))
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    assert (kd[:, 1].view(np.int32) >= 0).any()
    same = np.all(kd.view(np.uint32) == wide.view(np.uint32), axis=1)
    assert same.all(), (int((~same).sum()), rays[~same][:2], kd[~same][:2], wide[~same][:2])
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


@pytest.mark.parametrize("length", [1e-38, 1e-30, 1e-20, 1e20, 1e30, 1e38])
def test_directions_of_any_length(cuda, length):
    s = _soup(_random_tris(3000, 10, size=0.1) * 50)
    ds = pt.DeviceScene(s, pt.Accel(s))
    rays = _rays(s, 4000, 19)
    rays[:, 4:7] = (rays[:, 4:7].astype(np.float64) * length).astype(np.float32)
    kd, _ = gpu_trace(cuda, ds, rays, counts=True)
    wide, _ = gpu_trace(cuda, ds, rays)
    assert np.array_equal(kd.view(np.uint32), wide.view(np.uint32))
    assert np.array_equal(gpu_any(cuda, ds, rays) != 0, kd[:, 1].view(np.int32) >= 0)


def _overlaid(kind):
    """Every triangle twice, with two materials; "none": and one whose coordinates the hierarchy does not hold."""
    b = SceneBuilder()
    m = [b.material(diffuse(0.8)), b.material(diffuse(0.1)), b.material(dielectric(1.5))]
    t = _random_tris(300, 5, size=0.4).astype(np.float32)
    n = np.broadcast_to(np.float32([0, 0, 1]), t.shape)
    for k in (0, 1, 0, 2):
        b.add(f"t{k}", t[::-1] if k else t, n, m[k])
    b.add_quad_light("l", (0.0, 0.0, 2.5), (0.5, 0.0, 0.0), (0.0, 0.5, 0.0), 8.0, m[0])
    if kind == "none":
        for x in (-2.9e37, 2.9e37):
            b.add(f"far{x}", np.float32([[[x, 0, 0], [x, 1, 0], [x, 0, 1]]]), np.float32([[[1, 0, 0]] * 3]), m[0])
    if kind == "spheres":
        b.add_sphere((0.2, 0.1, 0.3), 0.2, m[1])
    return b.build(camera(eye=(0, 0, 3), look=(0, 0, -1), up=(0, 1, 0), height_angle=40.0, aspect=1.0))


@pytest.mark.parametrize("whole", [0, -1])
def test_overlaid_surfaces_do_not_depend_on_the_batch(cuda, whole):
    # which of two coincident triangles a ray reports is decided by its scene, whatever shares the wave and
    # whichever structure the scene's rays traverse
    scenes = {k: _overlaid(k) for k in ("plain", "spheres", "none")}
    ds = {k: pt.DeviceScene(s, pt.Accel(s)) for k, s in scenes.items()}
    st = pt.RenderSettings(45, 37, 4, max_depth=4, rr_start_depth=3, seed=12)

    def films(kinds, batch):
        out = [pt.Film(45, 37) for _ in kinds]
        if batch:
            b = pt.Batch()
            for k, f in zip(kinds, out):
                b.add(ds[k], st, f)
            b.render()
        else:
            for k, f in zip(kinds, out):
                pt.render(ds[k], st, f)
        return {k: np.array(f.raw()).view(np.uint32) for k, f in zip(kinds, out)}

    try:
        pt.tune("whole_paths", whole)
        alone = films(scenes, False)
        assert all(a.any() for a in alone.values())
        groups = [films(g, True) for g in (("plain", "spheres"), ("plain", "none"), ("spheres", "none"),
                                           ("plain", "spheres", "none"))]
        pt.tune("wide", 0)
        groups += [films(scenes, False), films(scenes, True)]
    finally:
        pt.tune("wide", 1)
        pt.tune("whole_paths", -1)
    for i, g in enumerate(groups):
        for k, a in g.items():
            assert np.array_equal(alone[k], a), (i, k, int((alone[k] != a).sum()))
