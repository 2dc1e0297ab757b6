"""Sorted queues against unsorted ones, and the carveout, where the waves run bounce by bounce: no ray is lost or
duplicated by the sort, and no knob changes an image."""
import numpy as np
import pytest

from milton_gb300 import pathtracer as pt
from milton_gb300 import scenegen
from milton_gb300.scene import dielectric

pytestmark = pytest.mark.gpu


@pytest.fixture
def knobs():
    names = ("whole_paths", "bin_extension", "bin_min_paths", "carveout")
    saved = {k: pt.tune_get(k) for k in names}
    yield
    for k, v in saved.items():
        pt.tune(k, v)


def _render(scenes, w, h, depth):
    films = [pt.Film(w, h) for _ in scenes]
    st = pt.RenderSettings(w, h, 8, no_direct_samples=2, max_depth=depth, rr_start_depth=3, seed=4)
    if len(scenes) == 1:
        pt.render(scenes[0], st, films[0])
    else:
        b = pt.Batch()
        for s, f in zip(scenes, films):
            b.add(s, st, f)
        b.render()
    r = pt.render_stats()
    return [np.array(f.raw()).view(np.uint32) for f in films], (r["extension_rays"], r["shadow_rays"], r["paths"])


# the last two: a wave without a depth cap that is drained to its end, and one whose tail of at most 500 rays
# leaves a sorted queue for one launch of whole paths
@pytest.mark.parametrize("kind,depth,whole", [("one", 6, 0), ("batch", 6, 0), ("one", 0, 0), ("one", 0, 500)])
@pytest.mark.parametrize("w,h", [(48, 40), (131, 77)])
def test_sorted_and_unsorted_queues_give_the_same_film(cuda, knobs, kind, depth, whole, w, h):
    scenes = [scenegen.random_scene(12, 20_000)] + ([scenegen.plain(4), scenegen.textured(5)] if kind == "batch" else [])
    scenes[0].materials[scenes[0].tri_mat[0]] = dielectric(1.5)
    ds = [pt.DeviceScene(s, pt.Accel(s)) for s in scenes]
    pt.tune("whole_paths", whole)
    pt.tune("bin_min_paths", 0)
    out = []
    for bins in (0, 1):
        pt.tune("bin_extension", bins)
        launches = pt.launch_count()
        out.append(_render(ds, w, h, depth) + (pt.launch_count() - launches,))
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0]))
    assert out[0][1] == out[1][1]
    assert out[1][2] > out[0][2]  # the sort ran


def test_the_carveout_changes_no_film(cuda, knobs):
    s = scenegen.random_scene(12, 20_000)
    ds = [pt.DeviceScene(s, pt.Accel(s))]
    out = []
    for whole in (0, -1):
        pt.tune("whole_paths", whole)
        for cv in (-2, -1, 0, 20, 100, -2):
            pt.tune("carveout", cv)
            out.append(_render(ds, 48, 40, 6))
    assert all(np.array_equal(o[0][0], out[0][0][0]) and o[1] == out[0][1] for o in out)


@pytest.mark.parametrize("kind", ["plain", "random", "textured"])
def test_whole_paths_and_waves_count_alike(cuda, knobs, kind):
    s = {"plain": scenegen.plain(3), "textured": scenegen.textured(5)}.get(kind) or scenegen.random_scene(9, 20_000)
    ds = [pt.DeviceScene(s, pt.Accel(s))]
    for depth in (0, 1, 5):
        out = []
        for whole in (0, 400, -1, 1 << 20):
            pt.tune("whole_paths", whole)
            f, n = _render(ds, 61, 33, depth)
            out.append((f[0], n + (pt.render_stats()["bounces"],)))
        assert all(np.array_equal(o[0], out[0][0]) and o[1] == out[0][1] for o in out), [o[1] for o in out]
