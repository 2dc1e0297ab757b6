"""Creating scenes beside other work, and the memory that they take."""
import ctypes as C

import numpy as np
import pytest

from milton_gb300 import _native as N
from milton_gb300 import pathtracer as pt
from milton_gb300 import scenegen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [0, 30_000])
def test_it_waits_for_no_other_stream(cuda, tris):
    # both sides of the size above which the hierarchy is built by more than one block
    big = scenegen.random_scene(3, 60_000)
    s = scenegen.random_scene(4, tris) if tris else scenegen.plain(1)
    big_ds, acc = pt.DeviceScene(big, pt.Accel(big)), pt.Accel(s)
    film = pt.Film(1024, 1024)
    st = pt.RenderSettings(1024, 1024, 64, max_depth=8, rr_start_depth=3, seed=1)
    pt.render(big_ds, st, film)
    first = pt.DeviceScene(s, acc)  # kernels loaded, staging page-locked
    a, b = cuda.cuda.Stream(), cuda.cuda.Stream()
    cuda.cuda.synchronize()
    ev = cuda.cuda.Event()
    with cuda.cuda.stream(a):
        for _ in range(3):
            pt.render(big_ds, st, film)
        ev.record()
    second = pt.DeviceScene(s, acc, stream=b)
    assert not ev.query()
    cuda.cuda.synchronize()
    assert second.hierarchy_nodes == first.hierarchy_nodes > 0


@pytest.mark.parametrize("depth", [0, 1, 24])
@pytest.mark.parametrize("tris", [500, 2048, 5000])
def test_bytes_are_those_announced(cuda, tris, depth):
    # kd-trees of few records: the build's scratch is larger than the arrays whose place it takes
    rng = np.random.default_rng(5)
    s = scenegen.random_scene(6, 500)
    keep = rng.integers(0, s.ntri, tris)
    s.tri_v, s.tri_n = (np.ascontiguousarray(x[keep]) for x in (s.tri_v, s.tri_n))
    s.tri_mat, s.tri_light, s.tri_flags = (np.ascontiguousarray(x[keep]) for x in (s.tri_mat, s.tri_light, s.tri_flags))
    if s.tri_uv is not None:
        s.tri_uv = np.ascontiguousarray(s.tri_uv[keep])
    acc = pt.Accel(s, pt.KdSettings(max_depth=depth))
    ds = pt.DeviceScene(s, acc)
    n = C.c_uint64()
    N.check(N.load().mgpu_scene_device_bytes(C.byref(pt._desc(s)), acc.handle, C.byref(n)))
    assert ds.nbytes == n.value and ds.hierarchy_nodes > 0
    f, g = pt.Film(40, 30), pt.Film(40, 30)
    st = pt.RenderSettings(40, 30, 4, max_depth=4, rr_start_depth=3, seed=2)
    pt.render(ds, st, f)
    try:
        pt.tune("wide", 0)
        pt.render(ds, st, g)
    finally:
        pt.tune("wide", 1)
    assert np.array_equal(f.raw().view(np.uint32), g.raw().view(np.uint32))
