"""Film reads into page-locked and pageable arrays, at the sizes where the pieces end, and the pool of
page-locked result arrays."""
import ctypes as C
import gc

import numpy as np
import pytest

from milton_gb300 import _native as N
from milton_gb300 import hostmem
from milton_gb300 import pathtracer as pt
from milton_gb300 import scenegen

pytestmark = pytest.mark.gpu


# 65,536 x 4 = one piece exactly, + 4 one more, 2 pieces and a remainder, one pixel, a tile of 256 and more
@pytest.mark.parametrize("w,h", [(1, 1), (16, 16), (257, 1), (512, 512), (65537, 4), (1025, 770)])
@pytest.mark.parametrize("kind", ["none", "mitchell"])
def test_mean_is_the_same_in_any_memory(cuda, w, h, kind):
    s = scenegen.plain(0)
    ds = pt.DeviceScene(s, pt.Accel(s))
    f = pt.Film(w, h)
    if kind != "none":
        f.set_filter(kind, 3.0)
    pt.render(ds, pt.RenderSettings(w, h, 2, max_depth=2, rr_start_depth=3, seed=3), f)
    pinned = f.mean()
    pageable = np.full((h, w, 3), np.nan)
    N.check(N.load().mgpu_film_read(f.handle, N.ptr(pageable), None))
    assert np.array_equal(pinned, pageable)
    if kind == "none":
        raw = f.raw().astype(np.float64)
        n = raw[0, ..., 3:4]
        assert np.array_equal(pageable, (raw[0, ..., :3] - raw[1, ..., :3]) / n)
        # the estimate of the kernel against the same formula on the host (FP64 sums in another order)
        assert pt.film_error([f])[0] == pytest.approx(pt.rmse_estimate(f.raw()), rel=1e-9, abs=1e-15)
    rgba = np.zeros((h, w, 4), np.uint8)
    N.check(N.load().mgpu_film_tonemap(f.handle, N.ptr(rgba), None))
    assert np.array_equal(rgba, f.tonemap())


def test_pool_gives_blocks_back_and_stays_bounded(cuda):
    before = hostmem._total
    a = hostmem.empty((1 << 17,), np.float64)
    a[:] = 1.0
    view = a[5:10]
    addr = a.ctypes.data
    del a
    gc.collect()
    b = hostmem.empty((1 << 17,), np.float64)  # the view still holds the first block
    assert b.ctypes.data != addr and np.all(view == 1.0)
    del view
    gc.collect()
    c = hostmem.empty((1 << 17,), np.float64)
    assert c.ctypes.data == addr
    del b, c
    gc.collect()
    keep = [hostmem.empty((48 << 20,), np.uint8) for _ in range(8)]  # beyond the limit: ordinary arrays
    assert hostmem._total <= hostmem.LIMIT and all(k.nbytes == 48 << 20 for k in keep)
    del keep
    gc.collect()
    assert hostmem._total <= max(before, hostmem.LIMIT)
    p = C.c_void_p()
    assert N.load().mgpu_host_alloc(0, C.byref(p)) != N.MGPU_OK


def test_a_failed_allocation_does_not_fail_the_next_call(cuda):
    s = scenegen.plain(0)
    ds = pt.DeviceScene(s, pt.Accel(s))
    st = pt.RenderSettings(64, 48, 2, max_depth=2, rr_start_depth=3, seed=3)
    f, g = pt.Film(64, 48), pt.Film(64, 48)
    pt.render(ds, st, f)
    want = f.mean(), f.tonemap()
    lib = N.load()

    def fail():
        p = C.c_void_p()
        assert lib.mgpu_host_alloc(1 << 60, C.byref(p)) != N.MGPU_OK and not p.value

    fail()
    pt.render(ds, st, g)
    fail()
    assert np.array_equal(g.mean(), want[0])
    fail()
    assert np.array_equal(g.tonemap(), want[1])
    fail()
    assert pt.film_error([g])[0] == pt.film_error([f])[0]
    fail()
    assert pt.DeviceScene(s, pt.Accel(s)).nbytes == ds.nbytes


@pytest.mark.parametrize("kind", ["none", "triangle"])
@pytest.mark.parametrize("part", ["pageable", "head", "tail", "whole", "two", "block", "inside", "beyond"])
def test_arrays_of_which_a_part_is_page_locked(cuda, kind, part):
    # the device writes only what lies in one block of mgpu_host_alloc; any other memory is filled by copies, be
    # its first byte page-locked or not
    page = 1 << 16
    w, h = 173, 211
    s = scenegen.plain(0)
    ds = pt.DeviceScene(s, pt.Accel(s))
    f = pt.Film(w, h)
    if kind != "none":
        f.set_filter(kind, 2.0)
    pt.render(ds, pt.RenderSettings(w, h, 2, max_depth=2, rr_start_depth=3, seed=3), f)
    want = np.array(f.mean()), np.array(f.tonemap())
    lib, rt = N.load(), cuda.cuda.cudart()
    for img, read in zip(want, (lib.mgpu_film_read, lib.mgpu_film_tonemap)):
        size = -(-img.nbytes // page) * page + 2 * page
        block, ranges = C.c_void_p(), []
        if part in ("block", "inside", "beyond"):
            # the array: the whole block, its end, or ordinary memory
            N.check(lib.mgpu_host_alloc(img.nbytes + (page if part == "inside" else 0), C.byref(block)))
            at = block.value + (page if part == "inside" else 0)
            if part == "beyond":
                raw = np.zeros(size, np.uint8)
                at = -(-raw.ctypes.data // page) * page
        else:
            raw = np.zeros(size, np.uint8)
            at = -(-raw.ctypes.data // page) * page
            half = img.nbytes // 2 // page * page
            ranges = {"pageable": [], "head": [(0, half)], "tail": [(half, page)], "whole": [(0, size - page)],
                      "two": [(0, half), (half, page)]}[part]
        for first, n in ranges:
            assert n > 0 and int(rt.cudaHostRegister(at + first, n, 0)) == 0
        try:
            N.check(read(f.handle, at, None))
            got = np.ctypeslib.as_array((C.c_uint8 * img.nbytes).from_address(at)).view(img.dtype).reshape(img.shape)
            assert np.array_equal(got, img)
            del got
        finally:
            for first, _ in ranges:
                rt.cudaHostUnregister(at + first)
            if block:
                N.check(lib.mgpu_host_free(block))


def test_a_copy_from_a_result_outlives_it(cuda):
    # a copy that waits behind a frame on another stream; its source, a temporary result, is gone and the next
    # result is read meanwhile
    s = scenegen.random_scene(3, 20_000)
    ds = pt.DeviceScene(s, pt.Accel(s))
    films = [pt.Film(256, 200) for _ in range(2)]
    for k, f in enumerate(films):
        pt.render(ds, pt.RenderSettings(256, 200, 2, max_depth=2, rr_start_depth=3, seed=k), f)
    want = [np.array(f.mean()) for f in films]
    assert not np.array_equal(*want)
    side, big = cuda.cuda.Stream(), pt.Film(1024, 1024)
    cuda.cuda.synchronize()
    for read, want in ((pt.Film.mean, want), (pt.Film.raw, [np.array(f.raw()) for f in films])):
        with cuda.cuda.stream(side):
            pt.render(ds, pt.RenderSettings(1024, 1024, 16, max_depth=6, rr_start_depth=3, seed=5), big)
            got = cuda.from_numpy(read(films[0], stream=cuda.cuda.default_stream())).to("cuda", non_blocking=True)
        again = read(films[1], stream=cuda.cuda.default_stream())
        cuda.cuda.synchronize()
        assert np.array_equal(got.cpu().numpy(), want[0]) and np.array_equal(again, want[1])


def test_error_estimates_of_films_of_uneven_size(cuda):
    # each film by itself and all in one call give the same bits, and the scratch follows the sum of the sizes
    s = scenegen.plain(0)
    ds = pt.DeviceScene(s, pt.Accel(s))
    films = []
    for k, (w, h) in enumerate([(1, 1), (37, 23), (1600, 1400), (256, 513), (2, 3)] + [(8, 8)] * 60):
        films.append(pt.Film(w, h))
        pt.render(ds, pt.RenderSettings(w, h, 4, max_depth=2, rr_start_depth=3, seed=k), films[-1])
    alone = [pt.film_error([f])[0] for f in films]
    assert np.array_equal(pt.film_error(films), alone)
    assert np.array_equal(pt.film_error(films[::-1]), alone[::-1])
    many = [films[2]] + [films[5]] * 20_000
    free = cuda.cuda.mem_get_info()[0]
    pt.film_error(many)
    assert free - cuda.cuda.mem_get_info()[0] < 64 << 20  # 21 MB, not a row of the largest film's blocks for each
    got = pt.film_error(many)
    assert got[0] == alone[2] and (got[1:] == alone[5]).all()


@pytest.mark.parametrize("w,h", [(2048, 2048), (2048, 2049), (2897, 2897)])
@pytest.mark.parametrize("kind", ["none", "box"])
def test_means_of_more_pixels_than_the_scratch_holds(cuda, w, h, kind):
    # one piece exactly, one row more, two pieces and a remainder, against the one store of a page-locked array
    s = scenegen.plain(0)
    ds = pt.DeviceScene(s, pt.Accel(s))
    f = pt.Film(w, h)
    if kind != "none":
        f.set_filter(kind, 1.0)
    pt.render(ds, pt.RenderSettings(w, h, 1, max_depth=1, rr_start_depth=3, seed=3), f)
    lib, p = N.load(), C.c_void_p()
    N.check(lib.mgpu_host_alloc(w * h * 24, C.byref(p)))
    try:
        N.check(lib.mgpu_film_read(f.handle, p, None))
        direct = np.ctypeslib.as_array((C.c_double * (w * h * 3)).from_address(p.value)).reshape(h, w, 3)
        assert direct.any() and np.array_equal(f.mean(), direct)
        del direct
    finally:
        N.check(lib.mgpu_host_free(p))


@pytest.mark.parametrize("off", [0, 8, 24])
@pytest.mark.parametrize("new", [False, True])
def test_a_result_inside_a_larger_array(cuda, off, new):
    # the pages of a result are made before the copy: with the bytes beside it in them, new and old ones
    w, h = 150, 111
    ds = pt.DeviceScene(scenegen.plain(0), pt.Accel(scenegen.plain(0)))
    f = pt.Film(w, h)
    pt.render(ds, pt.RenderSettings(w, h, 1, max_depth=2), f)
    want, n = f.mean(), h * w * 3
    lib = pt.N.load()
    big = np.zeros(n + 4 * 16384) if new else np.full(n + 4 * 16384, 7.0)
    keep = 0.0 if new else 7.0
    part = big[16384 + off // 8:][:n]
    pt.N.check(lib.mgpu_film_read(f.handle, pt.N.ptr(part), None))
    assert np.array_equal(part.reshape(h, w, 3), want)
    assert np.all(big[:16384 + off // 8] == keep) and np.all(big[16384 + off // 8 + n:] == keep)
