"""The library's host code over a device that computes nothing (fake_device.py):
what it allocates, keeps and hands to the kernels when memory runs short."""
import pytest

import fake_device


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_device.build(tmp_path_factory.mktemp("fake"))


def small_scene(ctx):
    from cenote_b200 import Scene, scenes

    return Scene(ctx, scenes.cornell())


def refused(call):
    from cenote_b200 import CenoteError

    with pytest.raises(CenoteError, match="out of memory"):
        call()


def a_refused_one_shot_image(lib):
    """A one-shot render whose image cannot be allocated fails, and the next one
    of that size or a smaller one allocates again: it never runs without an image."""
    from cenote_b200 import Context, Film, Renderer

    ctx = Context(0)
    scene, r = small_scene(ctx), Renderer(ctx, 2)
    r.accumulate(scene, Film(ctx, 512, 512), 1)  # the pool holds any of the waves below
    for w, h in ((100, 80), (256, 256), (300, 300)):
        lib.fake_refuse_after(0)
        refused(lambda: r.render(scene, w, h))
        assert r.render(scene, w // 2, h // 2).shape == (h // 2, w // 2, 4)
        assert r.render(scene, w, h).shape == (h, w, 4)
        assert lib.fake_bad_launches() == 0


def refused_growth(lib, make, small, large):
    """Refuse each allocation of a growth in turn: afterwards the small call, and
    then the large one, run on buffers that are theirs."""
    k = 0
    while True:
        state = make()
        small(state)
        lib.fake_refuse_after(k)
        try:
            large(state)
        except Exception as e:
            assert "out of memory" in str(e)
        else:
            break  # every allocation of the growth went through
        small(state)
        large(state)
        assert lib.fake_bad_launches() == 0, k
        k += 1
    lib.fake_refuse_after(-1)
    return k


def a_refused_pool(lib):
    from cenote_b200 import Context, Film, Guide, Renderer

    ctx = Context(0)
    scene = small_scene(ctx)
    films = Film(ctx, 32, 32), Film(ctx, 200, 100)
    guide = Guide(ctx, 1)

    def call(film):
        return lambda r: r.accumulate(scene, film, 2)

    def guided():
        r = Renderer(ctx, 2)
        r.set_guide(guide, 0.5, 0)
        return r

    for make, fields in ((lambda: Renderer(ctx, 2), 13), (guided, 15)):
        assert refused_growth(lib, make, call(films[0]), call(films[1])) >= fields


def refused_guide_lanes(lib):
    """The guide's lanes, refused on a pool that stays as it is."""
    from cenote_b200 import Context, Film, Guide, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 64, 64)
    guide = Guide(ctx, 1)

    def make():
        r = Renderer(ctx, 2)
        r.accumulate(scene, film, 1)
        return r

    def small(r):
        r.set_guide(None)
        r.accumulate(scene, film, 1)

    def large(r):
        r.set_guide(guide, 0.5, 0)
        r.accumulate(scene, film, 1)

    assert refused_growth(lib, make, small, large) >= 5


def a_refused_guide_batch(lib):
    import numpy as np

    from cenote_b200 import Context, Guide

    ctx = Context(0)

    def forward(n):
        return lambda g: g.forward(np.zeros((n, 96), np.float32))

    assert refused_growth(lib, lambda: Guide(ctx, 1), forward(100), forward(1000)) >= 6


def guide_lanes_fit_the_guided_wave(lib):
    """A guide attached after a large film takes the lanes of its own waves, not
    of the pool that the film left."""
    from cenote_b200 import Context, Film, Guide, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 1024, 1024)
    guide = Guide(ctx, 1)
    taken = []
    for samples in (0, 64):  # a fresh renderer, and one whose pool holds 2^26 paths
        r = Renderer(ctx, 2)
        if samples:
            r.accumulate(scene, film, samples)
            assert lib.fake_largest_wave() == 1 << 26
        r.set_guide(guide, 0.5, 0)
        r.accumulate(scene, film, 1)
        before = lib.fake_live_bytes()
        r.accumulate(scene, film, 64)
        taken.append(lib.fake_live_bytes() - before)
        r.close()
        assert lib.fake_bad_launches() == 0
    lanes = (15 << 20) * (48 * 4 + 4)  # 48 floats and a record index for 2^24 - 2^20 more paths
    assert taken[1] == lanes < taken[0]


def the_same_call_gets_the_same_wave(lib):
    """A film's waves do not shrink because the first call's pool took the memory
    that the wave size was chosen by."""
    from cenote_b200 import Context, Film, Renderer

    ctx = Context(0)
    scene = small_scene(ctx)
    for gb in (300, 120, 100, 65, 50):
        for w, h, n in ((1920, 1080, 64), (1280, 720, 64), (333, 217, 64), (5000, 4000, 3)):
            lib.fake_limit(lib.fake_live_bytes() + (gb << 30))
            r, film = Renderer(ctx, 2), Film(ctx, w, h)
            waves = []
            for k in range(3):
                asked = lib.fake_meminfo_calls()
                r.accumulate(scene, film, n)
                waves.append(r.stats()["samples_per_wave"])
                # Only a first call looks at the memory, unless it was refused the largest wave.
                assert k == 0 or lib.fake_meminfo_calls() == asked or w * h * waves[k] < 1 << 25
            assert waves[0] == waves[1] == waves[2], (gb, w, h, waves)
            assert w * h * waves[0] <= 1 << 26
            r.close()
            film.close()
    assert lib.fake_bad_launches() == 0


def large_pools_are_given_back(lib):
    """What does not fit beside a renderer's large pool gets its memory: the pool
    was taken because memory was plentiful."""
    import numpy as np

    from cenote_b200 import Context, Film, Guide, Renderer, Server

    ctx = Context(0)
    scene, film, guide = small_scene(ctx), Film(ctx, 1024, 1024), Guide(ctx, 1)
    other, image = Renderer(ctx, 2), Film(ctx, 640, 360)
    kept = []

    for call in (lambda: kept.append(Film(ctx, 3000, 2000)), lambda: kept.append(small_scene(ctx)),
                 lambda: other.accumulate(scene, image, 4), lambda: other.render(scene, 1000, 700),
                 lambda: guide.forward(np.zeros((50000, 96), np.float32)),
                 lambda: kept.append(Server(ctx, 40 << 30, pool_paths=1 << 20))):
        lib.fake_limit(lib.fake_live_bytes() + (200 << 30))
        r = Renderer(ctx, 2)
        film.reset()
        r.accumulate(scene, film, 64)
        assert r.stats()["samples_per_wave"] == 64
        lib.fake_limit(lib.fake_live_bytes() + 1000)  # nothing of any size fits
        call()
        film.reset()
        r.accumulate(scene, film, 64)  # and the renderer carries on, in smaller waves
        assert r.stats()["samples_per_wave"] == 16
        assert lib.fake_bad_launches() == 0
        r.close()
    for o in kept:
        o.close()


def one_shot_images_are_given_back(lib):
    """An image kept for a renderer's next one-shot render makes room for others,
    but not in that renderer's own call."""
    from cenote_b200 import Context, Film, Renderer

    ctx = Context(0)
    scene, r, other = small_scene(ctx), Renderer(ctx, 2, capacity=1 << 14), Renderer(ctx, 2)
    for call in (lambda: Film(ctx, 400, 400).close(), lambda: other.render(scene, 100, 100)):
        lib.fake_limit(lib.fake_live_bytes() + (10 << 30))
        r.render(scene, 2000, 2000)  # 64 MB kept
        lib.fake_limit(lib.fake_live_bytes() + 1000)
        call()
        lib.fake_limit(lib.fake_live_bytes() + (1 << 30))
        r.render(scene, 2000, 2000)
        assert lib.fake_bad_launches() == 0
    # A renderer's own image stays while room is made for its pool.
    fresh = Renderer(ctx, 2)
    lib.fake_refuse_after(1)
    fresh.render(scene, 500, 400)
    assert lib.fake_bad_launches() == 0


def a_refused_large_wave_is_a_plain_one(lib):
    """Memory that the device reports free but does not give: the call runs in
    waves of 2^24 paths, then and later."""
    from cenote_b200 import Context, Film, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 1024, 1024)
    # The shadow records are a wave's largest field, 64 bytes a path: the large wave is
    # refused from its first field on, or there.
    for above in (64 << 24, 63 << 26):
        lib.fake_refuse_above(above)
        r = Renderer(ctx, 2)
        for k in range(2):
            film.reset()
            r.accumulate(scene, film, 64)
            assert r.stats()["samples_per_wave"] == 16
        assert lib.fake_bad_launches() == 0
        r.close()


def a_capacity_bounds_the_waves(lib):
    """A renderer made with a capacity keeps to waves of 2^24 paths."""
    from cenote_b200 import Context, Film, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 1024, 1024)
    for capacity, samples, wave in ((0, 64, 1 << 26), (1 << 20, 16, 1 << 24), (3 << 20, 16, 1 << 24),
                                    (1 << 27, 16, 1 << 24), (1000, 1, 1000)):
        r = Renderer(ctx, 2, capacity=capacity)
        waves = lib.fake_waves()
        film.reset()
        r.accumulate(scene, film, 64 if capacity != 1000 else 1)
        assert r.stats()["samples_per_wave"] == samples, capacity
        assert lib.fake_waves() - waves == -(-(64 << 20 if capacity != 1000 else 1 << 20) // wave), capacity
        r.close()


def the_l2_window_covers_every_walk(lib):
    """With the L2 window on, the shadow walks' stream carries it as well as the
    closest-hit walks', and none is left when the call returns."""
    from cenote_b200 import PROFILE_TIMING, Context, Film, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 64, 64)
    for flags in (0, PROFILE_TIMING):
        r = Renderer(ctx, 4)
        r.set_profiling(flags)
        r.accumulate(scene, film, 2)
        assert lib.fake_windowed_walks() == (0 if flags == 0 else 7)
        shadows = lib.fake_window_free_shadows()
        r.set_tuning(1, l2_window=1)
        r.accumulate(scene, film, 2)
        assert lib.fake_window_free_shadows() == shadows
        assert lib.fake_windowed_walks() == (7 if flags == 0 else 14)  # 4 closest-hit and 3 shadow walks
        assert lib.fake_open_windows() == 0
        r.set_tuning(1)
        r.accumulate(scene, film, 2)
        assert lib.fake_window_free_shadows() == shadows + 3


def waits_keep_their_bounds(lib):
    """Work that never ends is reported after the call's own bound: a minute for
    the guide's calls, ten for a render's."""
    import numpy as np

    from cenote_b200 import CenoteError, Context, Film, Guide, Renderer

    ctx = Context(0)
    scene, film, guide, r = small_scene(ctx), Film(ctx, 16, 16), Guide(ctx, 1), Renderer(ctx, 2)
    feats, dirs = np.zeros((10, 96), np.float32), np.ones((10, 3), np.float32)
    for bound, call in ((60, lambda: guide.forward(feats)),
                        (60, lambda: guide.train_step(feats, dirs, np.ones(10, np.float32), 0.0)),
                        (600, lambda: r.accumulate(scene, film, 1)), (600, lambda: film.averages()),
                        (600, lambda: film.sums())):
        lib.fake_hang(1)
        before = lib.fake_clock_ms()
        with pytest.raises(CenoteError, match="did not finish"):
            call()
        lib.fake_hang(0)
        assert bound <= (lib.fake_clock_ms() - before) / 1e3 <= bound + 1


def the_sort_stays_automatic_until_a_mode_is_chosen(lib):
    """Reading a renderer's knobs and writing them back, or setting another knob,
    leaves the automatic sort on; a mode holds for every wave."""
    from cenote_b200 import SORT_ALL, SORT_AUTO, SORT_NONE, SORT_SECONDARY, CenoteError, Context, Film, Renderer

    ctx = Context(0)
    scene, film = small_scene(ctx), Film(ctx, 32, 32)  # a wave that skips the sort

    def sorts(r):
        before = lib.fake_sorts()
        r.accumulate(scene, film, 1)
        return lib.fake_sorts() - before

    r = Renderer(ctx, 3)
    assert sorts(r) == 0
    t = r.tuning()
    assert t["material_sort"] == SORT_AUTO
    t.pop("ms_per_sample")
    r.set_tuning(**t)
    assert r.tuning()["material_sort"] == SORT_AUTO and sorts(r) == 0
    r.set_tuning(**{**t, "refill_idle": 8})
    assert sorts(r) == 0
    for mode, n in ((SORT_ALL, 3), (SORT_SECONDARY, 2), (SORT_NONE, 0)):
        r.set_material_sort(mode)
        assert r.tuning()["material_sort"] == mode and sorts(r) == n
        r.set_tuning(**{**t, "material_sort": mode, "refill_idle": 4})
        assert sorts(r) == n
    for bad in (3, 0xFFFFFFFE):
        with pytest.raises(CenoteError):
            r.set_material_sort(bad)
        with pytest.raises(CenoteError):
            r.set_tuning(bad)
    r.set_material_sort(SORT_AUTO)
    assert sorts(r) == 0
    before = r.tuning()
    lib.fake_refuse_after(5)  # the film is there, the pool is not
    refused(lambda: r.autotune(scene, 256, 256))
    assert r.tuning() == before
    assert r.autotune(scene, 32, 32)["material_sort"] in (SORT_NONE, SORT_ALL, SORT_SECONDARY)


def meshes_are_staged_and_given_back(lib):
    """Whatever the meshes' sizes, the device finds their streams end to end, and
    staging memory of 64 MB and more is gone before the tree is built."""
    import ctypes

    import numpy as np

    from cenote_b200 import BVH_GPU_SAH, BVH_HOST_SAH, Context, Scene, scenes

    ctx = Context(0)
    rng = np.random.default_rng(3)

    def mesh(vertices, triangles):
        f = lambda n: rng.random((vertices, n), np.float32)
        return scenes.Mesh(f(3), f(3), f(2), rng.integers(0, vertices, (triangles, 3)).astype(np.uint32))

    # Runs below, at and above the sizes that are gathered (64 KB) and flushed (256 KB).
    sizes = [(1, 1), (3, 0), (5461, 5461), (5462, 5462), (8191, 5461), (8192, 3), (3, 5462), (30000, 40000)]
    sizes += [(5000, 5000)] * 9 + [(1, 0)]
    late = 0
    for builder in (BVH_HOST_SAH, BVH_GPU_SAH):
        ctx.set_bvh_builder(builder)
        for order in (sizes, sizes[::-1], sizes[:1], sizes[1:2], [(1, 1), (2 << 20, 5), (3, 2)]):
            spec = scenes.cornell()
            meshes = [mesh(*n) for n in order]
            spec.objects = [scenes.Object(m, scenes.rows(np.eye(4)), scenes.matte((0.5, 0.5, 0.5))) for m in meshes]
            Scene(ctx, spec).close()
            for k, name in enumerate(("positions", "normals", "uvs", "indices")):
                n = ctypes.c_uint64()
                data = lib.fake_stream(k, ctypes.byref(n))
                want = b"".join(np.ascontiguousarray(getattr(m, name)).tobytes() for m in meshes)
                assert ctypes.string_at(data, n.value) == want, (k, len(order))
            staged = 32 * sum(v for v, _ in order) + 12 * sum(t for _, t in order)
            late += staged < 64 << 20
            assert lib.fake_late_stages() == late
    assert late == 8  # of ten scenes, all but the two with the large mesh


def a_mesh_without_arrays_is_refused(lib):
    """Counts of an object that is refused are not acted on."""
    import ctypes

    import cenote_b200
    from cenote_b200 import CenoteError, Context, scenes

    ctx = Context(0)
    cam = cenote_b200._c_camera(scenes.cornell().camera)
    texel = (ctypes.c_float * 4)()
    env = cenote_b200.EnvironmentC(1, 1, ctypes.addressof(texel))
    objects = (cenote_b200.Object * 4096)()
    for o in objects:
        o.vertex_count, o.triangle_count = 0xFFFFFFFF, 0
        for slot in ("base_color", "specular_roughness", "metalness", "emission", "opacity", "normal"):
            setattr(o.material, slot + "_texture", 0xFFFFFFFF)
    h = ctypes.c_void_p()
    with pytest.raises(CenoteError, match="object 0 lacks attributes"):
        cenote_b200._check(lib.cenote_scene_create(ctx.handle, objects, len(objects), ctypes.byref(cam),
                                                   ctypes.byref(env), None, 0, ctypes.byref(h)))


SCENARIOS = {f.__name__: f for f in (a_refused_one_shot_image, a_refused_pool, refused_guide_lanes,
                                     a_refused_guide_batch, guide_lanes_fit_the_guided_wave,
                                     the_same_call_gets_the_same_wave, large_pools_are_given_back,
                                     one_shot_images_are_given_back, a_refused_large_wave_is_a_plain_one,
                                     a_capacity_bounds_the_waves,
                                     the_l2_window_covers_every_walk, waits_keep_their_bounds,
                                     the_sort_stays_automatic_until_a_mode_is_chosen,
                                     meshes_are_staged_and_given_back, a_mesh_without_arrays_is_refused)}


@pytest.mark.parametrize("name", SCENARIOS)
def test_host(fake, name):
    fake_device.run(fake, __file__, name)


if __name__ == "__main__":
    fake_device.main(SCENARIOS)
