"""Waves around the sizes where the persistent grids change how they share a
queue (fewer items than warps, one batch a warp, more than the first batches
hold), with the shadow walks beside the next bounce and, when stage times are
taken, in turn on one stream: a film is the same bits however its samples are
split into waves and launched."""
import numpy as np
import pytest

from cenote_b200 import PROFILE_TIMING, Film, Renderer, Scene, scenes

pytestmark = pytest.mark.gpu


def film(ctx, scene, w, h, spp, bounces, spw=0, profiling=0):
    r, f = Renderer(ctx, bounces, samples_per_wave=spw), Film(ctx, w, h)
    r.set_profiling(profiling)
    r.accumulate(scene, f, spp)
    st = r.stats()
    assert st["overflow"] == 0
    return f.all_averages(), (st["extension_rays"], st["shadow_rays"])


@pytest.mark.parametrize("name", ["cornell", "chart", "textured"])
@pytest.mark.parametrize("w,h,spp,bounces", [(1, 1, 1, 1), (1, 1, 3, 2), (31, 1, 2, 8), (33, 7, 2, 8), (96, 99, 4, 5),
                                             (211, 90, 8, 3)])
def test_film_is_the_same_in_any_wave(ctx, name, w, h, spp, bounces):
    spec = {"cornell": scenes.cornell, "chart": lambda: scenes.chart(env_size=(64, 32)),
            "textured": lambda: scenes.textured(size=16)}[name]()
    scene = Scene(ctx, spec)
    base, rays = film(ctx, scene, w, h, spp, bounces)
    for kw in (dict(spw=1), dict(profiling=PROFILE_TIMING), dict(spw=2, profiling=PROFILE_TIMING)):
        got, n = film(ctx, scene, w, h, spp, bounces, **kw)
        assert n == rays, kw
        for k in base:
            assert np.array_equal(got[k], base[k], equal_nan=True), (kw, k)


def test_one_large_wave_is_the_small_waves(ctx):
    """More than 2^24 paths go in one wave where memory is plentiful; a guide
    that trains per wave keeps its 2^24; the films are the same bits."""
    from cenote_b200 import Guide

    scene = Scene(ctx, scenes.cornell())
    r, f = Renderer(ctx, 3), Film(ctx, 1024, 1024)
    r.accumulate(scene, f, 17)
    assert r.stats()["samples_per_wave"] == 17
    base = f.all_averages()
    r.set_samples_per_wave(16)
    f.reset()
    r.accumulate(scene, f, 17)
    for k, v in f.all_averages().items():
        assert np.array_equal(v, base[k], equal_nan=True), k
    guided = Renderer(ctx, 2)
    guided.set_guide(Guide(ctx, 1), 0.5, 0)
    f.reset()
    guided.accumulate(scene, f, 17)
    assert guided.stats()["samples_per_wave"] == 16


@pytest.mark.parametrize("name,w,h,sorts", [("chart", 511, 513, False), ("chart", 512, 512, True),
                                            ("textured", 511, 513, False), ("textured", 512, 512, True),
                                            ("cornell", 512, 512, False)])
def test_the_automatic_sort_changes_no_film(ctx, name, w, h, sorts):
    """On both sides of 2^18 paths, where the default starts to sort (a scene of
    one closure class never does), its film is each chosen mode's."""
    from cenote_b200 import SORT_ALL, SORT_NONE

    spec = {"cornell": scenes.cornell, "chart": lambda: scenes.chart(env_size=(64, 32)),
            "textured": lambda: scenes.textured(size=16)}[name]()
    scene, out = Scene(ctx, spec), []
    for mode in (None, SORT_ALL, SORT_NONE):
        r, f = Renderer(ctx, 4, material_sort=mode), Film(ctx, w, h)
        r.accumulate(scene, f, 1)
        out.append((f.all_averages(), r.stats()["kernel_launches"]))
    assert out[0][1] == out[1 if sorts else 2][1] and out[1][1] != out[2][1]
    for other, _ in out[1:]:
        for k, v in other.items():
            assert np.array_equal(v, out[0][0][k], equal_nan=True), k


def test_renderers_of_one_context_in_turn(ctx):
    """Two renderers taking turns, one with the L2 window on and both with their
    own side streams, draw the films they draw alone."""
    spec = scenes.chart(env_size=(64, 32))
    scene, other = Scene(ctx, spec), Scene(ctx, scenes.textured(size=16))

    def make():
        a, b = Renderer(ctx, 6), Renderer(ctx, 5)
        a.set_tuning(1, l2_window=1)
        return a, b

    sizes = (200, 121), (97, 300)
    alone = []
    for k, s in enumerate((scene, other)):
        r, f = make()[k], Film(ctx, *sizes[k])
        for n in (1, 3, 2):
            r.accumulate(s, f, n)
        alone.append(f.all_averages())
    plain = Film(ctx, *sizes[0])
    Renderer(ctx, 6).accumulate(scene, plain, 6)
    for k, v in plain.all_averages().items():
        assert np.array_equal(v, alone[0][k], equal_nan=True), k
    (a, b), (fa, fb) = make(), (Film(ctx, *sizes[0]), Film(ctx, *sizes[1]))
    shot = b.render(scene, 50, 40, 2)
    for n in (1, 3, 2):
        a.accumulate(scene, fa, n)
        b.accumulate(other, fb, n)
        assert np.array_equal(b.render(scene, 50, 40, 2), shot)
    for film, want in ((fa, alone[0]), (fb, alone[1])):
        for k, v in film.all_averages().items():
            assert np.array_equal(v, want[k], equal_nan=True), k
