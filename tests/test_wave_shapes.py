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
