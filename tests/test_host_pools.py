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


SCENARIOS = {f.__name__: f for f in (a_refused_one_shot_image,)}


@pytest.mark.parametrize("name", SCENARIOS)
def test_host(fake, name):
    fake_device.run(fake, __file__, name)


if __name__ == "__main__":
    fake_device.main(SCENARIOS)
