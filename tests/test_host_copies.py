"""Images read back into pageable, pinned and unaligned host memory are the
same bytes, and a one-shot render's kept image buffer serves sizes up and down."""
import numpy as np
import pytest

from cenote_b200 import Film, Renderer, Scene, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (16, 16), (513, 512), (1024, 769)])
def test_film_reads_agree(ctx, w, h):
    torch = pytest.importorskip("torch")
    spec = scenes.cornell()
    scene, r, f = Scene(ctx, spec), Renderer(ctx, 2), Film(ctx, w, h)
    r.accumulate(scene, f, 1)
    pinned = torch.zeros((h, w, 4), dtype=torch.float32).pin_memory()
    f.averages_into(pinned.data_ptr())
    av = f.all_averages()
    assert np.array_equal(av["beauty"], pinned.numpy())
    assert np.array_equal(f.sums(), pinned.numpy())  # one sample: the sums are the averages
    assert np.array_equal(r.render(scene, w, h, 0), pinned.numpy())
    odd = np.zeros(w * h * 4 + 3, np.float32)[3:].reshape(h, w, 4)  # not 16-byte aligned
    assert np.array_equal(f.averages(odd), pinned.numpy())


def test_small_renders_after_large_ones(ctx):
    spec = scenes.cornell()
    scene, r = Scene(ctx, spec), Renderer(ctx, 3)
    small = r.render(scene, 20, 10, 5)
    r.render(scene, 700, 600, 5)
    assert np.array_equal(r.render(scene, 20, 10, 5), small)
