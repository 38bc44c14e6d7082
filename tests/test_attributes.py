"""The per-triangle attribute records: the device finds each triangle's
instance among the concatenated meshes, so a mesh without triangles anywhere
in the list, and meshes of one triangle, must not shift the others'."""
import dataclasses

import numpy as np
import pytest

from cenote_b200 import Film, Renderer, Scene, scenes

pytestmark = pytest.mark.gpu


def film(ctx, spec):
    f = Film(ctx, 40, 30)
    Renderer(ctx, 6).accumulate(Scene(ctx, spec), f, 4)
    return f.all_averages()


@pytest.mark.parametrize("at", [0, 1, 4, 5])
@pytest.mark.parametrize("empty", [True, False])
def test_extra_meshes_leave_the_render_alone(ctx, at, empty):
    spec = scenes.textured(40, 30, 4, 6, size=16)
    base = film(ctx, spec)
    tri = scenes.Mesh(np.float32([[0, 500, 0], [1, 500, 0], [0, 500, 1]]), np.float32([[0, 1, 0]] * 3),
                      np.float32([[0, 0], [1, 0], [0, 1]]), np.uint32([[0, 2, 1]]))
    if empty:
        tri = dataclasses.replace(tri, indices=np.zeros((0, 3), np.uint32))
    objs = list(spec.objects)
    # Far above every surface and out of sight of the camera; no hit lands on it.
    objs[at:at] = [scenes.Object(tri, scenes.rows(np.eye(4)), scenes.matte((0.5, 0.5, 0.5)), camera_visible=False)] * 2
    got = film(ctx, dataclasses.replace(spec, objects=objs))
    for k in base:
        if empty:
            assert np.array_equal(got[k], base[k], equal_nan=True), k
        else:  # a stray ray may reach the triangle
            assert np.mean(np.all(np.atleast_1d(got[k] == base[k]), axis=-1)) > 0.98, k
