"""The traversal walks where the node test and the warp triangle queue can go
wrong: rays along the axes (zero, negative-zero and vanishing direction
components), unnormalised directions, geometry far from and close to the
origin's scale, flat boxes, and coincident triangles of several instances,
whose exact ties resolve by (instance, primitive). Closest hits are bit-equal
to the oracle's brute arithmetic through both walks, at ray counts around a
warp's width."""
import numpy as np
import pytest

import oracle
from cenote_b200 import Scene, scenes

pytestmark = pytest.mark.gpu


def stacked(scale, offset):
    """Coincident quads and boxes: every surface appears in several instances."""
    at = scenes.translate(*offset) @ scenes.scale(scale)
    grey = scenes.matte((0.5, 0.5, 0.5))
    quad = scenes.quad([(-1, 0, -1), (-1, 0, 1), (1, 0, 1), (1, 0, -1)])
    wall = scenes.quad([(0, -1, -1), (0, 1, -1), (0, 1, 1), (0, -1, 1)])
    objs = []
    for _ in range(5):
        objs += [scenes.Object(quad, scenes.rows(at), grey), scenes.Object(wall, scenes.rows(at), grey),
                 scenes.Object(scenes.box(1.5, 1.5, 1.5), scenes.rows(at), grey)]
    ball = scenes.icosphere(2)
    objs += [scenes.Object(ball, scenes.rows(at @ scenes.translate(k * 0.1, 0, 0) @ scenes.scale(0.4)), grey)
             for k in range(3)]
    spec = scenes.furnace(grey)
    spec.objects = objs
    return spec


def edge_rays(n, scale, offset, seed):
    rng = np.random.default_rng(seed)
    org = rng.uniform(-2, 2, (n, 3))
    d = rng.normal(size=(n, 3))
    k = np.arange(n)
    axis = rng.integers(0, 3, n)
    for a in range(3):  # along an axis, with zeros of either sign and vanishing components
        on = (k % 4 == 0) & (axis != a)
        d[on, a] = np.where(rng.random(on.sum()) < 0.5, 0.0, -0.0)
        on = (k % 4 == 1) & (axis == a)
        d[on, a] = rng.choice([1e-20, -1e-20, 1e-37, -1e-37], on.sum())
        on = (k % 8 == 2) & (axis == a)  # origins on the surfaces' planes
        org[on, a] = rng.choice([-0.75, 0.0, 0.75, 1.0], on.sum())
    length = np.where(k % 5 == 0, rng.choice([1e-6, 1e6], n), 1.0)
    d = d / np.linalg.norm(d, axis=1, keepdims=True) * length[:, None]
    return ((org * scale + np.asarray(offset)).astype(np.float32)), d.astype(np.float32)


@pytest.mark.parametrize("scale,offset", [(1.0, (0, 0, 0)), (1e-3, (0, 0, 0)), (1.0, (3000.0, -70.0, 12345.0)),
                                          (1e4, (-5e4, 0, 2e4))])
def test_edge_rays_hit_as_the_oracle_says(ctx, scale, offset):
    spec = stacked(scale, offset)
    dev, ref = Scene(ctx, spec), oracle.OracleScene(spec)
    for n in (1, 31, 33, 40000):
        org, d = edge_rays(n, scale, offset, seed=n)
        rh, rt = ref.intersect(org, d)
        for queued in (False, True):
            hits, t = dev.probe_intersect(org, d, queued=queued)
            assert np.array_equal(hits, rh)
            assert np.array_equal(t, rt)
