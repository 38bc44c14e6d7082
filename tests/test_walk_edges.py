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


@pytest.mark.parametrize("name", ["stacked", "chart", "cornell", "axis_light"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (5, 1, 1), (67, 71, 1), (67, 71, 3), (137, 138, 1), (160, 120, 4)])
def test_short_queues_walk_to_the_same_hits(ctx, name, w, h, spp):
    """A queue of at most a few rays per warp is walked by eight lanes a ray,
    longer ones by a lane a ray with shared triangle tests, and on request by
    a lane a ray alone: the films and ray counts are the same, bit for bit,
    with coincident surfaces, axis-parallel rays and shadow rays to a target
    or to none. The sizes straddle the lengths where the walk changes."""
    from cenote_b200 import Film, Renderer

    if name == "stacked":
        spec = stacked(1.0, (0, 0, 0))
        spec.objects.append(scenes.Object(scenes.quad([(-1, 3, -1), (1, 3, -1), (1, 3, 1), (-1, 3, 1)]),
                                          scenes.rows(np.eye(4)), scenes.emitter((5.0, 5.0, 5.0))))
        spec.camera = scenes.Camera((2.5, 2.0, 3.0), (0.0, 0.0, 0.0))
    elif name == "axis_light":  # a distant light straight down: every shadow ray is axis-parallel
        spec = scenes.chart(env_size=(8, 4))
        spec.delta_lights = [scenes.DeltaLight(1, (0.0, -1.0, 0.0), (3.0, 3.0, 3.0))]
    else:
        spec = {"chart": lambda: scenes.chart(env_size=(64, 32)), "cornell": scenes.cornell}[name]()
    scene = Scene(ctx, spec)
    films = []
    for per_lane in (0, 1):
        r, f = Renderer(ctx, 8), Film(ctx, w, h)
        r.set_tuning(0, per_lane_triangles=per_lane)
        r.accumulate(scene, f, spp)
        st = r.stats()
        assert st["overflow"] == 0
        films.append((f.all_averages(), st["extension_rays"], st["shadow_rays"]))
    (a, *na), (b, *nb) = films
    assert na == nb
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
