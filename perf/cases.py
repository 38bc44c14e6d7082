"""The renderer's measured cases: what a user has it do, through the package's public API.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (a resident scene, a renderer, a film, an output buffer), `run` is one
call as a program makes it, `work` the bytes and operations it cannot do
without. Renders have no 64-bit counterpart to compare with (a path tracer's
Monte Carlo estimate follows every rounding of its own paths), so `exact`
answers for the learned guide's training step and the loaded scene's hits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cenote_b200 import (LIGHT_SAMPLING_BSDF, LIGHT_SAMPLING_MIS, LIGHT_SAMPLING_NEE, Context, Film, Guide, Renderer,
                         Scene, Server, scenes)

SAMPLING = {"mis": LIGHT_SAMPLING_MIS, "bsdf": LIGHT_SAMPLING_BSDF, "nee": LIGHT_SAMPLING_NEE}

# ---- the cases ------------------------------------------------------------------
#
# kind "snapshot": Renderer.render, one sample of every pixel into host memory.
# kind "viewport": an interactive step: the film reset, a few samples, the
#                  display frame tonemapped into device memory.
# kind "film":     an offline frame: all samples, then the beauty averages into
#                  pinned host memory.
# kind "aov":      an offline frame with every denoiser guide read back.
# kind "serve":    a batch of progressive jobs through the server.
# kind "train":    one training step of the learned guide over a batch.
# kind "load":     a scene built from host arrays, then probed with rays.


def _render(name, kind, scene, width, height, spp, bounces, **more):
    return dict(name=name, kind=kind, scene=scene, width=width, height=height, spp=spp, bounces=bounces,
                sampling="mis", **more)


def listed():
    return [
        # The smallest call: a thumbnail of a simple scene, where launches and the host's share count.
        _render("snapshot_box_64", "snapshot", "box", 64, 64, 1, 8),
        # The closed box at its own size and sample count: a frame of 1 M paths.
        _render("film_box_256", "film", "box", 256, 256, 16, 8),
        # A viewer moving through the material chart: one sample per displayed frame.
        _render("viewport_chart_640x360", "viewport", "chart", 640, 360, 1, 12),
        # A viewer over the large scene at an odd window size: textures, every lobe, many emitters.
        _render("viewport_terrain_853x479", "viewport", "terrain", 853, 479, 2, 16),
        # A draft of the chart at a ragged size: no side is a multiple of a tile.
        _render("film_chart_333x217", "film", "chart", 333, 217, 8, 12),
        # The material chart's frame: 59 M paths under an HDRI sun sky.
        _render("film_chart_1280x720", "film", "chart", 1280, 720, 64, 12),
        # The largest frame: the 3 M-triangle terrain at full size and sample count.
        _render("film_terrain_1920x1080", "film", "terrain", 1920, 1080, 64, 16),
        # Every texture slot with a cut-out leaf (fractional opacity), all guides read back for a denoiser.
        _render("aov_textured_957x541", "aov", "textured", 957, 541, 16, 6),
        # Directional guiding by a fixed network on a scene lit by one bounce.
        _render("film_guided_256", "film", "ceiling", 256, 256, 16, 8, guided=True),
        # Jobs of several sizes over two scenes, as a render service takes them.
        dict(name="serve_12_jobs", kind="serve", jobs=12, most_spp=16, side=640),
        # One step of online training at the renderer's batch size.
        dict(name="train_guide_65536", kind="train", rows=65536),
        # Opening a scene: host arrays to a resident, traceable scene.
        dict(name="load_terrain_grid256", kind="load", grid=256, env_width=512, rays=2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["snapshot", "viewport", "viewport", "film", "film", "film", "film", "aov", "aov", "serve",
                       "train", "load"])
    if kind == "serve":
        return dict(kind=kind, jobs=rng.randint(2, 16), most_spp=rng.randint(2, 16), side=_log_int(rng, 96, 800))
    if kind == "train":
        return dict(kind=kind, rows=_log_int(rng, 100, 65536))
    if kind == "load":
        return dict(kind=kind, grid=_log_int(rng, 33, 600), env_width=2 * _log_int(rng, 16, 512), rays=2048)
    scene, bounces = rng.choice([("box", 8), ("chart", 12), ("chart", 12), ("terrain", 16), ("textured", 6),
                                 ("ceiling", 8)])
    width = _log_int(rng, 24, 1920)
    height = max(1, min(1080, int(width * rng.uniform(0.5, 1.1))))
    most = {"snapshot": 1, "viewport": 4}.get(kind, min(64, max(1, (1 << 26) // (width * height))))
    case = dict(kind=kind, scene=scene, width=width, height=height, spp=_log_int(rng, 1, most),
                bounces=rng.choice([bounces, bounces, rng.randint(2, bounces)]),
                sampling=rng.choice(["mis", "mis", "mis", "bsdf", "nee"]))
    if scene == "ceiling" and kind in ("film", "aov") and rng.random() < 0.7:
        case["guided"] = True
        case["spp"] = min(case["spp"], 16)
    return case


# ---- inputs ---------------------------------------------------------------------


def _recolour(spec, rng):
    """The scene with its diffuse and metal colours and its camera moved a little."""
    for o in spec.objects:
        m = o.material.copy()
        m["base_color"] = np.clip(m["base_color"] * rng.uniform(0.8, 1.1, 3), 0.0, 1.0)
        o.material = m
    c = spec.camera
    c.position = tuple(float(p + d) for p, d in zip(c.position, rng.uniform(-0.06, 0.06, 3)))
    return spec


def _spec(name, seed):
    rng = np.random.default_rng(seed)
    if name == "terrain":
        return scenes.large(texture_size=256, textures=128, seed=1 + seed % 1000003)
    if name == "chart":
        spec = scenes.chart(env_size=(4, 2))
        spec.environment = scenes.sky_hdri(2048, 1024, sun_azimuth_deg=float(rng.uniform(-60.0, 60.0)),
                                           sun_elevation_deg=float(rng.uniform(20.0, 60.0)))
        return _recolour(spec, rng)
    if name == "textured":
        return _recolour(scenes.textured(size=256, seed=7 + seed % 1000003), rng)
    if name == "ceiling":
        return _recolour(scenes.ceiling_box(), rng)
    return _recolour(scenes.cornell(), rng)


GUIDE_SIZES = [(64, 96), (64, 64), (64, 64), (40, 64)]  # (out, in) of the guide's four layers


def _guide_params(rng):
    """Seeded weights of the guide's four layers (He-uniform, small biases)."""
    parts = []
    for n, k in GUIDE_SIZES:
        lim = math.sqrt(6.0 / k)
        parts += [rng.uniform(-lim, lim, n * k), rng.uniform(-0.1, 0.1, n)]
    return np.concatenate(parts).astype(np.float32)


def _train_batch(case, seed):
    rng = np.random.default_rng(seed)
    n = case["rows"]
    params = _guide_params(rng)
    feats = rng.uniform(-1.0, 1.0, (n, 96)).astype(np.float32)
    dirs = rng.normal(size=(n, 3))
    dirs = (dirs / np.linalg.norm(dirs, axis=1, keepdims=True)).astype(np.float32)
    weights = rng.lognormal(0.0, 1.0, n).astype(np.float32)
    return params, feats, dirs, weights


def _load_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = case["grid"]
    spec = scenes.large(grid=g, instances=24, emitters=64, texture_size=64, textures=8, seed=1 + seed % 1000003)
    spec.environment = scenes.sky_hdri(case["env_width"], case["env_width"] // 2, sun_sigma_deg=2.0, sun_peak=800.0,
                                       sun_azimuth_deg=float(rng.uniform(0.0, 90.0)))
    n = case["rays"]
    org = np.stack([rng.uniform(-50, 50, n), np.full(n, 80.0), rng.uniform(-50, 50, n)], 1).astype(np.float32)
    d = np.stack([rng.uniform(-0.4, 0.4, n), np.full(n, -1.0), rng.uniform(-0.4, 0.4, n)], 1)
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return spec, org, d


def prepare(case, seed):
    ctx = Context(0)
    kind = case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "train":
        params, s["feats"], s["dirs"], s["weights"] = _train_batch(case, seed)
        s["guide"] = Guide(ctx, 1)
        s["guide"].set_params(params)
        return s
    if kind == "load":
        s["spec"], s["org"], s["dir"] = _load_inputs(case, seed)
        return s
    if kind == "serve":
        rng = np.random.default_rng(seed)
        s["scenes"] = [(Scene(ctx, _spec("box", seed)), 8), (Scene(ctx, _spec("chart", seed)), 12)]
        s["jobs"] = []
        for k in range(case["jobs"]):
            w = max(16, int(case["side"] / (1, 2, 3, 4)[k % 4]))
            h = max(9, w * 9 // 16)
            s["jobs"].append((k % 2, w, h, int(rng.integers(1, case["most_spp"] + 1))))
        s["server"] = Server(ctx, 40 << 30, frame_spp=4)
        return s
    w, h = case["width"], case["height"]
    s["scene"] = Scene(ctx, _spec(case["scene"], seed))
    s["renderer"] = Renderer(ctx, case["bounces"], SAMPLING[case["sampling"]])
    s["sample"] = seed % 1024
    if kind == "snapshot":
        return s
    s["film"] = Film(ctx, w, h)
    if case.get("guided"):
        s["guide"] = Guide(ctx, 1)
        s["guide"].set_params(_guide_params(np.random.default_rng(seed)))
        s["renderer"].set_guide(s["guide"], 0.5, 0)
    if kind == "viewport":
        s["frame"] = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
    if kind == "film":
        s["image"] = torch.zeros((h, w, 4), dtype=torch.float32).pin_memory()
    return s


# ---- one pass -------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        loss, grads = s["guide"].train_step(s["feats"], s["dirs"], s["weights"], 0.0, grads=True)
        return {"loss": loss, "grads": grads}
    if kind == "load":
        scene = Scene(s["ctx"], s["spec"])
        hits, t = scene.probe_intersect(s["org"], s["dir"])
        scene.close()
        return {"hits": hits, "t": t}
    if kind == "serve":
        server = s["server"]
        ids = [server.submit(*s["scenes"][k][:1], w, h, spp, s["scenes"][k][1]) for k, w, h, spp in s["jobs"]]
        out = []
        for j in ids:
            server.wait(j)
            out.append(server.result(j))
            server.release(j)
        return out
    if kind == "snapshot":
        return s["renderer"].render(s["scene"], case["width"], case["height"], s["sample"])
    film = s["film"]
    film.reset()
    s["renderer"].accumulate(s["scene"], film, case["spp"])
    if kind == "viewport":
        film.tonemap_device(0.0, s["frame"].data_ptr())
        return s["frame"]
    if kind == "aov":
        return film.all_averages()
    film.averages_into(s["image"].data_ptr())
    return s["image"]


# ---- what a pass cannot do without -------------------------------------------------

# Per scene, from instrumented frames: rays per camera path (closest-hit and
# shadow), wide nodes and triangles per ray, surface vertices per path. A ray
# reads its origin and direction and writes its hit (48 B) and reads 80 B per
# node and 36 B per triangle; a surface vertex reads its state, three vertices,
# its material and textures and writes the next ray (584 B).
SCENE_COST = {
    "box": (8.0, 5.5, 3.0, 4.0, 7.0), "ceiling": (8.0, 5.5, 3.0, 4.0, 7.0), "chart": (2.2, 0.9, 5.5, 4.6, 1.2),
    "terrain": (2.3, 0.63, 17.3, 6.5, 1.46), "textured": (2.5, 1.2, 3.0, 4.0, 1.5),
}


def _path_work(scene, paths):
    rays, shadows, nodes, tris, vertices = SCENE_COST[scene]
    n = rays + shadows
    return dict(bytes=paths * (n * (52 + 80 * nodes + 36 * tris) + 584 * vertices),
                flops=paths * (n * (nodes * 8 * 15 + tris * 50) + 1500 * vertices))


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["rows"]
        return dict(bytes=n * (96 + 3 + 1) * 4 + 17128 * 4 * 2, flops=n * 3 * 2 * sum(a * b for a, b in GUIDE_SIZES))
    if kind == "load":
        tris = 2 * (case["grid"] - 1) ** 2 + 24 * 2000
        texels = case["env_width"] ** 2 // 2
        return dict(bytes=tris * (16 + 12 + 48 + 20) + texels * 24, flops=tris * 400 + texels * 40)
    if kind == "serve":
        total = dict(bytes=0.0, flops=0.0)
        for k in range(case["jobs"]):
            w = max(16, int(case["side"] / (1, 2, 3, 4)[k % 4]))
            one = _path_work(("box", "chart")[k % 2], w * max(9, w * 9 // 16) * (case["most_spp"] + 1) / 2)
            total = {q: total[q] + one[q] for q in total}
        return total
    px = case["width"] * case["height"]
    out = _path_work(case["scene"], px * case["spp"])
    out["bytes"] += px * {"snapshot": 16, "viewport": 4, "film": 16, "aov": 52}[kind]
    if case.get("guided"):
        vertices = SCENE_COST[case["scene"]][4] * px * case["spp"]
        out["bytes"] += vertices * 400
        out["flops"] += vertices * 2 * sum(a * b for a, b in GUIDE_SIZES)
    return out


# ---- 64-bit answers ----------------------------------------------------------------


def _exact_train(case, seed):
    """Loss and gradient of the guide in float64: four dense layers, ReLU
    between them, and the KL estimator -sum(w log q)/n of an 8-lobe von
    Mises-Fisher mixture whose lobe takes 5 outputs (axis, concentration,
    weight)."""
    params, feats, dirs, weights = _train_batch(case, seed)
    dev = "cuda"
    layers, o = [], 0
    for n, k in GUIDE_SIZES:
        w = torch.tensor(params[o:o + n * k], dtype=torch.float64, device=dev).reshape(n, k).requires_grad_()
        o += n * k
        b = torch.tensor(params[o:o + n], dtype=torch.float64, device=dev).requires_grad_()
        o += n
        layers.append((w, b))
    a = torch.tensor(feats, dtype=torch.float64, device=dev)
    for i, (w, b) in enumerate(layers):
        a = a @ w.T + b
        if i < 3:
            a = torch.relu(a)
    lobes = a.reshape(-1, 8, 5)
    axis = lobes[..., :3]
    mu = axis / torch.sqrt((axis ** 2).sum(-1, keepdim=True) + 1e-12)
    kappa = 0.01 + torch.log1p(torch.exp(torch.clamp(lobes[..., 3], -20, 20)))
    share = torch.softmax(lobes[..., 4], -1)
    d = torch.tensor(dirs, dtype=torch.float64, device=dev)
    cosine = (mu * d[:, None, :]).sum(-1)
    q = (share * kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa))) * torch.exp(kappa * (cosine - 1))).sum(-1)
    loss = -(torch.tensor(weights, dtype=torch.float64, device=dev) * torch.log(torch.clamp(q, min=1e-20))).mean()
    loss.backward()
    grads = torch.cat([torch.cat([w.grad.reshape(-1), b.grad]) for w, b in layers])
    return {"loss": float(loss.detach()), "grads": grads.cpu().numpy()}


def _exact_load(case, seed):
    """The rays' nearest distances in float64, every ray against every triangle."""
    spec, org, d = _load_inputs(case, seed)
    dev = "cuda"
    corners = []
    for o in spec.objects:
        m = np.asarray(o.transform, np.float64).reshape(3, 4)
        p = o.mesh.positions.astype(np.float64) @ m[:, :3].T + m[:, 3]
        corners.append(p[o.mesh.indices.astype(np.int64)])
    v = torch.tensor(np.concatenate(corners), device=dev)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = []
    step = max(1, int(4e6) // len(v))
    for k in range(0, len(org), step):
        ro = torch.tensor(org[k:k + step], dtype=torch.float64, device=dev)[:, None]
        rd = torch.tensor(d[k:k + step], dtype=torch.float64, device=dev)[:, None]
        p = torch.linalg.cross(rd.expand(-1, len(v), -1), e2[None].expand(len(ro), -1, -1))
        det = (e1[None] * p).sum(-1)
        s = ro - v[None, :, 0]
        b1 = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand(len(ro), -1, -1))
        b2 = (rd * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        hit = (b1 >= -1e-9) & (b2 >= -1e-9) & (b1 + b2 <= 1 + 1e-9) & (t >= 0)
        out.append(torch.where(hit, t, torch.full_like(t, math.inf)).amin(1))
    return {"hits": None, "t": torch.cat(out).cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "load" and case["grid"] <= 300:
        return _exact_load(case, seed)
    return None  # a Monte Carlo render follows its own paths' rounding: see the module's docstring
