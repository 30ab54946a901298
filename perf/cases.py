"""The framework's work as a user's program calls it: sized cases over its public entry points.

listed() are fixed cases, draw() gives others of the same ranges, prepare() makes what a
program holds before the call (scene handles, parameters, host buffers), run() is one pass
through the entry point and work() what such a pass cannot do without.

Every case has a "kind", which names the entry point:

  render    luz_gpu_render (film "host": a pinned host film) or luz_gpu_render_device
            (film "device": a device tensor on the caller's stream)
  batch     luz_gpu_batch_render over several scenes
  denoised  luz_gpu_render_denoised: adaptive sampling, NFOR buffers and the NFOR image
  nfor      luz_gpu_nfor_denoise on host buffers
  adjoint   one step of a texture fit: luz_gpu_adjoint_forward, then luz_gpu_adjoint_backward
  emission  luz_gpu_adjoint_emission
  cache     luz_gpu_cache_gradient and luz_gpu_cache_predict on host rows
  rays      luz_gpu_trace_rays, closest hits and occlusion of the same rays
"""
import math

import numpy as np
import torch

from luz_b200 import desc, native, scenes

TEXTURE = 32      # side of the fitted albedo texture
CACHE_LAYERS = ((128, 64), (64, 64), (64, 64), (64, 64), (64, 16))


def listed():
    return [
        # An interactive preview of a small mixed scene: one sample per pixel, every object
        # kind and most materials; the time is launches and latency.
        dict(name="preview_mixed", kind="render", film="device", scene="mixed", size=0, width=96, height=64, spp=1,
             bounces=6),
        # The Cornell box as the benchmark renders it (instanced boxes, one area light).
        dict(name="cornell_300", kind="render", film="host", scene="cornell", size=0, width=300, height=300, spp=50,
             bounces=8),
        # The headline frame: 1.31 M triangles, glass and metal, environment light, 1080p.
        dict(name="glossy_1080p", kind="render", film="host", scene="glossy", size=8, width=1920, height=1080, spp=64,
             bounces=12),
        # A draft frame of a medium mesh at few samples, the way a scene is set up.
        dict(name="glossy_draft", kind="render", film="host", scene="glossy", size=6, width=640, height=360, spp=4,
             bounces=12),
        # 1e5 instances in a scattering medium, 720p: the two-level traversal.
        dict(name="instances_720p", kind="render", film="host", scene="instances", size=100_000, width=1280,
             height=720, spp=8, bounces=16),
        # Odd sizes over analytic primitives only: spheres of every glossy kind under a sky.
        dict(name="spheres_odd", kind="render", film="host", scene="spheres", size=40, width=517, height=389, spp=7,
             bounces=12),
        # Many small independent scenes in one call (dataset rendering, thumbnails).
        dict(name="batch_small", kind="batch", count=12, side_lo=64, side_hi=256, spp_lo=1, spp_hi=16),
        # A finished still: adaptive sampling, then the denoiser on the device buffers.
        dict(name="denoised_cornell", kind="denoised", scene="cornell", size=0, width=300, height=300, spp=128,
             bounces=8, min_samples=32, interval=32),
        # The denoiser alone on another renderer's buffers, half of 1080p each way.
        dict(name="nfor_540p", kind="nfor", width=960, height=540),
        # One step of an albedo-texture fit in the textured Cornell box: forward and backward.
        dict(name="adjoint_256", kind="adjoint", width=256, height=256, spp=64, bounces=8),
        # The radiance cache's network on its own: one training batch's gradient and a frame
        # row block's predictions.
        dict(name="cache_16k", kind="cache", rows=16384, queries=65536),
        # Ray queries against a mesh (visibility, picking, baking), an odd count.
        dict(name="rays_300k", kind="rays", size=6, rays=300_007),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["batch", "denoised", "nfor", "adjoint", "emission", "cache", "rays"])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 16), side_lo=_log(rng, 32, 96), side_hi=_log(rng, 128, 320),
                    spp_lo=1, spp_hi=_log(rng, 4, 24))
    if kind == "nfor":
        return dict(kind=kind, width=_log(rng, 64, 960), height=_log(rng, 64, 540))
    if kind == "cache":
        return dict(kind=kind, rows=_log(rng, 100, 16384), queries=_log(rng, 100, 200_000))
    if kind == "rays":
        return dict(kind=kind, size=rng.randint(3, 6), rays=_log(rng, 1000, 600_000))
    w, h = _log(rng, 48, 640), _log(rng, 48, 480)
    if kind in ("adjoint", "emission"):
        return dict(kind=kind, width=min(w, 400), height=min(h, 400), spp=_log(rng, 4, 64), bounces=rng.randint(3, 10))
    scene = rng.choice(["mixed", "cornell", "glossy", "glossy", "instances", "spheres", "ies", "atmosphere", "caustics"])
    size = {"glossy": rng.randint(3, 7), "instances": _log(rng, 500, 100_000), "spheres": _log(rng, 10, 120),
            "caustics": _log(rng, 4000, 60_000)}.get(scene, 0)
    if kind == "denoised":
        return dict(kind=kind, scene=scene, size=size, width=w, height=h, spp=_log(rng, 24, 128),
                    bounces=rng.randint(3, 10), min_samples=_log(rng, 8, 32), interval=_log(rng, 8, 32))
    heavy = scene in ("instances", "atmosphere")
    return dict(kind=kind, film=rng.choice(["host", "device"]), scene=scene, size=size, width=w, height=h,
                spp=_log(rng, 1, 8 if heavy else 64), bounces=rng.randint(2, 16))


def _workload(case, seed):
    """The scene of a case: its geometry, colours or lights follow the seed."""
    w, h, spp, b = case["width"], case["height"], case["spp"], case["bounces"]
    rng = np.random.default_rng(seed)
    kind, size = case["scene"], case["size"]
    if kind == "glossy":
        wl = scenes.mesh_glossy(w, h, spp, b, level=size, seed=seed % 100_000)
    elif kind == "instances":
        wl = scenes.instancing_volumes(w, h, spp, b, count=size, seed=seed % 100_000)
    elif kind == "spheres":
        wl = scenes.spheres_linear_sky(w, h, spp, b, count=size, seed=seed % 100_000)
    elif kind == "caustics":
        wl = scenes.caustic_pool(w, h, spp, b, photons=size)
    else:
        wl = {"mixed": scenes.tiny_mixed, "cornell": scenes.cornell, "ies": scenes.ies_room,
              "atmosphere": scenes.atmosphere_hills}[kind](w, h, spp, b)
    if kind in ("mixed", "cornell", "ies", "caustics"):   # the same room lit a little differently
        gain = float(rng.uniform(0.8, 1.25))
        for m in wl.scene.materials:
            if m["type"] == desc.MAT_EMISSIVE:
                m["color"] = tuple(gain * float(c) for c in m["color"])
    wl.seed = int(rng.integers(1, 1 << 31))
    return wl


def _params(wl):
    return native.params(wl.width, wl.height, wl.spp, wl.max_bounces, wl.seed)


def _cache_rows(case, seed):
    """Cache weights, training rows and queries: positions in the unit box, unit directions
    and normals, roughness; the targets a smooth radiance field with a bright side."""
    rng = np.random.default_rng(seed)
    w = np.concatenate([(rng.uniform(-1.0, 1.0, k * n) * math.sqrt(6.0 / k)) for k, n in CACHE_LAYERS])

    def rows(n):
        d = rng.normal(size=(n, 6))
        d[:, :3] /= np.linalg.norm(d[:, :3], axis=1, keepdims=True)
        d[:, 3:] /= np.linalg.norm(d[:, 3:], axis=1, keepdims=True)
        return np.concatenate([rng.random((n, 3)), d, rng.random((n, 1))], 1).astype(np.float32)

    x = rows(case["rows"])
    t = np.stack([0.5 + np.sin(3.0 * x[:, 0] + c) * x[:, 4] + 2.0 * (x[:, 1] > 0.8) for c in range(3)], 1)
    return w.astype(np.float32), x, np.maximum(t, 0.0).astype(np.float32), rows(case["queries"])


def _nfor_buffers(case, seed):
    """Two noisy halves of an image with edges and a few bright outliers, its eleven features
    (coordinates, hit mask, depth, normal, albedo, material) and their variances."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    y, x = np.meshgrid(np.linspace(0.0, 1.0, h), np.linspace(0.0, 1.0, w), indexing="ij")
    cells = (np.floor(x * 9 + 0.3 * np.sin(7 * y)) + np.floor(y * 6)).astype(int) % 7
    albedo = rng.uniform(0.1, 0.9, (7, 3))[cells]
    shade = 0.6 + 0.4 * np.sin(5.0 * x + rng.uniform(0, 6)) * np.cos(4.0 * y)
    base = albedo * shade[..., None]
    sigma = 0.05 + 0.25 * rng.random((7,))[cells]
    feats = np.concatenate([x[..., None], y[..., None], np.ones((h, w, 1)), (0.3 + 0.5 * y * shade)[..., None],
                            np.stack([0.5 + 0.5 * np.sin(6 * x), 0.5 + 0.5 * np.cos(5 * y), shade], -1),
                            albedo, (cells[..., None] % 3) / 6.0], -1)
    noise = np.array([0, 0, 0, 1, 1, 1, 1, 1, 1, 1, 0]) * 0.02

    def half():
        c = np.maximum(base + rng.normal(size=(h, w, 3)) * sigma[..., None] * base, 0.0)
        c[rng.random((h, w)) < 0.002] *= 12.0
        return np.ascontiguousarray(c), np.ascontiguousarray(feats + rng.normal(size=feats.shape) * noise)

    ca, fa = half()
    cb, fb = half()
    return {"color_a": ca, "color_b": cb, "color_variance": np.mean((ca - cb) ** 2, -1) * 0.25 + 1e-4,
            "features_a": fa, "features_b": fb,
            "feature_variance": np.broadcast_to(noise * noise * 0.5, feats.shape).copy()}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "render":
        wl = _workload(case, seed)
        s["scene"], s["params"] = native.GpuScene(wl.scene.build()), _params(wl)
        if case["film"] == "host":
            s["film"] = torch.empty((wl.height, wl.width, 3), dtype=torch.float32, pin_memory=True).numpy()
        else:
            s["image"] = torch.zeros((wl.height, wl.width, 3), dtype=torch.float32, device="cuda")
    elif kind == "batch":
        s["scenes"], s["params"] = [], []
        for i, (level, side, spp, depth) in enumerate(_batch_plan(case)):   # the sizes stay, what is in the scenes changes
            wl = scenes.mesh_glossy(side, side, spp, depth, level=level, seed=(seed + i) % 100_000)
            s["scenes"].append(native.GpuScene(wl.scene.build()))
            s["params"].append(native.params(side, side, spp, depth, (seed + i) & 0x7FFFFFFF))
    elif kind == "denoised":
        wl = _workload(case, seed)
        s["scene"], s["params"] = native.GpuScene(wl.scene.build()), _params(wl)
        s["adaptive"] = native.adaptive(case["min_samples"], case["interval"])
    elif kind == "nfor":
        s["buffers"] = _nfor_buffers(case, seed)
    elif kind in ("adjoint", "emission"):
        wl = scenes.cornell_textured(case["width"], case["height"], case["spp"], case["bounces"], seed=seed)
        s["scene"], s["params"] = native.GpuScene(wl.scene.build()), _params(wl)
        s["params"].seed = 1 + seed % (1 << 30)
        s["texels"] = np.array(wl.scene.textures[0])
        s["goal"] = np.random.default_rng(seed + 1).uniform(0.0, 0.6, (wl.height, wl.width, 3)).astype(np.float32)
    elif kind == "cache":
        w, s["inputs"], s["targets"], s["queries"] = _cache_rows(case, seed)
        s["cache"] = native.RadianceCache(desc.cache_params(seed=1))
        s["cache"].set_weights(w)
    elif kind == "rays":
        wl = scenes.mesh_glossy(64, 64, 1, 1, level=case["size"], seed=seed % 100_000)
        s["scene"] = native.GpuScene(wl.scene.build())
        rng = np.random.default_rng(seed)
        n = case["rays"]
        o = rng.normal(size=(n, 3))
        o *= 3.0 / np.linalg.norm(o, axis=1, keepdims=True)
        o[:, 1] = np.abs(o[:, 1])
        d = rng.normal(size=(n, 3)) * 0.6 - o
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        s["rays"] = np.concatenate([o, np.full((n, 1), 1e-3), d, np.full((n, 1), 100.0)], 1).astype(np.float32)
    return s


def _batch_plan(case):
    """Mesh level, image side, samples and depth of each scene of a batch: log-uniform sides
    and samples, 1e3 to 3e5 triangles."""
    rng = np.random.default_rng(case["count"])
    return [(int(rng.integers(3, 8)),
             int(math.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"])))),
             int(math.exp(rng.uniform(math.log(case["spp_lo"]), math.log(case["spp_hi"] + 0.999)))),
             int(rng.integers(4, 17))) for _ in range(case["count"])]


def run(s):
    kind = s["kind"]
    if kind == "render":
        if "film" in s:
            return s["scene"].render(s["params"], s["film"])[0]
        s["scene"].render_device(s["params"], s["image"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["image"]
    if kind == "batch":
        return native.batch_render(s["scenes"], s["params"])[0]
    if kind == "denoised":
        film, image, used, _ = s["scene"].render_denoised(s["params"], s["adaptive"])
        return film, image, used
    if kind == "nfor":
        return native.nfor_denoise(s["buffers"])
    if kind == "adjoint":
        film, _ = s["scene"].adjoint_forward(s["params"], 0, s["texels"])
        adj = (2.0 / film.size) * (film - s["goal"])
        grad, _ = s["scene"].adjoint_backward(s["params"], 0, adj, s["texels"].shape)
        return film, grad
    if kind == "emission":
        return s["scene"].adjoint_emission(s["params"], s["goal"])[0]
    if kind == "cache":
        grad, loss = s["cache"].gradient(s["inputs"], s["targets"])
        return grad, loss, s["cache"].predict(s["queries"])
    hits = s["scene"].trace_rays(s["rays"])
    shadow = s["scene"].trace_rays(s["rays"], any_hit=True)
    return {**{k: np.ascontiguousarray(hits[k]) for k in hits.dtype.names if hits.dtype[k].kind in "fiu"},
            "occluded": np.ascontiguousarray(shadow[shadow.dtype.names[1]])}


# Rays (extension and shadow) a sample of each scene takes on the way, measured once, and the
# primitives its hierarchy is over.
RAYS = {"mixed": 3.8, "cornell": 5.1, "glossy": 2.7, "instances": 6.6, "spheres": 2.3, "ies": 4.2, "atmosphere": 2.0,
        "caustics": 4.7}
PRIMITIVES = {"mixed": 40, "cornell": 30, "ies": 10, "atmosphere": 5, "caustics": 700}


def _render_work(scene, size, width, height, spp):
    """Scene read once and film written once; per ray a balanced binary descent (two boxes of
    24 operations a level) with four triangle tests of 40, and 400 operations of shading."""
    n = 20 * 4 ** size if scene == "glossy" else max(size, PRIMITIVES.get(scene, 0))
    per_prim = 160 if scene == "instances" else 90
    env = 16 * 1024 * 512 if scene == "glossy" else 0
    flops = width * height * spp * RAYS[scene] * (48.0 * math.log2(n + 1) + 560.0)
    return {"bytes": float(n * per_prim + env + 12 * width * height), "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("render", "denoised"):
        w = _render_work(case["scene"], case["size"], case["width"], case["height"], case["spp"])
        if kind == "denoised":   # the minimum number of samples, the buffers read once, the image written
            px = case["width"] * case["height"]
            w["flops"] = w["flops"] * case["min_samples"] / case["spp"] + px * 30_000.0
            w["bytes"] += px * 40.0
        return w
    if kind == "batch":
        ws = [_render_work("glossy", level, side, side, spp) for level, side, spp, _ in _batch_plan(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "nfor":   # 43 doubles a pixel in and out; five 12 x 12 systems over 25 neighbours, filters
        px = case["width"] * case["height"]
        return {"bytes": px * 43 * 8.0, "flops": px * 5 * (25 * 12 * 15 * 1.5 + 12 * 12 * 15 * 2.0)}
    if kind in ("adjoint", "emission"):
        w = _render_work("cornell", 0, case["width"], case["height"], case["spp"])
        n = 3.0 if kind == "adjoint" else 1.0   # the image, the paths' values and their replay
        return {"bytes": w["bytes"] * 2 + TEXTURE * TEXTURE * 48, "flops": w["flops"] * n}
    if kind == "cache":
        mac = float(sum(k * n for k, n in CACHE_LAYERS))
        return {"bytes": case["rows"] * 52.0 + case["queries"] * 52.0 + 8 * mac,
                "flops": 2 * mac * (3 * case["rows"] + case["queries"])}
    n = 20 * 4 ** case["size"]
    return {"bytes": n * 90.0 + case["rays"] * 2 * 52.0, "flops": 2 * case["rays"] * (48.0 * math.log2(n) + 160.0)}


def _cache_exact(case, seed):
    """The network, its relative loss and the gradient in 64 bits."""
    w, x, t, q = (torch.from_numpy(a) for a in _cache_rows(case, seed))
    layers, at = [], 0
    for k, n in CACHE_LAYERS:
        layers.append(w[at:at + k * n].double().reshape(k, n).requires_grad_())
        at += k * n

    def forward(v):
        a = v.double()[:, :, None] * (2.0 ** torch.arange(6, dtype=torch.float64)) * math.pi
        e = torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(v.shape[0], 120)
        h = torch.cat([e, torch.ones(v.shape[0], 1, dtype=torch.float64),
                       torch.zeros(v.shape[0], 7, dtype=torch.float64)], 1)
        for layer in layers[:-1]:
            h = torch.relu(h @ layer)
        return (h @ layers[-1])[:, :3]

    y = forward(x)
    loss = ((y - t.double()) ** 2 / (y.detach() ** 2 + 0.01)).sum() / x.shape[0]
    grad = torch.cat([g.reshape(-1) for g in torch.autograd.grad(loss, layers)])
    with torch.no_grad():
        p = forward(q)
    return grad.numpy(), float(loss.detach()), p.numpy()


def exact(case, seed):
    # A film is a sum over paths whose every bounce is decided by 32-bit values, hits follow the
    # same, and the denoiser's and the gradients' outputs are 64-bit sums already: only the
    # network has a value of its own in 64 bits.
    return _cache_exact(case, seed) if case["kind"] == "cache" else None
