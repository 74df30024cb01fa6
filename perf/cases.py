"""The work a user of this framework has it do, as measurable cases.

Seven families, each through the framework's public entry points:

  render   the reference's whole compute pass of one image: camera ray, closest
           hit, colour, into a device image (Context.render_frame)
  frame    primary closest hits and shadow any-hits of one image
           (Context.trace_frame)
  trace    stored rays against one BVH (Context.trace): plain, ordered by the
           coherence key or by the learned predictor, closest or any hit
  build    the BVH of a triangle buffer, rebuilt into its handle, and its node
           array in the reference's layout (Bvh.rebuild, Bvh.nodes)
  refit    a moved scene: Bvh.refit, then one image's hits
  batch    many scenes of uneven size, built and traced by one captured graph
           (Batch.run)
  learn    one training step's forward and backward pass of the hit predictor
           and its inference (crt_predictor_gradients, Predictor.infer)

Sizes come from the repository's own workloads (65,536-triangle soup at
512x512; 1,310,720-triangle displaced sphere at 1920x1080; 4,194,304-triangle
clustered soup with 8,388,608 bounce rays; 16,777,216-triangle soup; 64 uneven
scenes) and from small and odd sizes of the same ranges.
"""
import ctypes
import math

import numpy as np
import torch

from realtimeraytracing_gb300 import crt
from realtimeraytracing_gb300 import scenes as S

DEV = "cuda:0"
WT = crt.TRI_WATERTIGHT
ORDERS = {"plain": 0, "sorted": crt.SORT_RAYS, "learned": crt.PREDICTOR_ORDER}


def listed():
    return [
        # A preview image of a small model: the smallest call, all launch and host latency.
        {"name": "render_preview", "family": "render", "scene": "soup", "tris": 2003, "width": 160, "height": 120,
         "wire": True},
        # The reference's own scene limit and window: 65,536 triangles, 512x512, the shader's predicate.
        {"name": "render_65k", "family": "render", "scene": "soup", "tris": 65536, "width": 512, "height": 512,
         "wire": False},
        # A full-HD frame of a million-triangle mesh with shadow rays: coherent primary and secondary rays.
        {"name": "frame_hd", "family": "frame", "scene": "sphere", "tris": 1310720, "width": 1920, "height": 1080},
        # Path-tracing secondary rays: 8M incoherent bounce rays over 4M triangles, in the caller's order ...
        {"name": "bounce_plain", "family": "trace", "scene": "clustered", "tris": 4194304, "rays": 8388608,
         "order": "plain", "any": False, "watertight": True},
        # ... ordered by the learned hit predictor, the framework's headline mode ...
        {"name": "bounce_learned", "family": "trace", "scene": "clustered", "tris": 4194304, "rays": 8388608,
         "order": "learned", "any": False, "watertight": True},
        # ... and a smaller odd batch over a smaller scene, ordered by the coherence key.
        {"name": "bounce_sorted", "family": "trace", "scene": "soup", "tris": 300007, "rays": 1500001,
         "order": "sorted", "any": False, "watertight": True},
        # The BVH the reference builds when it loads a scene: a part of its zero-padded 65,536-entry buffer.
        {"name": "build_padded", "family": "build", "scene": "soup", "tris": 20011, "buffer": 65536},
        # A million-triangle mesh rebuilt each frame.
        {"name": "build_1m", "family": "build", "scene": "sphere", "tris": 1310720, "buffer": 1310720},
        # The largest build of the repository's workloads.
        {"name": "build_16m", "family": "build", "scene": "soup", "tris": 16777216, "buffer": 16777216},
        # A moving clustered scene, refit instead of rebuilt, then a frame's primary hits.
        {"name": "refit_frame", "family": "refit", "scene": "clustered", "tris": 2000003, "width": 1280, "height": 720},
        # Many uneven scenes at once, build and trace replayed from one graph.
        {"name": "batch_64", "family": "batch", "scenes": 64, "tri_lo": 1000, "tri_hi": 250000, "ray_lo": 16384,
         "ray_hi": 524288},
        # The predictor's online training: forward, backward and inference on one frame's sampled rays.
        {"name": "learn_step", "family": "learn", "scene": "clustered", "tris": 100003, "rays": 262145},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n | rng.randint(0, 1)))


def draw(rng):
    family = rng.choice(["render", "frame", "trace", "trace", "trace", "build", "build", "refit", "batch", "learn"])
    scene = rng.choice(["soup", "clustered"])
    if family == "render":
        return {"family": family, "scene": scene, "tris": _log_int(rng, 2000, 200000),
                "width": _log_int(rng, 160, 1280), "height": _log_int(rng, 120, 720), "wire": rng.random() < 0.5}
    if family == "frame":
        return {"family": family, "scene": rng.choice(["sphere", "soup", "clustered"]),
                "tris": rng.choice([20 * 4 ** rng.randint(4, 8), _log_int(rng, 5000, 1310720)]),
                "width": _log_int(rng, 320, 1920), "height": _log_int(rng, 200, 1080)}
    if family == "trace":
        any_hit = rng.random() < 0.25
        return {"family": family, "scene": scene, "tris": _log_int(rng, 2000, 4194304),
                "rays": _log_int(rng, 1000, 8388608),
                "order": rng.choice(["plain", "sorted"] if any_hit else ["plain", "sorted", "learned"]),
                "any": any_hit, "watertight": rng.random() < 0.75}
    if family == "build":
        n = _log_int(rng, 1000, 16777216)
        return {"family": family, "scene": scene, "tris": n, "buffer": max(n, 65536) if rng.random() < 0.3 else n}
    if family == "refit":
        return {"family": family, "scene": scene, "tris": _log_int(rng, 5000, 4194304),
                "width": _log_int(rng, 320, 1920), "height": _log_int(rng, 200, 1080)}
    if family == "batch":
        return {"family": family, "scenes": rng.randint(2, 64), "tri_lo": 1000, "tri_hi": _log_int(rng, 5000, 250000),
                "ray_lo": 4096, "ray_hi": _log_int(rng, 16384, 524288)}
    return {"family": family, "scene": scene, "tris": _log_int(rng, 2000, 200000),
            "rays": _log_int(rng, 4096, 1000000)}


def _batch_sizes(case):
    """Triangle and ray counts of a batch's scenes: log-uniform, in an order of their own each."""
    r = np.random.RandomState(case["scenes"])
    u = (np.arange(case["scenes"]) + 0.5) / case["scenes"]
    sizes = [lo * (hi / lo) ** r.permutation(u) for lo, hi in ((case["tri_lo"], case["tri_hi"]),
                                                               (case["ray_lo"], case["ray_hi"]))]
    return [s.astype(np.int64) for s in sizes]


# ------------------------------------------------------------------- inputs
def _generator(seed, stream=0):
    gen = torch.Generator(device=DEV)
    gen.manual_seed((int(seed) * 1000003 + stream * 7919 + 17) & 0x7FFFFFFFFFFFFFFF)
    return gen


def _sphere(n, gen):
    """A displaced icosphere of n = 20 * 4^level triangles (the next lower such n otherwise): radius 1, shared
    vertices moved radially by up to 0.05 of three octaves of smooth noise."""
    level = 0
    while 20 * 4 ** (level + 1) <= n:
        level += 1
    verts, faces = S.icosphere(0)
    tri = torch.from_numpy(verts)[torch.from_numpy(faces.astype(np.int64))].to(DEV)  # (20, 3, 3) float64
    for _ in range(level):
        a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
        ab, bc, ca = a + b, b + c, c + a
        ab, bc, ca = (m / m.norm(dim=1, keepdim=True) for m in (ab, bc, ca))
        tri = torch.stack([torch.stack(t, 1) for t in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))], 1)
        tri = tri.reshape(-1, 3, 3)
    h = torch.zeros(tri.shape[:2], dtype=torch.float64, device=DEV)
    for freq, weight in ((4.0, 1.0), (9.0, 0.5), (19.0, 0.25)):
        waves = torch.randn((3, 3), generator=gen, device=DEV, dtype=torch.float64) * freq
        phase = torch.rand(3, generator=gen, device=DEV, dtype=torch.float64) * (2 * math.pi)
        for k in range(3):
            h += weight / 3 * torch.sin((tri * waves[k]).sum(-1) + phase[k])
    tri = tri * (1.0 + 0.05 / 1.75 * h)[..., None]
    out = torch.zeros((tri.shape[0], 16), dtype=torch.float32, device=DEV)
    for k in range(3):
        out[:, 4 * k:4 * k + 3] = tri[:, k].float()
        out[:, 4 * k + 3] = 1.0
    return out


def _triangles(scene, n, seed, buffer=0):
    gen = _generator(seed, 1)
    if scene == "sphere":
        tris = _sphere(n, gen)
    elif scene == "clustered":
        tris = S.device_soup(n, gen, clustered=True, clusters=max(8, min(256, n // 4096)), sigma=0.02, edge_mu=0.003,
                             edge_sigma=0.6)
    else:
        tris = S.device_soup(n, gen)
    if buffer > tris.shape[0]:  # the reference's padded buffer: zero records after the scene's
        tris = torch.cat([tris, torch.zeros((buffer - tris.shape[0], 16), dtype=torch.float32, device=DEV)])
    return tris


def _camera(scene, width, height, seed):
    """Looking along +z at the scene, a little off its axis, 45 degrees."""
    r = np.random.RandomState(seed & 0x7FFFFFFF).uniform(-0.05, 0.05, 2)
    eye = (r[0], r[1], -3.0) if scene == "sphere" else (0.5 + r[0], 0.5 + r[1], -1.5)
    return S.camera_gpu_data(eye, aspect=width / height)


def _models(seed, count=1):
    models = S.models_with_materials(np.arange(count))
    colors = np.random.RandomState(seed & 0x7FFFFFFF).uniform(0.1, 1.0, (count, 4))
    return models, S.materials(colors)


def _hits(h):
    return {"tri": h.view(torch.int32)[:, 0], "tuv": h[:, 1:]}


def _learn_inputs(case, seed):
    """Flat parameters, rays from inside the scene and their target classes (a coarse origin cell, or miss)."""
    tris = _triangles(case["scene"], case["tris"], seed)
    gen = _generator(seed, 3)
    n = case["rays"]
    at = torch.randint(0, tris.shape[0], (n,), generator=gen, device=DEV)
    rays = torch.zeros((n, 8), dtype=torch.float32, device=DEV)
    rays[:, 0:3] = tris[at, 0:3]
    d = torch.randn((n, 3), generator=gen, device=DEV)
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 3], rays[:, 7] = 1e-4, float("inf")
    c = (rays[:, 0:3].clamp(0, 0.999) * 5).long()
    target = (c[:, 0] * 5 + c[:, 1]) * 5 + c[:, 2]
    target[torch.rand(n, generator=gen, device=DEV) < 0.3] = 127
    shapes = ((64 * 32, 32 ** -0.5), (64, 0.05), (64 * 64, 0.125), (64, 0.05), (128 * 64, 0.125), (128, 0.05),
              (64 ** 3 * 16, 0.3), (1024 * 16, 0.3))
    params = torch.cat([torch.randn(k, generator=gen, device=DEV) * s for k, s in shapes])
    return tris, rays, target, params


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    family = case["family"]
    ctx = crt.Context()
    state = {"family": family, "ctx": ctx}
    if family == "batch":
        nt, nr = _batch_sizes(case)
        gen = _generator(seed, 2)
        state["tris"] = torch.cat([S.device_soup(int(n), gen, clustered=bool(k % 2)) for k, n in enumerate(nt)])
        state["rays"] = S.device_sphere_rays(int(nr.sum()), gen)
        state["hits"] = torch.empty((int(nr.sum()), 4), dtype=torch.float32, device=DEV)
        state["batch"] = crt.Batch(ctx, nt, nr)
        return state
    if family == "learn":
        tris, rays, target, params = _learn_inputs(case, seed)
        bvh = ctx.build(tris)
        pred = crt.Predictor(ctx, bvh)
        pred.set_params(params.cpu().numpy())
        state.update(bvh=bvh, pred=pred, rays=rays, target=target.to(torch.int16),
                     grad=torch.empty(crt.PREDICTOR_PARAMS, dtype=torch.float32, device=DEV),
                     classes=torch.empty(case["rays"], dtype=torch.int16, device=DEV))
        return state
    tris = _triangles(case["scene"], case["tris"], seed, case.get("buffer", 0))
    n = case["tris"] if "buffer" in case else int(tris.shape[0])
    n = min(n, int(tris.shape[0]))
    models, materials = _models(seed)
    bvh = ctx.build(tris, n_tris=n, models=models)
    state.update(bvh=bvh, tris=tris, n=n, models=models)
    if family == "build":
        state["nodes"] = torch.empty((2 * n - 1, 12), dtype=torch.float32, device=DEV)
    elif family == "trace":
        # bounce rays leave the closest hits of a square image's primary rays
        side = max(64, min(2048, int(math.isqrt(case["rays"]))))
        cam = _camera(case["scene"], side, side, seed)
        prim = torch.empty((side * side, 8), dtype=torch.float32, device=DEV)
        ctx.raygen(cam, side, side, out=prim)
        ph = ctx.trace(bvh, prim, WT, out=torch.empty((side * side, 4), dtype=torch.float32, device=DEV))
        rays = ctx.bounce_rays(bvh, prim, ph, case["rays"], seed=seed & 0xFFFF,
                               out=torch.empty((case["rays"], 8), dtype=torch.float32, device=DEV))
        state["rays"] = rays
        state["hits"] = torch.empty((case["rays"], 4), dtype=torch.float32, device=DEV)
        state["any"] = case["any"]
        state["flags"] = (ORDERS[case["order"]] | (WT if case["watertight"] else 0) |
                          (crt.TRACE_ANY if case["any"] else 0))
        if case["order"] == "learned":
            state["pred"] = crt.Predictor(ctx, bvh)
            for k in range(8):  # trained on its own traces' hits, as in use
                state["pred"].train(rays, ctx.trace(bvh, rays, WT, out=state["hits"]), offset=k)
    else:
        w, h = case["width"], case["height"]
        state.update(cam=torch.from_numpy(_camera(case["scene"], w, h, seed)).to(DEV), width=w, height=h)
        if family == "render":
            state.update(materials=materials, shade=crt.SHADE_WIREFRAME if case["wire"] else 0,
                         image=torch.empty((w * h, 4), dtype=torch.float32, device=DEV))
        else:
            state["hits"] = torch.empty((w * h, 4), dtype=torch.float32, device=DEV)
        if family == "frame":
            state["light"] = np.array([2.0, 2.0, -2.0], np.float32)
            state["shadow"] = torch.empty((w * h, 4), dtype=torch.float32, device=DEV)
        if family == "refit":  # the next frame's vertices: a wave along x moves them along y
            moved = tris.clone()
            for k in (0, 4, 8):
                moved[:, k + 1] += 0.01 * torch.sin(1.0 + 7.0 * moved[:, k])
            state["moved"] = moved
    return state


# ---------------------------------------------------------------------- run
def run(s):
    ctx, family = s["ctx"], s["family"]
    if family == "render":
        return ctx.render_frame(s["bvh"], s["cam"], s["width"], s["height"], models=s["models"],
                                materials=s["materials"], shade_flags=s["shade"], out=s["image"])
    if family == "frame":
        ctx.trace_frame(s["bvh"], s["cam"], s["width"], s["height"], s["light"], WT, hits_primary=s["hits"],
                        hits_shadow=s["shadow"])
        # which occluder an any-hit names is unspecified: the answer is whether there is one
        return {**_hits(s["hits"]), "shadowed": s["shadow"].view(torch.int32)[:, 0] != -1}
    if family == "trace":
        ctx.trace(s["bvh"], s["rays"], s["flags"], out=s["hits"])
        return {"hit": s["hits"].view(torch.int32)[:, 0] != -1} if s["any"] else _hits(s["hits"])
    if family == "build":
        s["bvh"].rebuild(s["tris"], n_tris=s["n"], models=s["models"])
        return s["bvh"].nodes(out=s["nodes"]).view(torch.int32)
    if family == "refit":
        s["bvh"].refit(s["moved"], models=s["models"])
        ctx.trace_frame(s["bvh"], s["cam"], s["width"], s["height"], None, WT, hits_primary=s["hits"])
        return _hits(s["hits"])
    if family == "batch":
        s["batch"].run(s["tris"], s["rays"], s["hits"], WT, graph=True)
        return _hits(s["hits"])
    pred, n = s["pred"], s["rays"].shape[0]
    ctx._after_torch()
    loss = ctypes.c_float()
    crt._check(crt.lib().crt_predictor_gradients(ctx.handle, pred.handle, crt._ptr(s["rays"]), crt._ptr(s["target"]), n,
                                                 crt._ptr(s["grad"]), ctypes.byref(loss)))
    pred.infer(s["rays"], out=s["classes"])
    return {"grad": s["grad"], "loss": loss.value, "classes": s["classes"]}


# --------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; per ray two child boxes (24 operations each) per tree level and one
    triangle (60), per triangle one box, code and the 32 neighbour areas (17 operations each) of one PLOC pass."""
    def walk(rays, tris):
        return rays * (48.0 * math.log2(max(2, tris)) + 60.0)

    family = case["family"]
    if family == "batch":
        nt, nr = _batch_sizes(case)
        return {"bytes": float(nt.sum()) * (64 + 2 * 48) + float(nr.sum()) * 48,
                "flops": float(nt.sum()) * 600.0 + sum(walk(float(r), int(t)) for t, r in zip(nt, nr))}
    n = case["tris"]
    if case.get("scene") == "sphere":
        n = 20 * 4 ** int(math.log(n / 20, 4) + 1e-9)
    if family == "learn":
        macs = 32 * 64 + 64 * 64 + 64 * 128
        return {"bytes": case["rays"] * (32 + 2 + 2) + 2 * 4 * crt.PREDICTOR_PARAMS,
                "flops": case["rays"] * macs * 2.0 * 4}
    if family == "build":
        return {"bytes": max(n, case["buffer"]) * 64 + (2 * n - 1) * 48, "flops": n * 600.0}
    tree = n * 48 + (2 * n - 1) * 32
    if family == "trace":
        return {"bytes": tree + case["rays"] * 48, "flops": walk(case["rays"], n)}
    px = case["width"] * case["height"]
    if family == "refit":
        return {"bytes": n * 64 + 2 * tree + px * 16, "flops": n * 30.0 + walk(px, n)}
    return {"bytes": tree + px * (32 if family == "frame" else 16), "flops": walk(px, n)}


# -------------------------------------------------------------------- exact
def _exact_camera_rays(cam, width, height):
    cam = torch.from_numpy(np.asarray(cam, np.float64)).to(DEV)
    m, eye = cam[0:16].reshape(4, 4), cam[16:20]  # rows of m: the matrix's columns
    y, x = torch.meshgrid(torch.arange(height, device=DEV, dtype=torch.float64) / height,
                          torch.arange(width, device=DEV, dtype=torch.float64) / width, indexing="ij")
    v = torch.stack([(x - 0.5) * cam[20], (y - 0.5) * cam[21], torch.full_like(x, float(cam[22])),
                     torch.ones_like(x)], -1).reshape(-1, 4)
    d = v @ m - eye
    d = d / d.norm(dim=1, keepdim=True)
    return eye[:3].expand(d.shape[0], 3), d[:, :3]


def _exact_hits(tris, o, d, tmin, cull):
    """Closest hit by testing every triangle: (t, u, v, hit) with u, v the weights of p1, p2.  cull: the shader's
    predicate (front faces only, |det| of at least 1e-4, weights named the other way round)."""
    p0, p1, p2 = (tris[:, k:k + 3].double() for k in (0, 4, 8))
    e1, e2 = p1 - p0, p2 - p0
    step = max(1, (1 << 25) // max(1, tris.shape[0]))
    out = []
    for a in range(0, o.shape[0], step):
        oo, dd, tm = o[a:a + step, None], d[a:a + step, None], tmin[a:a + step, None]
        q = torch.linalg.cross(dd, e2[None], dim=-1)
        det = (e1[None] * q).sum(-1)
        s = oo - p0[None]
        u = (s * q).sum(-1) / det
        r = torch.linalg.cross(s, e1[None].expand_as(s), dim=-1)
        v = (dd * r).sum(-1) / det
        t = (e2[None] * r).sum(-1) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tm)
        if cull:
            ok &= (det.abs() >= 1e-4) & ((torch.linalg.cross(e1, e2, dim=-1)[None] * dd).sum(-1) < 0)
        best, k = torch.where(ok, t, torch.full_like(t, math.inf)).min(dim=1)
        hit = torch.isfinite(best)
        pick = lambda x: torch.where(hit, x.gather(1, k[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        uu, vv = pick(u), pick(v)
        out.append(torch.stack([torch.where(hit, best, torch.zeros_like(best)), *((vv, uu) if cull else (uu, vv)),
                                hit.double()], 1))
    return torch.cat(out)


def exact(case, seed):
    family = case["family"]
    if family == "learn":
        return _exact_learn(case, seed)
    if family not in ("render", "frame") or case["tris"] * case["width"] * case["height"] > 2e10:
        return None  # whole numbers, or every ray against every triangle would take minutes
    w, h = case["width"], case["height"]
    tris = _triangles(case["scene"], case["tris"], seed)
    o, d = _exact_camera_rays(_camera(case["scene"], w, h, seed), w, h)
    hit = _exact_hits(tris, o, d, torch.zeros(w * h, dtype=torch.float64, device=DEV), cull=family == "render")
    if family == "frame":
        return {"tri": None, "tuv": hit[:, :3], "shadowed": None}
    _, materials = _models(seed)
    image = torch.zeros((w * h, 4), dtype=torch.float64, device=DEV)
    image[:, 3] = 1.0
    image += hit[:, 3:] * torch.from_numpy(materials.astype(np.float64)).to(DEV)[0]
    if case["wire"]:
        edge = (hit[:, 3] > 0) & ((hit[:, 1] < 0.02) | (hit[:, 2] < 0.02) | (1 - hit[:, 1] - hit[:, 2] < 0.02))
        image[edge] = torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=torch.float64, device=DEV)
    return image


def _exact_learn(case, seed):
    """Summed gradients and loss of softmax cross-entropy through the 32-64-64-128 network, in 64 bits."""
    tris, rays, target, params = _learn_inputs(case, seed)
    corner = torch.cat([tris[:, k:k + 3] for k in (0, 4, 8)])
    lo, hi = corner.amin(0), corner.amax(0)
    cell = ((rays[:, 0:3] - lo) * (64.0 / (hi - lo))).floor().long().clamp(0, 63)  # bins as the network's inputs
    cell = (cell[:, 0] * 64 + cell[:, 1]) * 64 + cell[:, 2]
    d = rays[:, 4:7]
    p = d[:, :2] / d.abs().sum(1, keepdim=True)
    sign = torch.where(p >= 0, 1.0, -1.0)
    p = torch.where(d[:, 2:] < 0, (1 - p.flip(1).abs()) * sign, p)
    b = ((p + 1) * 16.0).long().clamp(0, 31)
    b = b[:, 0] * 32 + b[:, 1]
    flat = params.double().requires_grad_()
    sizes = (64 * 32, 64, 64 * 64, 64, 128 * 64, 128, 64 ** 3 * 16, 1024 * 16)
    w1, b1, w2, b2, w3, b3, eo, ed = flat.split(sizes)
    x = torch.cat([eo.reshape(-1, 16)[cell], ed.reshape(-1, 16)[b]], 1)
    x = torch.relu(x @ w1.reshape(64, 32).T + b1)
    x = torch.relu(x @ w2.reshape(64, 64).T + b2)
    loss = torch.nn.functional.cross_entropy(x @ w3.reshape(128, 64).T + b3, target, reduction="sum")
    loss.backward()
    return {"grad": flat.grad, "loss": float(loss), "classes": None}
