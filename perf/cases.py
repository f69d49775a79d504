"""The calls whose speed this repository tracks: what a program that uses the framework has it do, each
through the package's public classes.

Sizes come from bench.py's workloads (the 4M-ray terrain sets, the Cornell box at 512 x 512 x 16, the
sphere field of three material families, batches of uneven orbit views, the radiance cache's batch of
16,384 rows) and from sizes around them, odd ones included. A case names a `kind`:

  trace    DeviceBVH.intersect on device rays (closest or any hit, short or full hit records)
  host     DeviceBVH.intersect_host on page-locked host rays, the whole call with both copies
  render   Renderer.render_native of one view
  compat   Renderer.render_compat, one frame of the reference's own path tracer
  batch    Batch.render of several uneven views through a captured graph
  infer    Cache.infer, the radiance cache's network
  train    Cache.train, its online Adam steps

Host scenes and their SBVHs are built once per process and kept (a program loads its scene once); every
state uploads its own device copy and keeps its own renderer, batch or cache.
"""
import math

import numpy as np
import torch

from trenchanttracer_gb300 import (Batch, BVHCompact, Cache, DeviceBVH, Renderer, Scene, make_camera_meta,
                                   render_meta, render_params, scenes)


def listed():
    return [
        # picking or a probe grid: one small ray set, bound by launches and latency
        {"name": "pick_1k_closest", "kind": "trace", "scene": "spheres", "size": 24, "rays": "surface", "n": 1000,
         "closest": 1, "ext": 0},
        # the primary rays of a frame: coherent, closest hit
        {"name": "camera_4m_closest", "kind": "trace", "scene": "terrain", "size": 1024, "rays": "camera",
         "n": 2048 * 2048, "closest": 1, "ext": 0},
        # one diffuse bounce of a frame: incoherent, closest hit
        {"name": "bounce_4m_closest", "kind": "trace", "scene": "terrain", "size": 1024, "rays": "surface",
         "n": 2048 * 2048, "closest": 1, "ext": 0},
        # shadow rays towards a light, any hit, a ragged count
        {"name": "shadow_1m_any", "kind": "trace", "scene": "spheres", "size": 100, "rays": "shadow", "n": 1000003,
         "closest": 0, "ext": 0},
        # a bounce with full hit records (material and normal), for a caller that shades by itself
        {"name": "bounce_250k_records", "kind": "trace", "scene": "cornell", "size": 5, "rays": "surface", "n": 250000,
         "closest": 1, "ext": 1},
        # rays and hits in page-locked host memory: the call of a host renderer
        {"name": "host_2m_bounce", "kind": "host", "scene": "terrain", "size": 512, "rays": "surface",
         "n": 2097152, "closest": 1},
        # an interior lit by an area light: the Cornell box of bench.py
        {"name": "render_cornell_512", "kind": "render", "scene": "cornell", "size": 5, "w": 512, "h": 512, "spp": 16,
         "depth": 8, "ordered": 0},
        # diffuse, metal and glass objects under a sky with a sun, deep paths
        {"name": "render_spheres_960x540", "kind": "render", "scene": "spheres", "size": 400, "w": 960, "h": 540,
         "spp": 16, "depth": 16, "ordered": 1},
        # a frame of the reference's own path tracer
        {"name": "compat_cornell_640x360", "kind": "compat", "scene": "cornell", "size": 5, "w": 640, "h": 360, "spp": 4},
        # many small views in one call: turntables, dataset rendering
        {"name": "batch_12_views", "kind": "batch", "scene": "terrain", "size": 512, "views": 12, "depth": 8},
        # the radiance cache's network over a frame's queries
        {"name": "cache_infer_1m", "kind": "infer", "n": 1036800},
        # its training: the four steps that follow a frame
        {"name": "cache_train_16k", "kind": "train", "rows": 16384, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "host", "render", "render", "compat", "batch", "infer", "train"])
    scene = rng.choice(["terrain", "spheres", "cornell"])
    size = {"terrain": _log_int(rng, 48, 512), "spheres": rng.randint(8, 120), "cornell": rng.randint(2, 5)}[scene]
    if kind == "trace":
        return {"kind": kind, "scene": scene, "size": size, "rays": rng.choice(["camera", "surface", "shadow"]),
                "n": _log_int(rng, 500, 3000000), "closest": rng.randint(0, 1), "ext": rng.randint(0, 1)}
    if kind == "host":
        return {"kind": kind, "scene": scene, "size": size, "rays": rng.choice(["camera", "surface"]),
                "n": _log_int(rng, 5000, 3000000), "closest": rng.randint(0, 1)}
    if kind == "render":
        return {"kind": kind, "scene": scene, "size": size, "w": rng.randint(100, 800), "h": rng.randint(100, 600),
                "spp": rng.randint(1, 12), "depth": rng.randint(2, 12), "ordered": rng.randint(0, 1)}
    if kind == "compat":
        return {"kind": kind, "scene": "cornell", "size": size if scene == "cornell" else 4, "w": rng.randint(64, 640),
                "h": rng.randint(64, 360), "spp": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "scene": "terrain", "size": _log_int(rng, 48, 512), "views": rng.randint(2, 10),
                "depth": rng.randint(3, 8)}
    if kind == "infer":
        return {"kind": kind, "n": _log_int(rng, 200, 1000000)}
    return {"kind": kind, "rows": _log_int(rng, 1000, 16384), "steps": rng.randint(1, 4)}


# ---- scenes ------------------------------------------------------------------------------------------
_SCENES = {}


def _scene(case):
    """(Scene, BVHCompact, mesh, running sum of the triangle areas) of the case, built once per process."""
    key = (case["scene"], case["size"])
    if key not in _SCENES:
        name, size = key
        if name == "terrain":
            mesh = scenes.terrain(size, 8.0)
        elif name == "spheres":
            mesh = scenes.multi_material(size, 4)
        else:
            mesh = scenes.cornell(size)
        sc = Scene.from_mesh(mesh)
        if name != "cornell":
            sc.set_env(scenes.sky_env(1024, 512, sun_radiance=5e2, sun_diameter_deg=2.0))
        a, b, c = (mesh.vertices[mesh.vidx[:, k]].astype(np.float64) for k in range(3))
        area = np.cumsum(np.linalg.norm(np.cross(b - a, c - a), axis=1))
        _SCENES[key] = (sc, BVHCompact.build(sc, 1e-5, 1, 8), mesh, area)
    return _SCENES[key]


def _eye(case, g):
    """A camera position and what it looks at, moved a little by the seed."""
    j = g.uniform(-1.0, 1.0, 3)
    if case["scene"] == "terrain":
        return np.array([0.0, 7.2, 12.8]) + j * 0.4, np.array([0.0, 0.0, 0.8])
    if case["scene"] == "spheres":
        return np.array([0.0, 14.0, 34.0]) + j, np.array([0.0, 2.0, 0.0])
    return np.array([0.0, 0.0, 1.55]) + j * 0.02, np.array([0.0, 0.0, 0.0])


def _rays(case, seed):
    """(n, 8) float32 CUDA rays."""
    _, _, mesh, area = _scene(case)
    g = np.random.default_rng(seed)
    n = case["n"]
    if case["rays"] == "camera":
        side = int(math.isqrt(n - 1)) + 1
        eye, target = _eye(case, g)
        return torch.from_numpy(scenes.pinhole_rays(side, side, eye, target, 0.45)[:n].copy()).cuda()
    gen = torch.Generator("cuda").manual_seed(seed)
    v = torch.from_numpy(mesh.vertices).cuda()
    t = torch.from_numpy(mesh.vidx.astype(np.int64)).cuda()
    # points spread over the surface, one per ray
    a, b, c = (v[t[:, k]] for k in range(3))
    face = torch.linalg.cross(b - a, c - a)
    area = torch.from_numpy(area).cuda()
    pick = torch.searchsorted(area, torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * area[-1])
    pick = pick.clamp_(max=area.numel() - 1)
    u = torch.rand(n, 2, generator=gen, device="cuda")
    s = u[:, 0:1].sqrt()
    p = a[pick] * (1 - s) + b[pick] * (s * (1 - u[:, 1:2])) + c[pick] * (s * u[:, 1:2])
    nrm = torch.nn.functional.normalize(face[pick], dim=1)
    rays = torch.empty(n, 8, device="cuda")
    eps = 1e-3 * float(v.abs().max())
    rays[:, 0:3] = p + eps * nrm
    if case["rays"] == "shadow":
        lo, hi = v.amin(0), v.amax(0)
        light = (lo + hi) / 2
        light[1] = hi[1] + (0.5 * (hi[1] - lo[1]) if case["scene"] != "cornell" else -0.01)
        light[0] += float(g.uniform(-0.3, 0.3)) * float(hi[0] - lo[0])
        to = light - rays[:, 0:3]
        dist = torch.linalg.norm(to, dim=1, keepdim=True)
        rays[:, 3:6] = to / dist
        rays[:, 7] = dist[:, 0]
    else:  # cosine-distributed about the face normal
        d = torch.randn(n, 3, generator=gen, device="cuda")
        rays[:, 3:6] = torch.nn.functional.normalize(nrm + torch.nn.functional.normalize(d, dim=1) * 0.999, dim=1)
        rays[:, 7] = 1e20
    rays[:, 6] = eps * 0.1
    return rays.contiguous()


# ---- the radiance cache's inputs ------------------------------------------------------------------------
_LO, _HI = [-2.0, -2.0, -2.0], [2.0, 2.0, 2.0]
_LAYERS = [(64, 160), (64, 64), (64, 64), (64, 64), (64, 64), (8, 64)]  # [out][in]


def _records(n, g):
    rec = np.zeros((n, 16), np.float32)
    rec[:, 0:3] = g.uniform(-2, 2, (n, 3))
    for k in (3, 6):
        d = g.normal(size=(n, 3))
        rec[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rec[:, 9] = g.uniform(0, 1, n)
    rec[:, 10:13] = g.uniform(0, 1, (n, 3))
    rec[:, 13] = g.integers(0, 7, n) / 8.0
    return rec


def _targets(rec):
    ph = (rec[:, 0:3] + 2.0) / 4.0
    base = 0.6 + 0.5 * np.sin(2 * np.pi * ph[:, 0:1]) * np.cos(np.pi * ph[:, 2:3]) + 0.3 * rec[:, 4:5]
    return (np.exp(base) * rec[:, 10:13] + 0.05).astype(np.float32)


def _weights(g):
    ws = []
    for out, inn in _LAYERS:
        s = math.sqrt(6.0 / inn) * (0.1 if out == 8 else 1.0)
        w = g.uniform(-s, s, (out, inn))
        if out == 8:
            w[3:] = 0.0
        ws.append(w.ravel())
    return np.concatenate(ws).astype(np.float32)


def _cache_inputs(case, seed):
    g = np.random.default_rng(seed)
    n = case["n"] if case["kind"] == "infer" else case["rows"] * case["steps"]
    rec = _records(n, g)
    return rec, _targets(rec), _weights(g)


# ---- one pass --------------------------------------------------------------------------------------------
def _camera(case, g):
    eye, target = _eye(case, g)
    fx = 60.0 if case["scene"] == "spheres" else 45.0
    fy = 2.0 * math.degrees(math.atan(math.tan(math.radians(fx / 2)) * case["h"] / case["w"]))
    return make_camera_meta(case["w"], case["h"], list(eye), list(target - eye), fov=(fx, fy))


def _views(case, seed):
    """Square orbit views of uneven sizes and sample counts; the seed moves the poses alone."""
    kw = dict(scale=8.0, sizes=(128, 200, 256, 384), spps=(4, 7, 16))
    shapes = scenes.orbit_views(case["views"], seed=5, **kw)
    views = []
    for (c, spp, *_), (pose, *_) in zip(shapes, scenes.orbit_views(case["views"], seed=6 + seed, **kw)):
        cam = make_camera_meta(c.width, c.height, list(pose.position), list(pose.view), fov=tuple(pose.fov))
        views.append((cam, spp, 0, 1 + seed + len(views)))
    return views


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("infer", "train"):
        rec, target, w = _cache_inputs(case, seed)
        s["cache"] = Cache(_LO, _HI, batch=case.get("rows", 16384))
        s["cache"].set_weights(w)
        s["rec"], s["target"] = torch.from_numpy(rec).cuda(), torch.from_numpy(target).cuda()
        return s
    sc, bvh = _scene(case)[:2]
    dbvh = DeviceBVH(bvh)
    if kind in ("trace", "host"):
        s["dbvh"] = dbvh
        rays = _rays(case, seed)
        if kind == "trace":
            s["rays"] = rays
            s["hits"] = torch.empty(rays.shape[0], 6 if case["ext"] else 2, dtype=torch.int32, device="cuda")
        else:
            s["rays"] = torch.empty(rays.shape, pin_memory=True).copy_(rays)
            s["hits"] = torch.empty(rays.shape[0], 2, dtype=torch.int32).pin_memory()
            s["np"] = (s["rays"].numpy(), s["hits"].numpy())
        return s
    r = s["renderer"] = Renderer(dbvh, sc)
    g = np.random.default_rng(seed)
    if kind == "batch":
        r.set_launch(128, 8, 1 << 22, 1, 1)
        s["batch"] = Batch(r, _views(case, seed), render_params(max_depth=case["depth"], rr_depth=4))
        s["accum"] = torch.empty(s["batch"].accum_elems, device="cuda")
        return s
    s["cam"] = _camera(case, g)
    s["accum"] = torch.empty(case["w"] * case["h"] * 3, device="cuda")
    if kind == "compat":
        s["meta"] = render_meta(1 + seed % 1000, case["spp"])
    else:
        if case["ordered"]:
            r.set_launch(128, 8, 1 << 22, 1, 1)
        s["params"] = render_params(spp=case["spp"], max_depth=case["depth"], rr_depth=4, seed=1 + seed)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "trace":
        s["dbvh"].intersect(s["rays"], s["hits"], closest=bool(case["closest"]), stream=stream, ext=bool(case["ext"]))
        return s["hits"]
    if kind == "host":
        s["dbvh"].intersect_host(s["np"][0], s["np"][1], closest=bool(case["closest"]), stream=stream)
        return s["np"][1]
    if kind == "infer":
        return s["cache"].infer(s["rec"])
    if kind == "train":
        loss = s["cache"].train(s["rec"], s["target"], steps=case["steps"])
        return {"loss": loss, "weights": s["cache"].weights(0)}
    s["accum"].zero_()
    if kind == "batch":
        s["batch"].render(s["accum"], stream=stream)
    elif kind == "compat":
        s["renderer"].render_compat(s["cam"], s["meta"], s["accum"], stream=stream)
    else:
        s["renderer"].render_native(s["cam"], s["params"], s["accum"], stream=stream)
    return s["accum"]


def work(case):
    """Rays in and hits out; an image out (the scene's share that a ray set or view touches is left out: it
    depends on the view); records in, radiance or weights out. Network operations are 2 per weight and row,
    three times that for training. Traversal has no fixed number of operations."""
    kind = case["kind"]
    if kind in ("trace", "host"):
        return {"bytes": case["n"] * (32 + (24 if case.get("ext") else 8)), "flops": 0}
    if kind == "batch":
        return {"bytes": sum(12 * c.width * c.height for c, *_ in _views(case, 0)), "flops": 0}
    if kind in ("render", "compat"):
        return {"bytes": 12 * case["w"] * case["h"], "flops": 0}
    params = sum(o * i for o, i in _LAYERS)
    if kind == "infer":
        return {"bytes": case["n"] * (64 + 12) + 2 * params, "flops": 2 * params * case["n"]}
    rows = case["rows"] * case["steps"]
    return {"bytes": rows * (64 + 12) + 4 * 2 * params, "flops": 6 * params * rows}


# ---- the same in 64 bits -----------------------------------------------------------------------------------
def _encode64(rec):
    """The network's inputs: sines and cosines of position, direction and normal at doubling frequencies, and
    the raw values."""
    rec = rec.double()
    n = rec.shape[0]
    lo = torch.tensor(_LO, dtype=torch.float64, device=rec.device)
    hi = torch.tensor(_HI, dtype=torch.float64, device=rec.device)
    ph = (rec[:, 0:3] - lo) / (hi - lo)
    e = torch.zeros(n, 160, dtype=torch.float64, device=rec.device)
    for x, at, freqs in ((ph, 0, 12), ((rec[:, 3:6] + 1) / 2, 72, 6), ((rec[:, 6:9] + 1) / 2, 108, 6)):
        for i in range(3):
            for k in range(freqs):
                a = math.pi * x[:, i] * 2.0 ** k
                e[:, at + 2 * freqs * i + 2 * k], e[:, at + 2 * freqs * i + 2 * k + 1] = a.sin(), a.cos()
    e[:, 144] = rec[:, 9]
    e[:, 145:148] = rec[:, 10:13]
    e[:, 148] = 1.0
    e[:, 149:155] = rec[:, 3:9]
    e[:, 155:158] = ph
    e[:, 158] = rec[:, 13]
    return e


def _forward64(e, ws):
    for w in ws[:-1]:
        e = torch.relu(e @ w.T)
    return torch.exp(torch.clamp((e @ ws[-1].T)[:, :3], max=20.0))


def exact(case, seed):
    """The cache's network in FP64. Hit records and images are compared as they are: their values follow from
    which triangle a ray meets and from a path's random numbers, which no other program reproduces."""
    if case["kind"] not in ("infer", "train"):
        return None
    rec, target, w = (torch.from_numpy(x).cuda() for x in _cache_inputs(case, seed))
    ws, at = [], 0
    for out, inn in _LAYERS:
        ws.append(w[at:at + out * inn].double().reshape(out, inn))
        at += out * inn
    if case["kind"] == "infer":
        return torch.cat([_forward64(_encode64(c), ws) for c in rec.split(1 << 17)])
    lr, b1, b2, eps = 1e-2, 0.9, 0.99, 1e-10
    m, v = [torch.zeros_like(x) for x in ws], [torch.zeros_like(x) for x in ws]
    losses = []
    for k, (r, t) in enumerate(zip(rec.split(case["rows"]), target.double().split(case["rows"]))):
        ws = [x.detach().requires_grad_() for x in ws]
        p = _forward64(_encode64(r), ws)
        loss = ((p - t) ** 2 / (p.detach() ** 2 + 0.01)).sum() / r.shape[0]
        grads = torch.autograd.grad(loss, ws)
        losses.append(float(loss))
        for i, gr in enumerate(grads):
            m[i] = b1 * m[i] + (1 - b1) * gr
            v[i] = b2 * v[i] + (1 - b2) * gr * gr
            ws[i] = (ws[i] - lr * (m[i] / (1 - b1 ** (k + 1))) / ((v[i] / (1 - b2 ** (k + 1))).sqrt() + eps)).detach()
    return {"loss": sum(losses) / len(losses), "weights": torch.cat([x.reshape(-1) for x in ws]).cpu().numpy()}
