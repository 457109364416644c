"""Workloads for timing libaqua, each through the calls a renderer makes.

Six kinds of call, over the sizes they are used at:

  trace   aqua_trace on a caller's ray set (host arrays, or device buffers),
          closest hits or occlusion
  render  aqua_render of a scene with the path integrator (host or device film)
  frame   one aqua_render_nrc frame with online training
  batch   aqua_render_batch over jobs of several scenes
  infer   aqua_nrc_encode + aqua_nrc_forward on a frame's cache queries
  train   one aqua_nrc_train_step and the gradients it used

Scenes: the procedural ones of aqua_make_procedural_scene (Cornell boxes,
the 1.15M-triangle interior, the 4.0M-triangle sphere field) and the
Cornell scene files under tests/golden/cbox with every Principled lobe set
somewhere. A process keeps one context and loads a large scene once, as a
renderer does; rays, random-number seeds, features, targets and weights
come from the case's seed.
"""
from __future__ import annotations

import json
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "aqua-engine_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import aqua  # noqa: E402

CORNELL, CORNELL_GGX, INTERIOR, SPHERES = "cornell", "cornell_ggx", "interior", "spheres"
PRINCIPLED = "principled"
CONFIG = {CORNELL: 1, CORNELL_GGX: 2, INTERIOR: 3, SPHERES: 5}

# Per ray (closest hit, then occlusion): four-wide node visits and triangle
# tests of the canonical walk, from aqua_trace's counters; rays per camera
# path at depth 8. They size work() only.
WALK = {CORNELL: (2.9, 4.0), CORNELL_GGX: (2.9, 4.0), PRINCIPLED: (2.9, 4.0), INTERIOR: (20.0, 5.0), SPHERES: (15.0, 4.0)}
RAYS = {CORNELL: 5.0, CORNELL_GGX: 4.7, PRINCIPLED: 6.0, INTERIOR: 6.0, SPHERES: 3.0}
SCENE_BYTES = {CORNELL: 1 << 13, CORNELL_GGX: 1 << 13, PRINCIPLED: 1 << 13, INTERIOR: 220_000_000, SPHERES: 300_000_000}
NODE_FLOPS = 4 * 26.0   # four slab tests
TRI_FLOPS = 60.0        # one watertight triangle test
SHADE_FLOPS = 250.0     # one vertex: light sample, BSDF sample, two evaluations

NRC_DIMS = 5 * 64 * 64 + 3 * 64


# ---------------------------------------------------------------- cases
def listed():
    return [
        # A picking or visibility query of an editor: a few thousand rays from host arrays.
        {"name": "trace-pick", "kind": "trace", "scene": CORNELL_GGX, "rays": 4097, "any": False, "device": False},
        # A baker's closest-hit batch on device buffers, as many rays as a 1080p frame has pixels.
        {"name": "trace-interior", "kind": "trace", "scene": INTERIOR, "rays": 2_073_600, "any": False, "device": True},
        # Ambient-occlusion style visibility against millions of triangles, a ragged count.
        {"name": "occlusion-spheres", "kind": "trace", "scene": SPHERES, "rays": 1_000_003, "any": True,
         "device": True},
        # A material thumbnail with the integrator's default settings (4 spp, depth 5).
        {"name": "thumbnail", "kind": "render", "scene": CORNELL_GGX, "width": 64, "height": 64, "spp": 4, "depth": 5,
         "device": False},
        # The Lambertian Cornell box at the CPU configuration's size.
        {"name": "cornell-256", "kind": "render", "scene": CORNELL, "width": 256, "height": 256, "spp": 64,
         "depth": 5, "device": False},
        # The headline scene at a quarter of its samples.
        {"name": "cornell-ggx-1024", "kind": "render", "scene": CORNELL_GGX, "width": 1024, "height": 1024,
         "spp": 256, "depth": 8, "device": True},
        # A progressive pass over the textured interior at 1080p.
        {"name": "interior-1080p", "kind": "render", "scene": INTERIOR, "width": 1920, "height": 1080, "spp": 8,
         "depth": 8, "device": True},
        # A preview of loaded scene files: smooth normals, a point light, glass and clearcoat; odd sizes.
        {"name": "principled-preview", "kind": "render", "scene": PRINCIPLED, "width": 701, "height": 523, "spp": 9,
         "depth": 8, "device": False},
        # One 1080p frame of the cached renderer, 1 spp, 65,536 training records in batches of 16,384.
        {"name": "cached-frame", "kind": "frame", "scene": INTERIOR, "width": 1920, "height": 1080, "spp": 1,
         "depth": 8, "records": 65536, "batch": 16384},
        # Serving: uneven views of four scenes in one launch.
        {"name": "batch-serving", "kind": "batch", "jobs": 20, "side": 512, "spp": 48, "depth": 8, "plan": 5},
        # The cache queries of about one 1080p frame, features to radiance.
        {"name": "infer-2m", "kind": "infer", "rows": 2_000_003},
        # One large optimisation step of the cache, a ragged row count.
        {"name": "train-250k", "kind": "train", "rows": 250_007},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "render", "render", "render", "frame", "batch", "infer", "train"])
    if kind == "trace":
        return {"kind": kind, "scene": rng.choice([CORNELL, CORNELL_GGX, INTERIOR, SPHERES, PRINCIPLED]),
                "rays": _log(rng, 1000, 2_000_000), "any": rng.random() < 0.5, "device": rng.random() < 0.6}
    if kind == "render":
        scene = rng.choice([CORNELL, CORNELL_GGX, CORNELL_GGX, INTERIOR, SPHERES, PRINCIPLED])
        w, h = _log(rng, 48, 1400), _log(rng, 48, 1000)
        most = (60e6 if scene in (INTERIOR, SPHERES, PRINCIPLED) else 250e6) / 4 / (w * h)
        return {"kind": kind, "scene": scene, "width": w, "height": h, "spp": _log(rng, 1, max(1.0, min(256.0, most))),
                "depth": rng.randint(2, 10), "device": rng.random() < 0.5}
    if kind == "frame":
        return {"kind": kind, "scene": rng.choice([INTERIOR, INTERIOR, CORNELL_GGX]), "width": _log(rng, 320, 1920),
                "height": _log(rng, 180, 1080), "spp": 1, "depth": rng.randint(4, 10),
                "records": _log(rng, 8192, 65536), "batch": _log(rng, 2048, 16384)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 24), "side": _log(rng, 96, 512), "spp": _log(rng, 4, 48),
                "depth": rng.randint(3, 8), "plan": rng.randint(0, 1 << 20)}
    if kind == "infer":
        return {"kind": kind, "rows": _log(rng, 1000, 2_000_000)}
    return {"kind": kind, "rows": _log(rng, 512, 250_000)}


# ---------------------------------------------------------------- what a program keeps
_ctx = None
_big = {}


def _context():
    global _ctx
    if _ctx is None:
        torch.cuda.init()
        _ctx = aqua.Context(device=0)
    return _ctx


# Materials of the loaded Cornell scene: glass, clearcoat, sheen and tints beside the plain walls.
EDITS = {
    "tallBox": dict(transmission=1.0, ior=1.5, roughness=0.15, metallic=0.0, color=[0.9, 0.95, 1.0]),
    "shortBox": dict(clearcoat=1.0, clearcoat_roughness=0.1, sheen=0.5, sheen_tint=0.5, roughness=0.5, specular=0.5,
                     color=[0.7, 0.2, 0.15]),
    "backWall": dict(specular=0.6, specular_tint=1.0, roughness=0.3),
    "leftWall": dict(sheen=1.0, sheen_tint=1.0),
    "floor": dict(transmission=0.3, roughness=0.6, metallic=0.1),
}


def _principled(ctx):
    base = os.path.join(ROOT, "tests", "golden", "cbox")
    with open(os.path.join(base, "cbox.json")) as f:
        d = json.load(f)
    for name, values in EDITS.items():
        p = d["named_bsdfs"][name]["Principled"]
        for key, v in values.items():
            p[key] = {"Float3": v} if key == "color" else {"Float": v}
    for shape in d["shapes"]:
        shape["Mesh"][0] = os.path.join(base, shape["Mesh"][0])
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "cbox_principled.json")
        with open(path, "w") as f:
            json.dump(d, f)
        return ctx.load_scene(path)


class _Owned:
    """A scene or a network that goes when the state that holds it goes."""

    def __init__(self, it):
        self.it = it

    def __del__(self):
        try:
            self.it.free()
        except Exception:
            pass


def _scene(name, seed):
    """(scene, its owner): the large scenes are loaded once, a Cornell box per state."""
    ctx = _context()
    if name in (INTERIOR, SPHERES):
        if name not in _big:
            _big[name] = ctx.procedural(CONFIG[name], seed=0)
        return _big[name], None
    s = _principled(ctx) if name == PRINCIPLED else ctx.procedural(CONFIG[name], seed=seed)
    return s, _Owned(s)


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFF)


# ---------------------------------------------------------------- inputs
BOUNDS = {CORNELL: ((-0.6, -0.1, -0.6), (0.6, 1.1, 1.1)), CORNELL_GGX: ((-0.6, -0.1, -0.6), (0.6, 1.1, 1.1)),
          PRINCIPLED: ((-1.1, -0.1, -1.1), (1.1, 2.1, 2.0)), INTERIOR: ((-9.9, 0.05, -6.9), (9.9, 3.95, 6.9)),
          SPHERES: ((-40.0, 0.05, -40.0), (40.0, 8.0, 40.0))}


def _rays(case, scene, seed):
    """Half camera rays through jittered pixels, half rays between surfaces (origins in the scene's box, any
    direction); occlusion rays are all of the second kind and end somewhere on the way."""
    n, g = case["rays"], _gen(seed, 1)
    rays = torch.zeros((n, 8), device="cuda")
    lo, hi = (torch.tensor(b, device="cuda") for b in BOUNDS[case["scene"]])
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    d = torch.randn((n, 3), device="cuda", generator=g)
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    size = float((hi - lo).norm())
    if case["any"]:
        rays[:, 7] = size * (0.02 + 0.98 * torch.rand(n, device="cuda", generator=g))
        return rays
    rays[:, 7] = math.inf
    k = n // 2
    if k:
        c = scene.camera()
        w = max(1, int(math.sqrt(k * 16 / 9)))
        i = torch.arange(k, device="cuda")
        u = torch.rand((k, 2), device="cuda", generator=g)
        th = math.tan(0.5 * math.radians(c.fov_deg))
        h = (k + w - 1) // w
        sx = (2 * ((i % w) + u[:, 0]) / w - 1) * th * (w / h)
        sy = (1 - 2 * ((i // w) + u[:, 1]) / h) * th
        R, U, B = (torch.tensor(list(v), device="cuda") for v in (c.right, c.up, c.back))
        d = sx[:, None] * R + sy[:, None] * U - B
        rays[:k, 0:3] = torch.tensor(list(c.pos), device="cuda")
        rays[:k, 4:7] = d / d.norm(dim=1, keepdim=True)
    return rays


def _features(n, seed):
    """Raw cache features as path vertices have them: points in the unit box, unit directions and normals,
    roughness, albedo, specular F0."""
    g = _gen(seed, 2)
    raw = torch.rand((n, 16), device="cuda", generator=g)
    for a in (3, 6):
        v = torch.randn((n, 3), device="cuda", generator=g)
        raw[:, a:a + 3] = v / v.norm(dim=1, keepdim=True)
    raw[:, 13:16] *= 0.5
    return raw


def _weights(seed):
    """He-uniform weights, W1..W5 (64 x 64) then W6 (3 x 64)."""
    r = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    lim = np.full(NRC_DIMS, math.sqrt(6 / 64), np.float32)
    lim[5 * 4096:] = math.sqrt(3 / 64)
    return (r.uniform(-1, 1, NRC_DIMS).astype(np.float32) * lim).astype(np.float32)


def _encode64(raw):
    """The cache's input encoding in 64 bits (positions in the unit box)."""
    r = raw.double()

    def sph(v):
        u = torch.acos(v[:, 2].clamp(-1, 1)) / math.pi
        w = (torch.atan2(v[:, 1], v[:, 0]) + math.pi) / (2 * math.pi)
        return u.clamp(0, 1), w.clamp(0, 1)

    def blob(x, k):
        return [torch.exp(-0.5 * ((x - (b + 0.5) / k) * k) ** 2) for b in range(k)]

    cols = []
    p = r[:, 0:3].clamp(0, 1)
    for a in range(3):
        for f in range(8):
            cols += [torch.sin(math.pi * p[:, a] * 2 ** f), torch.cos(math.pi * p[:, a] * 2 ** f)]
    du, dv = sph(r[:, 3:6])
    nu, nv = sph(r[:, 6:9])
    cols += blob(du, 3) + blob(dv, 3) + blob(nu, 2) + blob(nv, 2)
    cols += [r[:, 9].clamp(0, 1), r[:, 10], r[:, 11], r[:, 12]]
    cols += [0.2126 * r[:, 13] + 0.7152 * r[:, 14] + 0.0722 * r[:, 15], torch.ones_like(r[:, 0])]
    return torch.stack(cols, dim=1)


def _mlp64(w, x):
    """The network in 64 bits: (outputs, the weight matrices as autograd leaves)."""
    w = torch.from_numpy(w).cuda().double()
    mats = [w[4096 * k:4096 * (k + 1)].reshape(64, 64).clone().requires_grad_(True) for k in range(5)]
    mats.append(w[5 * 4096:].reshape(3, 64).clone().requires_grad_(True))
    h = x
    for m in mats[:5]:
        h = torch.relu(h @ m.t())
    return h @ mats[5].t(), mats


def _train_inputs(n, seed):
    x = _encode64(_features(n, seed)).to(torch.bfloat16).contiguous()
    t = torch.exp(torch.randn((n, 3), device="cuda", generator=_gen(seed, 3)) - 0.5).contiguous()
    return x, t


# A late fine-tuning rate: one Adam step moves every weight by at most this.
TRAIN_LR = 1e-5


def _batch_jobs(case):
    """(scene, width, height, spp, depth) per job: uneven views, mostly of the small scenes."""
    import random

    rng = random.Random(case["plan"])
    jobs = []
    for k in range(case["jobs"]):
        scene = (CORNELL, CORNELL_GGX, INTERIOR, SPHERES)[k % 4]
        w, h = _log(rng, 48, case["side"]), _log(rng, 48, case["side"])
        jobs.append((scene, w, h, _log(rng, max(1, case["spp"] // 8), case["spp"]), case["depth"]))
    return jobs


# ---------------------------------------------------------------- prepare and run
def prepare(case, seed):
    ctx, seed = _context(), int(seed)
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx}
    if kind in ("trace", "render", "frame"):
        s["scene"], s["owner"] = _scene(case["scene"], seed)
    if kind == "trace":
        s["any"] = case["any"]
        rays = _rays(case, s["scene"], seed)
        if case["device"]:
            s["rays"] = rays
            s["hits"] = torch.zeros((case["rays"], 4), device="cuda")
        else:
            s["rays"] = rays.cpu().numpy()
    elif kind == "render":
        s["size"] = (case["width"], case["height"])
        s["cfg"] = ctx.integrator(spp=case["spp"], max_depth=case["depth"], rr_depth=3, seed=seed)
        shape = (case["height"], case["width"], 3)
        s["film"] = torch.zeros(shape, device="cuda") if case["device"] else np.zeros(shape, np.float32)
    elif kind == "frame":
        s["size"] = (case["width"], case["height"])
        s["cfg"] = ctx.integrator(type=aqua.INTEGRATOR_NRC, spp=1, max_depth=case["depth"], rr_depth=3, seed=seed,
                                  nrc_train_samples=case["records"], batch_size=case["batch"],
                                  training_iters=case["records"])
        s["film"] = torch.zeros((case["height"], case["width"], 3), device="cuda")
        s["weights"] = _weights(seed)
        s["nrc"] = aqua.Nrc(ctx, learning_rate=1e-3, seed=1)
        s["net"] = _Owned(s["nrc"])
    elif kind == "batch":
        s["films"], s["jobs"], s["owners"] = [], [], {}
        for k, (name, w, h, spp, depth) in enumerate(_batch_jobs(case)):
            if name not in s["owners"]:
                s["owners"][name] = _scene(name, seed)
            film = torch.zeros((h, w, 3), device="cuda")
            s["films"].append(film)
            s["jobs"].append((s["owners"][name][0], w, h, spp, depth, seed * 64 + k, film.data_ptr()))
    else:
        w = _weights(seed)
        s["nrc"] = aqua.Nrc(ctx, learning_rate=TRAIN_LR, seed=1)
        s["net"] = _Owned(s["nrc"])
        s["nrc"].set_weights(w)
        n = case["rows"]
        if kind == "infer":
            s["raw"] = _features(n, seed)
            s["x"] = torch.zeros((n, 64), device="cuda", dtype=torch.bfloat16)
            s["out"] = torch.zeros((n, 3), device="cuda")
        else:
            s["x"], s["target"] = _train_inputs(n, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "trace":
        if isinstance(s["rays"], np.ndarray):
            t, u, v, prim, _ = ctx.trace(s["scene"], s["rays"], any_hit=s["any"])
            return {"t": t, "u": u, "v": v, "prim": prim}
        flags = aqua.TRACE_DEVICE_PTRS | (aqua.TRACE_ANY_HIT if s["any"] else 0)
        ctx._check(ctx.lib.aqua_trace(ctx.handle, s["scene"].handle, s["rays"].data_ptr(), s["rays"].shape[0],
                                      s["hits"].data_ptr(), flags, None))
        h = s["hits"]
        return {"t": h[:, 0], "u": h[:, 1], "v": h[:, 2], "prim": h.view(torch.int32)[:, 3]}
    if kind == "render":
        s["scene"].set_resolution(*s["size"])
        if isinstance(s["film"], np.ndarray):
            ctx.render(s["scene"], s["cfg"], out=s["film"])
        else:
            ctx.render_device(s["scene"], s["cfg"], s["film"].data_ptr())
        return s["film"]
    if kind == "frame":
        # A worker that owns no history: the shot's weights in, one frame, the trained weights out.
        s["scene"].set_resolution(*s["size"])
        s["nrc"].set_weights(s["weights"])
        ctx.render_nrc(s["scene"], s["cfg"], s["nrc"], dev_ptr=s["film"].data_ptr())
        return {"film": s["film"], "weights": s["nrc"].weights()}
    if kind == "batch":
        ctx.render_batch(s["jobs"])
        return s["films"]
    if kind == "infer":
        n = s["raw"].shape[0]
        s["nrc"].encode_device(s["raw"].data_ptr(), n, s["x"].data_ptr())
        s["nrc"].forward_device(s["x"].data_ptr(), n, s["out"].data_ptr())
        return {"x": s["x"], "out": s["out"]}
    s["nrc"].train_step_device(s["x"].data_ptr(), s["target"].data_ptr(), s["x"].shape[0])
    return {"gradients": s["nrc"].gradients(), "weights": s["nrc"].weights()}


# ---------------------------------------------------------------- work
def _path_work(scene, paths, depth):
    rays = RAYS[scene] * paths * min(1.0, 0.3 + 0.7 * depth / 8)
    nodes, tris = WALK[scene]
    return rays * (nodes * NODE_FLOPS + tris * TRI_FLOPS + 0.5 * SHADE_FLOPS)


def work(case):
    kind = case["kind"]
    if kind == "trace":
        nodes, tris = WALK[case["scene"]]
        n = case["rays"]
        touched = min(SCENE_BYTES[case["scene"]], n * (nodes * 112 + tris * 48))
        return {"bytes": 48.0 * n + touched, "flops": n * (nodes * NODE_FLOPS + tris * TRI_FLOPS)}
    if kind in ("render", "frame"):
        px = case["width"] * case["height"]
        f = _path_work(case["scene"], px * case["spp"], case["depth"])
        b = 12.0 * px + min(SCENE_BYTES[case["scene"]], 1000.0 * px * case["spp"])
        if kind == "frame":
            # queries end most paths at the second vertex; the network's rows come on top
            f = 0.5 * f + 2.0 * 20672 * px + 6.0 * 20672 * case["records"]
            b += 3 * 4.0 * NRC_DIMS * 2
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0.0
        for scene, w, h, spp, depth in _batch_jobs(case):
            f += _path_work(scene, w * h * spp, depth)
            b += 12.0 * w * h
        return {"bytes": b + SCENE_BYTES[INTERIOR], "flops": f}
    n = case["rows"]
    if kind == "infer":
        return {"bytes": (64.0 + 128.0 + 128.0 + 12.0) * n + 4.0 * NRC_DIMS, "flops": 2.0 * NRC_DIMS * n}
    return {"bytes": (128.0 + 12.0) * n + 4.0 * 7 * NRC_DIMS, "flops": 6.0 * NRC_DIMS * n}


# ---------------------------------------------------------------- exact values
def _closest64(verts, rays):
    """Distance to the nearest triangle, 64-bit Moeller-Trumbore over all of them (0 on a miss)."""
    v = torch.from_numpy(verts).cuda().double().reshape(-1, 3, 3)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    out = []
    for r in rays.double().split(1 << 14):
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        p = torch.cross(d.expand(-1, v.shape[0], -1), e2[None].expand(r.shape[0], -1, -1), dim=2)
        det = (p * e1).sum(2)
        s = o - v[None, :, 0]
        u = (s * p).sum(2) / det
        q = torch.cross(s, e1[None].expand(r.shape[0], -1, -1), dim=2)
        w = (q * d).sum(2) / det
        t = (q * e2).sum(2) / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > r[:, None, 3]) & (t < r[:, None, 7])
        t = torch.where(ok, t, torch.inf).min(1).values
        out.append(torch.where(torch.isfinite(t), t, 0.0))
    return torch.cat(out)


def exact(case, seed):
    """64-bit values where they can be had: hit distances on the small scenes, the network and its gradients. A
    path-traced image has none (in 64 bits some of its paths take other branches), nor do barycentrics and ids
    where two triangles overlap."""
    kind, seed = case["kind"], int(seed)
    if kind == "trace":
        if case["any"] or case["scene"] in (INTERIOR, SPHERES):
            return None
        scene, owner = _scene(case["scene"], seed)
        t = _closest64(scene.triangles()[0], _rays(case, scene, seed))
        return {"t": t, "u": None, "v": None, "prim": None}
    if kind == "infer":
        x = _encode64(_features(case["rows"], seed))
        with torch.no_grad():
            return {"x": x, "out": torch.cat([_mlp64(_weights(seed), c)[0] for c in x.split(1 << 18)])}
    if kind == "train":
        x, t = _train_inputs(case["rows"], seed)
        w = _weights(seed)
        grads, n = None, case["rows"]
        for xc, tc in zip(x.double().split(1 << 17), t.double().split(1 << 17)):
            y, mats = _mlp64(w, xc)
            loss = ((y - tc) ** 2 / (y.detach() ** 2 + 0.01)).sum() / (3 * n)
            g = torch.cat([m.reshape(-1) for m in torch.autograd.grad(loss, mats)])
            grads = g if grads is None else grads + g
        new = torch.from_numpy(w).cuda().double() - TRAIN_LR * grads / (grads.abs() + 1e-8)
        return {"gradients": grads, "weights": new}
    return None
