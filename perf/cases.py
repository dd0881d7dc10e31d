"""The work that programs built on this library have it do, as cases that can be timed and compared.

Every case goes through a public entry point (`native`, `native_ext`) on the scenes of `scenes.py`: single primary-ray
images, path-traced frames with and without the learned skip, the drop-in render with its PNG, batched scenes, the
brick build and its renderer, and the training, prediction and labelling of the learned distance.  A seed moves the
camera, the scene's random numbers or the points; the sizes are the case's own.

There is no `exact` value for path-traced images (a path on a fractal amplifies the last bit of a hit point into
another path, so no 64-bit render has the same noise), for trained weights (hundreds of BF16 steps) or for whole
numbers.
"""
import math
import os
import tempfile

import numpy as np
import torch

from fractalpathtracer_gb300 import ffi, native, scenes
from fractalpathtracer_gb300 import native_ext as nx


def listed():
    return [
        # one still of primary rays: the smallest call of the library, where latency counts
        {"name": "primary_320x240", "op": "primary", "scene": "bulb8", "width": 320, "height": 240},
        # the drop-in call as the reference's host makes it for a preview: built-in scene, odd size, PNG written
        {"name": "metal_cornell_161x91", "op": "metal", "sdf": 0, "width": 161, "height": 91, "spp": 4},
        # a full path-traced frame into new arrays, as the plain call returns it
        {"name": "path_bulb_1080p", "op": "path", "scene": "bulb8", "width": 1920, "height": 1080, "spp": 16, "bounces": 4,
         "surrogate": 0, "kept": False},
        # the same frame with the learned skip, in a frame loop that keeps pinned result buffers
        {"name": "path_skip_1080p", "op": "path", "scene": "bulb8", "width": 1920, "height": 1080, "spp": 16, "bounces": 4,
         "surrogate": 1, "kept": True},
        # sponge on a plane under an equirect sky: short estimators, much shading
        {"name": "path_menger_720p", "op": "path", "scene": "menger", "width": 1280, "height": 720, "spp": 16, "bounces": 4,
         "surrogate": 0, "kept": False},
        # a preview frame of the box fractal, ragged size, few samples
        {"name": "path_box_333x217", "op": "path", "scene": "box", "width": 333, "height": 217, "spp": 2, "bounces": 3,
         "surrogate": 0, "kept": False},
        # many uneven scenes at once (data generation): the largest case
        {"name": "batch_64", "op": "batch", "count": 64, "spp": 4, "bounces": 3},
        # the brick build into a caller's own device buffers
        {"name": "voxel_static_512", "op": "voxel_static", "resolution": 512},
        # a new grid and its first frame
        {"name": "voxel_build_1024", "op": "voxel_build", "resolution": 1024, "width": 1920, "height": 1080},
        # a camera moving through a kept grid
        {"name": "voxel_render_1080p", "op": "voxel_render", "resolution": 1024, "width": 1920, "height": 1080},
        # training a surrogate (uniform points only: near-surface sampling keeps other points on every run)
        {"name": "mlp_train_16384", "op": "train", "points": 1 << 20, "batch": 16384, "steps": 300},
        # labelling points with the exact estimator and its gradients
        {"name": "sample_1m", "op": "sample", "scene": "bulb", "points": 1 << 20, "gradients": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["primary", "metal", "path", "path", "batch", "voxel_static", "voxel_build", "voxel_render", "train", "sample"])
    w = _log(rng, 48, 1920)
    h = max(32, min(1080, int(w * rng.uniform(0.5, 1.0))))
    if op == "primary":
        return {"op": op, "scene": rng.choice(["bulb8", "bulb", "box", "menger", "hybrid"]), "width": w, "height": h}
    if op == "metal":
        w = _log(rng, 48, 640)
        return {"op": op, "sdf": rng.choice([0, 8]), "width": w, "height": max(32, int(w * rng.uniform(0.5, 1.0))),
                "spp": rng.randint(1, 8)}
    if op == "path":
        surrogate = rng.choice([0, 0, 1, 2])
        scene = rng.choice(["bulb8", "box"] if surrogate else ["bulb8", "bulb", "box", "menger", "hybrid"])
        return {"op": op, "scene": scene, "width": w, "height": h, "spp": rng.randint(1, 16), "bounces": rng.randint(1, 5),
                "surrogate": surrogate, "kept": rng.random() < 0.5}
    if op == "batch":
        return {"op": op, "count": rng.randint(2, 40), "spp": rng.randint(1, 4), "bounces": rng.randint(1, 3)}
    if op == "voxel_static":
        return {"op": op, "resolution": _log(rng, 33, 512)}
    if op in ("voxel_build", "voxel_render"):
        return {"op": op, "resolution": _log(rng, 65, 1024), "width": w, "height": h}
    if op == "train":
        return {"op": op, "points": _log(rng, 1024, 1 << 20), "batch": _log(rng, 64, 32768), "steps": rng.randint(20, 300)}
    return {"op": op, "scene": rng.choice(["bulb8", "bulb", "box", "menger", "hybrid"]), "points": _log(rng, 33, 1 << 20),
            "gradients": rng.random() < 0.5}


# ------------------------------------------------------------------ scenes
_EYES = {"bulb8": 3.0, "bulb": 3.0, "box": 7.0, "hybrid": 3.5}


def _eye(dist, rng):
    az, el = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.05, 0.4)
    return (dist * math.cos(el) * math.sin(az), dist * math.sin(el), -dist * math.cos(el) * math.cos(az))


def _bundle(scene, width, height, spp, bounces, seed):
    """A path-tracing scene whose camera stands somewhere else for another seed."""
    rng = np.random.default_rng(seed)
    if scene == "menger":
        b = scenes.menger_plane(width, height, spp, seed=1)
        b.ext.seed = seed & 0x7fffffff
        scenes.look_at(b.cfg, (2.6 * rng.uniform(0.9, 1.1), 1.5 * rng.uniform(0.8, 1.3), -3.4 * rng.uniform(0.9, 1.1)), (0.0, -0.15, 0.0))
        b.cfg.render[0] = float(bounces)
        return b
    if scene == "box":
        b = scenes.mandelbox_path(width, height, spp, bounces)
    else:
        b = scenes.mandelbulb_path(width, height, spp, bounces)
        if scene == "bulb":
            b.ext.power = 7.3
        elif scene == "hybrid":
            for name, value in (("formula", ffi.FORMULA_BULB_MENGER_HYBRID), ("iterations", 9), ("menger_scale", 3.0),
                                ("hybrid_period", 3), ("bailout", 4.0)):
                setattr(b.ext, name, value)
            b.cfg.set_values[1], b.cfg.set_values[2] = 9.0, 4.0
    b.ext.seed = seed & 0x7fffffff
    scenes.look_at(b.cfg, _eye(_EYES[scene], rng), (0.0, 0.0, 0.0))
    return b


def _primary(case, seed):
    b = _bundle(case["scene"], case["width"], case["height"], 1, 1, seed)
    if case["scene"] != "menger":
        b.cfg.render[4] = 10.0 if case["scene"] != "box" else 12.0
    return b


def _voxel_scene(case, seed):
    rng = np.random.default_rng(seed)
    cfg, ext = scenes.voxel_mandelbox(case["resolution"], case.get("width", 64), case.get("height", 64))
    ext.box_scale = -1.5 - 0.02 * rng.random()
    scenes.look_at(cfg, (5.5 * rng.uniform(0.9, 1.1), 4.0 * rng.uniform(0.9, 1.1), -9.0 * rng.uniform(0.9, 1.1)), (0.0, 0.0, 0.0))
    return cfg, ext


def _points(case, seed):
    rng = np.random.default_rng(seed)
    reach = {"box": 2.5, "menger": 1.6}.get(case["scene"], 1.3)
    pts = np.zeros((case["points"], 4), np.float32)
    pts[:, :3] = rng.uniform(-reach, reach, (case["points"], 3))
    return pts


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    op = case["op"]
    s = {"op": op}
    if op == "primary":
        s["bundle"] = _primary(case, seed)
    elif op == "metal":
        cfg = ffi.default_config()
        cfg.sdf_id = case["sdf"]
        cfg.width, cfg.height, cfg.samples = case["width"], case["height"], case["spp"]
        rng = np.random.default_rng(seed)
        cfg.camera_position[:] = [float(rng.uniform(-0.2, 0.2)), float(rng.uniform(-0.2, 0.2)), -5.0]
        s["cfg"], s["path"] = cfg, os.path.join(tempfile.gettempdir(), "perf_case_%d.png" % os.getpid())
    elif op == "path":
        b = _bundle(case["scene"], case["width"], case["height"], case["spp"], case["bounces"], seed)
        if case["surrogate"]:
            # the model that such a program trained before; uniform points, so that one seed gives one model
            lo, hi = scenes.SURROGATE_BOXES["mandelbox" if case["scene"] == "box" else "mandelbulb"]
            model, _ = nx.mlp_create(b.cfg, b.ext, nx.mlp_config(lo, hi, points=1 << 18, near_fraction=0.0, batch=8192, steps=400,
                                                                 seed=1 + seed % 1000))
            b.ext.surrogate, b.ext.surrogate_model = case["surrogate"], model
        s["bundle"] = b
        n = case["width"] * case["height"] * 4
        s["linear"] = s["rgba"] = None
        if case["kept"]:
            s["linear"] = torch.zeros(n, dtype=torch.float32).pin_memory().numpy()
            s["rgba"] = torch.zeros(n, dtype=torch.uint8).pin_memory().numpy()
    elif op == "batch":
        s["bundles"] = scenes.batch_scenes(case["count"], case["spp"], case["bounces"])
        for k, b in enumerate(s["bundles"]):
            b.ext.seed = (seed * 97 + k) & 0x7fffffff
    elif op == "voxel_static":
        s["scene"] = _voxel_scene(case, seed)
        bricks = ((case["resolution"] + 7) // 8) ** 3
        cells = bricks * 512
        s["table"] = torch.zeros(bricks, dtype=torch.int32, device="cuda")
        s["occ"] = torch.zeros(cells, dtype=torch.uint8, device="cuda")
        s["dist"] = torch.zeros(cells, dtype=torch.int16, device="cuda")
    elif op == "voxel_build":
        s["scene"] = _voxel_scene(case, seed)
    elif op == "voxel_render":
        cfg, ext = _voxel_scene(case, seed)
        ext.box_scale = -1.5   # one grid, kept by the library; the camera moves
        nx.voxel_build(cfg, ext)
        s["scene"] = (cfg, ext)
    elif op == "train":
        cfg, ext = scenes.mandelbulb_primary()
        lo, hi = scenes.SURROGATE_BOXES["mandelbulb"]
        s["scene"] = (cfg, ext)
        s["mc"] = nx.mlp_config(lo, hi, points=case["points"], near_fraction=0.0, batch=case["batch"], steps=case["steps"],
                                seed=1 + seed % 100000)
    else:
        s["bundle"] = _bundle(case["scene"], 64, 64, 1, 1, seed)
        s["points"], s["gradients"] = _points(case, seed), case["gradients"]
    return s


def _fields(records):
    return {name: records[name] for name in records.dtype.names}


def run(state):
    op = state["op"]
    if op == "primary":
        hits, _ = native.trace_primary(state["bundle"].cfg, state["bundle"].ext)
        return _fields(hits)
    if op == "metal":
        return {"linear": native.metal_render(state["cfg"], state["path"])["linear"]}
    if op == "path":
        b = state["bundle"]
        linear, rgba, _ = native.cuda_render(b.cfg, b.ext, out_linear=state["linear"], out_rgba=state["rgba"])
        return {"linear": linear, "rgba": rgba}
    if op == "batch":
        return nx.render_batch(state["bundles"])[0]
    if op == "voxel_static":
        cfg, ext = state["scene"]
        info = nx.voxel_build_static(cfg, ext, state["table"].data_ptr(), state["table"].numel(), state["occ"].data_ptr(),
                                     state["dist"].data_ptr(), state["occ"].numel())
        n = info["active_bricks"] * 512
        return {"table": state["table"], "occupancy": state["occ"][:n], "distance": state["dist"][:n], "cells": info["active_cells"]}
    if op in ("voxel_build", "voxel_render"):
        cfg, ext = state["scene"]
        out = {}
        if op == "voxel_build":
            info = nx.voxel_build(cfg, ext)
            out["bricks"], out["cells"] = info["active_bricks"], info["active_cells"]
        hits, rgba, _ = nx.voxel_render(cfg, ext)
        return {**out, **_fields(hits), "rgba": rgba}
    if op == "train":
        cfg, ext = state["scene"]
        model, stats = nx.mlp_create(cfg, ext, state["mc"])
        params = nx.mlp_get_params(model)
        nx.mlp_destroy(model)
        return {"params": params, "loss": float(stats["loss_last"])}
    b = state["bundle"]
    got = native.sample_distance(b.cfg, b.ext, state["points"], gradients=state["gradients"])
    out, grads = got if state["gradients"] else (got, None)
    return {"distance": out[:, 0], "orbit": out[:, 1], "derivative": out[:, 2], "iterations": out[:, 3], "gradient": grads}


# ------------------------------------------------------------------ work
# FP32 operations of one distance evaluation: orbit iterations that an evaluation takes on average times the
# operations of the formula's step, and the finish.
_EVAL = {"bulb8": 3 * 53 + 40, "bulb": 3 * 80 + 40, "box": 8 * 30 + 20, "menger": 5 * 20 + 20, "hybrid": 4 * 45 + 40}
_ROW = 2 * (112 * 64 + 3 * 64 * 64 + 64)   # one forward pass of the distance network


def work(case):
    op = case["op"]
    pixels = case.get("width", 0) * case.get("height", 0)
    if op == "primary":
        return {"bytes": pixels * 24, "flops": pixels * 25 * _EVAL[case["scene"]]}
    if op == "metal":
        return {"bytes": pixels * 20, "flops": pixels * case["spp"] * 100 * 100}
    if op == "path":   # about 35 evaluations per path (camera ray, bounces, sun rays)
        return {"bytes": pixels * 20, "flops": pixels * case["spp"] * 35 * _EVAL[case["scene"]]}
    if op == "batch":
        paths = sum(b.cfg.width * b.cfg.height for b in scenes.batch_scenes(case["count"])) * case["spp"]
        return {"bytes": 16 * paths / case["spp"], "flops": paths * 30 * 300}
    if op == "voxel_static":
        return {"bytes": 4 * ((case["resolution"] + 7) // 8) ** 3 + 0.27 * case["resolution"] ** 3 * 3, "flops": case["resolution"] ** 3 * 100}
    if op == "voxel_build":
        return {"bytes": 4 * ((case["resolution"] + 7) // 8) ** 3 + 0.14 * case["resolution"] ** 3 * 3 + pixels * 28,
                "flops": case["resolution"] ** 3 * 100 + pixels * 95 * 10}
    if op == "voxel_render":   # about 95 visited cells a pixel at 1024^3, primary and shadow ray
        return {"bytes": pixels * 28 + 4 * ((case["resolution"] + 7) // 8) ** 3, "flops": pixels * 95 * 10 * case["resolution"] / 1024}
    if op == "train":
        return {"bytes": case["points"] * 16, "flops": 3 * _ROW * case["batch"] * case["steps"]}
    return {"bytes": case["points"] * (44 if case["gradients"] else 32),
            "flops": case["points"] * _EVAL[case["scene"]] * (4 if case["gradients"] else 1)}


# ------------------------------------------------------------------ the 64-bit values
def _field64(scene, cfg, ext, p):
    """The scene's distance at the points p (n, 3), in 64 bits, by the trigonometric and branching forms."""
    x, y, z = p[:, 0].clone(), p[:, 2].clone(), p[:, 1].clone()   # the field's axes: world x, z, y
    cx, cy, cz = x.clone(), y.clone(), z.clone()
    dr = torch.ones_like(x)
    r = torch.sqrt(x * x + y * y + z * z)
    live = torch.ones_like(x, dtype=torch.bool)
    for _ in range(ext.iterations):
        if scene == "box":
            nx_, ny_, nz_ = (torch.where(v.abs() > ext.box_fold_limit, torch.sign(v) * ext.box_fold_value - v, v) for v in (x, y, z))
            r2 = nx_ * nx_ + ny_ * ny_ + nz_ * nz_
            lo, hi = ext.box_min_radius ** 2, ext.box_fixed_radius ** 2
            f = torch.where(r2 < lo, torch.full_like(r2, hi / lo), torch.where(r2 < hi, hi / r2, torch.ones_like(r2)))
            nx_, ny_, nz_ = (v * f * ext.box_scale for v in (nx_, ny_, nz_))
            ndr = dr * f * abs(ext.box_scale) + 1.0
        else:
            p_ = float(ext.power)
            th, ph = torch.asin((z / r).clamp(-1.0, 1.0)) * p_, torch.atan2(y, x) * p_
            rp = r ** (p_ - 1.0)
            ndr = rp * dr * p_ + 1.0
            rp = rp * r
            nx_, ny_, nz_ = torch.cos(th) * torch.cos(ph) * rp, torch.cos(th) * torch.sin(ph) * rp, torch.sin(th) * rp
        x, y, z = (torch.where(live, n + c, o) for n, c, o in ((nx_, cx, x), (ny_, cy, y), (nz_, cz, z)))
        dr = torch.where(live, ndr, dr)
        r = torch.sqrt(x * x + y * y + z * z)
        live = live & (r <= ext.bailout)
        if not bool(live.any()):
            break
    if scene == "box":
        return r / dr
    return torch.where(r > 1.0, 0.5 * r * torch.log(r) / dr, torch.zeros_like(r))


def _primary64(case, seed):
    """Hit distances of the pixels' rays: the plain march and its refinement in 64 bits."""
    b = _primary(case, seed)
    cfg, ext = b.cfg, b.ext
    w, h = cfg.width, cfg.height
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    u = torch.arange(w, device=dev, dtype=torch.float64) / w - 0.5   # the field scenes' rays go through pixel corners
    v = (torch.arange(h, device=dev, dtype=torch.float64) + 1.0) / h - 0.5
    vv, uu = torch.meshgrid(v, u * (w / h), indexing="ij")
    focal = 1.0 / math.tan(cfg.camera_fov / 2.0 * math.pi / 180.0)
    d = torch.stack([uu.reshape(-1), vv.reshape(-1), torch.full((w * h,), focal, device=dev, dtype=torch.float64)], 1)
    d = d / d.norm(dim=1, keepdim=True)
    yaw, pitch = cfg.camera_yaw_pitch[0], cfg.camera_yaw_pitch[1]
    y = d[:, 2] * math.sin(pitch) + d[:, 1] * math.cos(pitch)
    z = d[:, 2] * math.cos(pitch) - d[:, 1] * math.sin(pitch)
    d = torch.stack([d[:, 0] * math.cos(yaw) + z * math.sin(yaw), y, -d[:, 0] * math.sin(yaw) + z * math.cos(yaw)], 1)
    cam = torch.tensor([float(c) for c in cfg.camera_position], device=dev, dtype=torch.float64)
    vs = cfg.vset_values
    t = torch.zeros(w * h, device=dev, dtype=torch.float64)
    step = torch.zeros_like(t)
    found = torch.zeros_like(t, dtype=torch.bool)
    at = torch.arange(w * h, device=dev)

    def field(idx, tt):
        dist = _field64(case["scene"], cfg, ext, cam + d[idx] * tt[:, None])
        return dist, (tt * vs[116]).clamp(vs[118], vs[119])

    for _ in range(int(cfg.render[1])):
        if not at.numel():
            break
        tt = t[at]
        dist, th = field(at, tt)
        near = dist < th
        found[at[near]] = True
        at, tt, dist, th = at[~near], tt[~near], dist[~near], th[~near]
        s = ((dist - 0.5 * th).clamp_min(0.0) * vs[113]).clamp_max(vs[110])
        step[at] = s
        t[at] = tt + s
        at = at[t[at] < cfg.render[4]]
    limit = 1.0 - 0.001 * max(vs[129], 0.0)
    at = torch.nonzero(found).reshape(-1)
    step = step * 0.5
    for _ in range(30):
        if not at.numel():
            break
        dist, th = field(at, t[at])
        out, ins = dist > th, dist < th * limit
        move = out | ins
        at, out = at[move], out[move]
        t[at] = t[at] + torch.where(out, step[at], -step[at])
        step[at] = step[at] * 0.5
    return t.reshape(h, w)


def exact(case, seed):
    if case["op"] == "primary" and case["scene"] in ("bulb8", "bulb", "box"):
        return {"distance": _primary64(case, seed), "normal": None, "steps": None, "hit": None}
    if case["op"] == "sample" and case["scene"] in ("bulb8", "bulb", "box"):
        b = _bundle(case["scene"], 64, 64, 1, 1, seed)
        p = torch.from_numpy(_points(case, seed)[:, :3].astype(np.float64))
        p = p.cuda() if torch.cuda.is_available() else p
        return {"distance": _field64(case["scene"], b.cfg, b.ext, p), "orbit": None, "derivative": None, "iterations": None, "gradient": None}
    return None
