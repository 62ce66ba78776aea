"""Timed cases of the framework: the calls its users make, over their range.

Every case runs one pass of a public entry point on inputs made from a seed.
Sizes and settings are those of rayengine_b200.configs, the tests and the
benchmark, from a 64x48 frame (launch latency) to full frames; odd and ragged
sizes are among them.  Scenes, plans (CUDA graph, tuning), weights and output
buffers are what a frame loop keeps, so they are made in prepare().

  primary     KDScene.trace_primary: closest hits of a frame over a triangle
              soup (culling on or off)
  rays        KDScene.trace_rays: a caller's own rays, closest or any hit
  ao          KDScene.render_ao: the ambient-occlusion frame of a heightfield
  sdf         sphere_trace: the exact terrain
  sdf_frame   render_sdf_frame: the shaded terrain frame, as RGBA8
  nsdf_frame  NeuralSDF.trace: the terrain through its neural surrogate
  nsdf_eval   NeuralSDF.eval: network inference on points
  nsdf_grad   NeuralSDF.loss_grad: forward and backward of a training batch
  batch       Batch.render: uneven scenes path traced in one graph launch
  voxel       VoxelGrid.brush and .trace: one edit of a voxel terrain and the
              frame that shows it

Hit records, masks and RGBA8 words are whole 32-bit values; network outputs,
gradients, radiance and voxels are floating point.
"""
import math

import numpy as np
import torch

import rayengine_b200 as rb
from rayengine_b200 import configs

# FP32 operations of one 8-octave field evaluation (8 x 75 + 4, an FMA as one)
FIELD_OPS = 604
# multiply-adds of one network row: 128 x 64, 3 x 64 x 64, 64
ROW_MACS = 128 * 64 + 3 * 64 * 64 + 64
NET_BOX = ((-40.0, -6.0, -20.0), (40.0, 11.0, 60.0))
NET_F0 = 0.5


def listed():
    return [
        # a thumbnail or a picking region: the latency of one call
        {"name": "primary_small", "kind": "primary", "tris": 4096, "width": 64, "height": 48,
         "one_sided": False, "lanes": 1},
        # the benchmark's 65,536-triangle soup, walked as its autotuner picks
        {"name": "primary_soup", "kind": "primary", "tris": 65536, "width": 512, "height": 512,
         "one_sided": False, "lanes": 32},
        # a frame that fills the GPU
        {"name": "primary_2k", "kind": "primary", "tris": 262144, "width": 2048, "height": 2048,
         "one_sided": False, "lanes": 1},
        # visibility queries of a caller, a ragged count
        {"name": "rays_any_hit", "kind": "rays", "tris": 65536, "rays": 300007, "any_hit": True},
        # the benchmark's default: 2.1M triangles, primary + shadow + 4 AO rays
        {"name": "ao_frame", "kind": "ao", "cells": 1024, "width": 1920, "height": 1080},
        # the exact sphere tracer, full frame
        {"name": "sdf_terrain", "kind": "sdf", "width": 1920, "height": 1080},
        # the render call's shaded frame, a window whose width is no tile multiple
        {"name": "sdf_frame", "kind": "sdf_frame", "width": 1366, "height": 768, "flags": 1},
        # the neural tracer's whole frame
        {"name": "nsdf_frame", "kind": "nsdf_frame", "width": 1920, "height": 1080},
        # inference on a point cloud, a ragged count
        {"name": "nsdf_eval", "kind": "nsdf_eval", "points": 1000003},
        # the training batch of the neural terrain
        {"name": "nsdf_grad", "kind": "nsdf_grad", "points": 65536},
        # path-traced scenes of uneven size
        {"name": "batch", "kind": "batch", "scenes": 6, "tris": 100000, "width": 640,
         "height": 360},
        # editing a voxel world: dig, then show it with the smooth lookup
        {"name": "voxel_edit", "kind": "voxel", "dim": 192, "quality": rb.VOXEL_HIGH,
         "width": 1280, "height": 720},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame(lo, hi):
        w = size(lo, hi)
        return {"width": w, "height": max(2, int(w * rng.uniform(0.5, 0.75)))}

    kind = rng.choice(["primary", "rays", "ao", "sdf", "sdf_frame", "nsdf_frame", "nsdf_eval",
                       "nsdf_grad", "batch", "voxel"])
    if kind == "primary":
        return {"kind": kind, "tris": size(4096, 262144), **frame(64, 2048),
                "one_sided": rng.random() < 0.5, "lanes": rng.choice([1, 32])}
    if kind == "rays":
        return {"kind": kind, "tris": size(4096, 262144), "rays": size(1000, 1000000),
                "any_hit": rng.random() < 0.5}
    if kind == "ao":
        return {"kind": kind, "cells": size(64, 512), **frame(160, 1920)}
    if kind == "sdf":
        return {"kind": kind, **frame(64, 1920)}
    if kind == "sdf_frame":
        return {"kind": kind, **frame(64, 1366), "flags": rng.choice([0, 1, 10, 15])}
    if kind == "nsdf_frame":
        return {"kind": kind, **frame(160, 1920)}
    if kind == "nsdf_eval":
        return {"kind": kind, "points": size(1000, 1000003)}
    if kind == "nsdf_grad":
        return {"kind": kind, "points": 512 * size(2, 128)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 6), "tris": size(10000, 100000),
                **frame(160, 640)}
    return {"kind": kind, "dim": size(32, 192), **frame(160, 1280),
            "quality": rng.choice([rb.VOXEL_LOW, rb.VOXEL_MEDIUM, rb.VOXEL_HIGH])}


# ---------------------------------------------------------------- inputs
def _camera(campos, lookat, fov_x, c):
    return rb.build_camera(campos, lookat,
                           (fov_x, rb.vertical_fov(fov_x, c["width"], c["height"])))


def _soup(tris, seed):
    cfg = configs.SoupConfig(num_tris=tris, seed=seed)
    return rb.KDScene.from_packed(cfg.packed(), cfg.kd_params())


def _hits(c):
    return torch.empty((c["width"] * c["height"], 4), dtype=torch.int32, device="cuda")


def _records(c):
    return torch.empty((c["width"] * c["height"], 8), dtype=torch.int32, device="cuda")


def _terrain(seed, c):
    return configs.TerrainConfig(seed=configs.PERLIN_SEED + seed % 100000, width=c["width"],
                                 height=c["height"])


def _rays(n, seed):
    """Rays from a sphere around the soup toward points inside it, re_ray
    layout {origin, tmax, direction, tag}."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    o = torch.randn((n, 3), generator=g, device="cuda")
    o = 3.0 * o / o.norm(dim=1, keepdim=True)
    d = 2.0 * torch.rand((n, 3), generator=g, device="cuda") - 1.0 - o
    rays = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3] = o
    rays[:, 3] = 1e20
    rays[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    rays[:, 7] = 0.0
    return rays


def _net_points(n, seed):
    lo, hi = (np.array(b, np.float32) for b in NET_BOX)
    return np.random.default_rng(seed).uniform(lo, hi, (n, 3)).astype(np.float32)


def _net_labels(pts, seed):
    """Signed distances to rolling hills, clipped as the training set's."""
    h = 2.0 * np.sin(0.21 * pts[:, 0]) * np.cos(0.17 * pts[:, 2])
    noise = np.random.default_rng(seed + 1).normal(0.0, 0.02, pts.shape[0])
    return np.clip(pts[:, 1] - h + noise, -4.0, 4.0).astype(np.float32)


def _net_params(seed):
    """Glorot-uniform weights and small biases, in the library's layout."""
    rng = np.random.default_rng(seed + 2)
    parts = []
    for fan_out, fan_in in ((64, 128), (64, 64), (64, 64), (64, 64), (1, 64)):
        a = math.sqrt(6.0 / (fan_in + fan_out))
        parts.append(rng.uniform(-a, a, fan_out * fan_in))
        parts.append(rng.uniform(-0.05, 0.05, fan_out))
    return np.concatenate(parts).astype(np.float32)


def _net_features(p, lo, hi, f0, dtype):
    lo = torch.as_tensor(np.asarray(lo), dtype=dtype, device=p.device)
    hi = torch.as_tensor(np.asarray(hi), dtype=dtype, device=p.device)
    q = (p.to(dtype) - 0.5 * (lo + hi)) * (2.0 / (hi - lo))
    cols = []
    for chain in range(2):
        for octave in range(8):
            a = 2.0 * math.pi * f0 * math.sqrt(2.0) ** chain * 2.0 ** octave * q
            cols.append(torch.stack([torch.sin(a), torch.cos(a)], 2).reshape(-1, 6))
    cols += [q, torch.zeros((q.shape[0], 29), dtype=dtype, device=p.device)]
    return torch.cat(cols, 1)


def _net_split(params):
    shapes = [(64, 128), (64,), (64, 64), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,)]
    out, at = [], 0
    for s in shapes:
        out.append(params[at:at + math.prod(s)].reshape(s))
        at += math.prod(s)
    return out


def _net_forward(w, x):
    for k in range(4):
        x = torch.nn.functional.softplus(x @ w[2 * k].T + w[2 * k + 1], threshold=100.0)
    return x @ w[8] + w[9]


def _trained_terrain(cfg, seed):
    """A NeuralSDF with the weights of a short offline fit to the terrain's
    own training set, as a program loads them from its checkpoint."""
    t = cfg.terrain
    lo, hi = cfg.box()
    net = rb.NeuralSDF(lo, hi, cfg.f0, cfg.init_seed)
    n = 1 << 17
    net.generate(t.params(), t.camera(), 1920, 1080, n, cfg.data_seed + seed % 100000)
    data = torch.from_numpy(net.data(n)).cuda()
    x = _net_features(data[:, :3], lo, hi, cfg.f0, torch.float32)
    params = torch.from_numpy(net.get_params()).cuda().requires_grad_()
    opt = torch.optim.Adam([params], lr=2e-3)
    for step in range(300):
        at = (step * 8192) % n
        loss = (_net_forward(_net_split(params), x[at:at + 8192]) - data[at:at + 8192, 3]).abs()
        opt.zero_grad()
        loss.mean().backward()
        opt.step()
    net.set_params(params.detach().cpu().numpy())
    return net, cfg.trace_params(net.lipschitz(20000, cfg.lipschitz_h, cfg.lipschitz_quantile))


def _hills(dim, seed):
    """A voxel terrain: {distance, material} of rolling hills."""
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.3, 0.6, 2)
    nx, ny, nz = dim, dim // 2, dim
    s = 24.0 / dim
    x = (np.arange(nx, dtype=np.float32) * s - 12.0)[None, None, :]
    y = (np.arange(ny, dtype=np.float32) * s - 6.0)[None, :, None]
    z = (np.arange(nz, dtype=np.float32) * s - 4.0)[:, None, None]
    d = y - 2.0 * np.sin(a * x) * np.cos(b * z) - 0.3 * np.sin(3.1 * x + 1.7 * z)
    data = np.zeros((nz, ny, nx, 2), np.float32)
    data[..., 0] = d
    data[..., 1] = np.floor(rng.uniform(0.0, 4.0))
    return (nx, ny, nz), (s, s, s), (-12.0, -6.0, -4.0), data


def _dig(seed):
    rng = np.random.default_rng(seed + 3)
    return [float(v) for v in rng.uniform((-4.0, -1.0, 1.0), (4.0, 1.0, 8.0))], 2.5


def _net_state(c, seed):
    net = rb.NeuralSDF(NET_BOX[0], NET_BOX[1], NET_F0, 1)
    net.set_params(_net_params(seed))
    return net


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "primary":
        s["scene"] = _soup(c["tris"], seed)
        s["scene"].set_tuning(1024, 0, 32, 32, c["lanes"])
        s["cam"] = _camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 60.0, c)
        s["out"] = _hits(c)
        s["flags"] = rb.TRACE_ONE_SIDED if c["one_sided"] else rb.TRACE_TWO_SIDED
    elif kind == "rays":
        s["scene"] = _soup(c["tris"], seed)
        s["rays"] = _rays(c["rays"], seed)
        s["out"] = torch.empty((c["rays"], 4), dtype=torch.int32, device="cuda")
        s["flags"] = rb.TRACE_ANY_HIT if c["any_hit"] else rb.TRACE_TWO_SIDED
    elif kind == "ao":
        cfg = configs.HeightfieldConfig(cells=c["cells"], seed=configs.PERLIN_SEED + seed % 100000,
                                        width=c["width"], height=c["height"])
        s["scene"] = rb.KDScene.from_mesh(*cfg.mesh_on_device())
        # what the frame's autotuner picks on B200
        s["scene"].set_tuning(0, 0, 8)
        s["cam"], s["cfg"] = cfg.camera(), cfg
        s["primary"] = _hits(c)
        s["mask"] = torch.empty(c["width"] * c["height"], dtype=torch.int32, device="cuda")
        s["nsec"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif kind in ("sdf", "sdf_frame", "nsdf_frame"):
        t = _terrain(seed, c)
        s["field"], s["cam"], s["hits"] = t.params(), t.camera(), _records(c)
        if kind == "sdf_frame":
            s["shade"] = rb.sdf_shade_params(flags=c["flags"])
            s["rgba"] = torch.empty(c["width"] * c["height"], dtype=torch.int32, device="cuda")
        elif kind == "nsdf_frame":
            s["net"], s["tp"] = _trained_terrain(configs.NeuralTerrainConfig(terrain=t), seed)
    elif kind == "nsdf_eval":
        s["net"] = _net_state(c, seed)
        s["pts"] = torch.from_numpy(_net_points(c["points"], seed)).cuda()
        s["out"] = torch.empty(c["points"], dtype=torch.float32, device="cuda")
    elif kind == "nsdf_grad":
        s["net"] = _net_state(c, seed)
        pts = _net_points(c["points"], seed)
        s["xyzl"] = torch.from_numpy(
            np.concatenate([pts, _net_labels(pts, seed)[:, None]], 1)).cuda()
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        scenes, s["meshes"] = [], []
        for i in range(c["scenes"]):
            # uneven sizes: every third scene is a terrain, the rest are soups
            size = {"width": max(2, c["width"] >> (i % 2)), "height": max(2, c["height"] >> (i % 2))}
            sc = dict(size, albedo=float(rng.uniform(0.5, 0.8)))
            if i % 3 == 1:
                t = configs.TerrainConfig(seed=configs.PERLIN_SEED + int(rng.integers(100000)),
                                          amplitude=float(rng.uniform(2.0, 3.5)), **size)
                sc.update(terrain=t.params(), camera=t.camera())
            else:
                mesh = _soup(max(1000, c["tris"] >> (i // 2)), int(rng.integers(1 << 30)))
                s["meshes"].append(mesh)
                sc.update(mesh=mesh, camera=_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 60.0, size))
            scenes.append(sc)
        s["batch"] = rb.Batch(scenes, 4, seed % 100000, 1e-4)
        s["out"] = torch.empty(s["batch"].total_pixels, dtype=torch.float32, device="cuda")
    else:
        dim, spacing, origin, data = _hills(c["dim"], seed)
        s["grid"] = rb.VoxelGrid(dim, spacing, origin, data)
        s["center"], s["radius"] = _dig(seed)
        s["march"] = rb.sdf_params(step_factor=0.6, eps=1e-3, tmax=100.0, max_steps=256)
        s["cam"] = _camera((0.0, 5.0, -14.0), (0.0, 0.0, 6.0), 60.0, c)
        s["hits"] = _records(c)
    return s


# ------------------------------------------------------------------ pass
def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "primary":
        return s["scene"].trace_primary(s["cam"], c["width"], c["height"], s["flags"], s["out"])
    if kind == "rays":
        return s["scene"].trace_rays(s["rays"], s["flags"], s["out"])
    if kind == "ao":
        f = s["cfg"]
        return s["scene"].render_ao(s["cam"], c["width"], c["height"], f.light_dir, f.ao_length,
                                    f.bias, f.ao_seed, s["primary"], s["mask"], s["nsec"])
    if kind == "sdf":
        return rb.sphere_trace(s["field"], s["cam"], c["width"], c["height"], s["hits"])
    if kind == "sdf_frame":
        return rb.render_sdf_frame(s["field"], s["shade"], s["cam"], c["width"], c["height"],
                                   s["hits"], s["rgba"])
    if kind == "nsdf_frame":
        return s["net"].trace(s["field"], s["tp"], s["cam"], c["width"], c["height"], s["hits"])
    if kind == "nsdf_eval":
        return s["net"].eval(s["pts"], s["out"])
    if kind == "nsdf_grad":
        return s["net"].loss_grad(s["xyzl"])
    if kind == "batch":
        return s["batch"].render(s["out"], graph=True)
    g = s["grid"]
    g.brush(rb.BRUSH_SPHERE_SUBTRACT, s["center"], s["radius"], 1.0)
    return g.trace(c["quality"], s["march"], s["cam"], c["width"], c["height"], s["hits"]), g.data


# ------------------------------------------------------------------ work
def work(case):
    """Bytes of the inputs and outputs, once each, and the operations of the
    algorithm (field evaluations per ray, tree steps and triangle tests as
    the counting calls and the benchmark report them, rounded)."""
    c, kind = case, case["kind"]
    if kind == "nsdf_eval":
        return {"bytes": 16 * c["points"], "flops": 2 * ROW_MACS * c["points"]}
    if kind == "nsdf_grad":
        return {"bytes": 20 * c["points"] + 8 * 20801, "flops": 6 * ROW_MACS * c["points"]}
    if kind == "rays":
        # 20 node steps of 4 operations and 15 tests of 50 per ray
        return {"bytes": 48 * c["rays"] + 160 * c["tris"], "flops": 830 * c["rays"]}
    n = c["width"] * c["height"]
    if kind == "primary":
        return {"bytes": 16 * n + 160 * c["tris"], "flops": 830 * n}
    if kind == "ao":
        # six rays per pixel; 96 bytes of tree per triangle
        return {"bytes": 20 * n + 192 * c["cells"] ** 2, "flops": 6 * 400 * n}
    if kind == "sdf":
        return {"bytes": 32 * n, "flops": 33 * FIELD_OPS * n}
    if kind == "sdf_frame":
        return {"bytes": 36 * n, "flops": (33 + 8 * (c["flags"] & 1)) * FIELD_OPS * n}
    if kind == "nsdf_frame":
        return {"bytes": 32 * n, "flops": 17 * FIELD_OPS * n + ROW_MACS * n}
    if kind == "batch":
        pixels = sum(max(2, c["width"] >> (i % 2)) * max(2, c["height"] >> (i % 2))
                     for i in range(c["scenes"]))
        return {"bytes": 4 * pixels + 160 * c["tris"] * 2, "flops": 3 * 5000 * pixels}
    # each voxel read and written by the edit; 12 lookups per pixel
    lookup = {rb.VOXEL_LOW: 10, rb.VOXEL_MEDIUM: 40, rb.VOXEL_HIGH: 250}[c["quality"]]
    return {"bytes": 16 * c["dim"] ** 2 * (c["dim"] // 2) + 32 * n, "flops": 12 * lookup * n}


# ----------------------------------------------------------------- exact
def exact(case, seed):
    """Network outputs, gradients and edited voxels in 64 bits.  Hit records,
    masks and pixels are whole values, and radiance depends on a path's
    random choices: they have none."""
    c, kind = case, case["kind"]
    if kind == "nsdf_eval":
        w = _net_split(torch.from_numpy(_net_params(seed)).cuda().double())
        pts = torch.from_numpy(_net_points(c["points"], seed)).cuda()
        return torch.cat([_net_forward(w, _net_features(p, *NET_BOX, NET_F0, torch.float64))
                          for p in pts.split(1 << 16)])
    if kind == "nsdf_grad":
        params = torch.from_numpy(_net_params(seed)).cuda().double().requires_grad_()
        pts = _net_points(c["points"], seed)
        labels = torch.from_numpy(_net_labels(pts, seed)).cuda().double()
        x = _net_features(torch.from_numpy(pts).cuda(), *NET_BOX, NET_F0, torch.float64)
        pred = _net_forward(_net_split(params), x)
        (pred - labels).abs().mean().backward()
        return params.grad, pred.detach()
    if kind == "voxel":
        dim, spacing, origin, data = _hills(c["dim"], seed)
        center, radius = _dig(seed)
        q = [origin[k] + np.arange(dim[k], dtype=np.float64) * np.float32(spacing[k])
             - np.float32(center[k]) for k in range(3)]
        ball = np.sqrt(q[0][None, None, :] ** 2 + q[1][None, :, None] ** 2
                       + q[2][:, None, None] ** 2) - radius
        out = data.astype(np.float64)
        dug = out[..., 0] <= -ball
        out[..., 0] = np.maximum(out[..., 0], -ball)
        out[..., 1] = np.where(dug, 1.0, out[..., 1])
        return None, out.reshape(-1)
    return None
