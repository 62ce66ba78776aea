"""Batches of one kind of scene or both, at the seed counts where the terrain
tables change form (12 | 13 and 16 | 17 distinct seeds), in scene orders that
mix the kinds: radiance, primary hits, ray counts and work counters against
the CPU oracle and the counting frame."""
import numpy as np
import pytest
import torch

import rayengine_b200 as rb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DEPTH, SEED, BIAS = 3, 5, 1e-4


def _mesh(i, meshes):
    cfg = rb.configs.SoupConfig(num_tris=2000 + 500 * i, seed=i)
    packed = cfg.packed()
    meshes.append(rb.KDScene.from_packed(packed, cfg.kd_params()))
    w, h = 31 + i, 17
    cam = rb.build_camera((0, 0, 3), (0, 0, 0), (60.0, rb.vertical_fov(60.0, w, h)))
    return dict(mesh=meshes[-1], packed=packed, camera=cam, width=w, height=h, albedo=0.7)


def _terrain(i):
    # octave counts 7 and 8: an odd count ends on half a pair
    tc = rb.configs.TerrainConfig(seed=300 + i, amplitude=1.5 + 0.1 * i, octaves=8 - i % 2,
                                  width=14, height=9 + i % 3)
    return dict(terrain=tc.params(), camera=tc.camera(), width=tc.width, height=tc.height,
                albedo=0.6)


@pytest.mark.parametrize("order", ["m", "t", "mt", "tmtm", "mmttm", "m" + 12 * "t", "m" + 13 * "t",
                                   16 * "t" + "m", 17 * "t"])
def test_kinds_and_tables(cuda, order):
    meshes = []
    specs = [_mesh(i, meshes) if k == "m" else _terrain(i) for i, k in enumerate(order)]
    scenes = []
    for s in specs:
        if "mesh" in s:
            nodes, leaves, tris = s["mesh"].export()
            st = s["mesh"].stats()
            scenes.append(dict(kind=0, tris=s["packed"], bmin=st["bmin"], bmax=st["bmax"],
                               cam=s["camera"], w=s["width"], h=s["height"], albedo=s["albedo"]))
        else:
            f = s["terrain"]
            scenes.append(dict(kind=1, seed=f.seed, octaves=f.octaves, scale=f.scale,
                               amp=f.amplitude, step_factor=f.step_factor, eps=f.eps,
                               tmax=f.tmax, max_steps=f.max_steps, cam=s["camera"],
                               w=s["width"], h=s["height"], albedo=s["albedo"]))
    with rb.Batch(specs, max_depth=DEPTH, seed=SEED, mesh_bias=BIAS) as b:
        prim = torch.empty((b.total_pixels, 4), dtype=torch.int32, device="cuda")
        rad = b.render(primary=prim).cpu().numpy()
        st = b.stats()
        assert st["error"] == 0
        g = np.arange(b.total_pixels, dtype=np.uint32)
        orad, oprim, onrays = po.batch_path(scenes, b.offsets, g, DEPTH, SEED, BIAS)
        assert np.array_equal(rad.view(np.uint32), orad.view(np.uint32))
        assert np.array_equal(prim.cpu().numpy()[:, :2], oprim[:, :2])
        kind = np.concatenate([np.full(s["w"] * s["h"], s["kind"]) for s in scenes])
        assert st["rays"][0, 0] == b.total_pixels
        for bounce in range(1, DEPTH):
            for k in (0, 1):
                assert st["rays"][bounce, k] == int(((onrays > bounce) & (kind == k)).sum())
        counts = b.counts()
        assert (counts["field_evals"] > 0) == ("t" in order)
        assert (counts["tests"] > 0) == ("m" in order)
        for tuning in ((256, 8, 0, 8), (64, 32, 64, 64), (128, 1, 0, 1)):
            b.set_tuning(*tuning)
            assert np.array_equal(b.render(graph=True).cpu().numpy(), rad), tuning
            assert b.counts() == counts, tuning  # work done once per ray, whatever the schedule
    for m in meshes:
        m.close()
