"""The batched renderer at its limits: claims of waiting warps, and shared
memory nearly full of staged nodes and terrain tables."""
import numpy as np
import pytest
import torch

import rayengine_b200 as rb

pytestmark = pytest.mark.gpu


def _cam(w, h):
    return rb.build_camera((0, 0, 3), (0, 0, 0), (60.0, rb.vertical_fov(60.0, w, h)))


@pytest.mark.parametrize("order", ["mt", "t"])
def test_waiting_warps_claim_once(cuda, order):
    """A few long terrain rays leave nearly every warp without work for most
    of the frame: each may ask the pixel cursors past their end once, or the
    32-bit cursors of a long enough frame would wrap and give pixels twice."""
    cfg = rb.configs.SoupConfig(num_tris=2000)
    mesh = rb.KDScene.from_packed(cfg.packed(), cfg.kd_params())
    # rays 200 long in steps of a fiftieth of the distance: some 4000 steps
    tc = rb.configs.TerrainConfig(width=16, height=9, step_factor=0.02, max_steps=4000)
    specs = {"m": dict(mesh=mesh, camera=_cam(33, 21), width=33, height=21, albedo=0.7),
             "t": dict(terrain=tc.params(), camera=tc.camera(), width=16, height=9, albedo=0.6)}
    pixels = np.array([33 * 21 * order.count("m"), 16 * 9 * order.count("t")])
    with rb.Batch([specs[k] for k in order], max_depth=2, seed=1, mesh_bias=1e-4) as b:
        rad = b.render().cpu().numpy()
        assert b.stats()["error"] == 0
        # at most 64 warps of 32 lanes are resident on each of the SMs
        warps = 64 * torch.cuda.get_device_properties(0).multi_processor_count
        claims = b.claims()
        assert (claims >= pixels).all()
        assert (claims <= pixels + 32 * warps).all(), claims
        assert np.array_equal(b.render(graph=True).cpu().numpy(), rad)
    mesh.close()


# scenes, block size, staged nodes per mesh: the paired tables of 12 seeds (48
# KB) do not fit beside the staged nodes, fit with fewer blocks per SM than the
# words (24 KB) in a batch of meshes and in one of terrains, and fit as often
@pytest.mark.parametrize("order,threads,stage", [
    ("m" * 6 + "t" * 12, 256, 4096), ("m" * 20 + "t" * 12, 256, 512),
    ("mm" + "t" * 12, 128, 0), ("m" * 44 + "t" * 12, 128, 0), ("mm" + "t" * 12, 256, 0)])
def test_tables_beside_staged_nodes(cuda, order, threads, stage):
    cfg = rb.configs.SoupConfig(num_tris=16384)
    mesh = rb.KDScene.from_packed(cfg.packed(), cfg.kd_params())
    assert mesh.stats()["num_nodes"] >= 4096
    specs = []
    for i, k in enumerate(order):
        if k == "m":
            specs.append(dict(mesh=mesh, camera=_cam(24, 18), width=24, height=18, albedo=0.7))
        else:
            tc = rb.configs.TerrainConfig(seed=900 + i, width=14, height=9)
            specs.append(dict(terrain=tc.params(), camera=tc.camera(), width=14, height=9,
                              albedo=0.6))
    with rb.Batch(specs, max_depth=3, seed=2, mesh_bias=1e-4) as b:
        want = b.render().cpu().numpy()  # the default tuning stages nothing
        counts = b.counts()
        b.set_tuning(threads, 8, stage, 8)
        for graph in (False, True):
            assert np.array_equal(b.render(graph=graph).cpu().numpy(), want)
        assert b.stats()["error"] == 0 and b.counts() == counts
    mesh.close()


def test_no_more_nodes_staged_than_there_are(cuda):
    """Eight trees of some 2200 nodes fit in shared memory; the 4096 asked for
    of each would not."""
    cfg = rb.configs.SoupConfig(num_tris=5000)
    mesh = rb.KDScene.from_packed(cfg.packed(), cfg.kd_params())
    assert 2048 < mesh.stats()["num_nodes"] < 3000
    scene = dict(mesh=mesh, camera=_cam(24, 18), width=24, height=18, albedo=0.7)
    with rb.Batch([scene] * 8, max_depth=3, seed=2, mesh_bias=1e-4) as b:
        want = b.render().cpu().numpy()
        b.set_tuning(256, 8, 4096, 8)
        assert np.array_equal(b.render().cpu().numpy(), want)
    mesh.close()


# fields that the paired form does not suit (few octaves, far coordinates) in
# most of the terrain pixels and in half of them
@pytest.mark.parametrize("fields", [[(3, 0.25), (3, 0.25), (8, 0.25)], [(1, 0.25), (8, 0.25)],
                                    [(8, 300.0), (8, 300.0), (7, 0.25)], [(2, 0.25)]])
def test_fields_the_pairs_do_not_suit(cuda, fields):
    from oracle import pyoracle as po

    specs, scenes = [], []
    for i, (octaves, scale) in enumerate(fields):
        tc = rb.configs.TerrainConfig(seed=40 + i, octaves=octaves, scale=scale, width=23, height=14)
        specs.append(dict(terrain=tc.params(), camera=tc.camera(), width=23, height=14, albedo=0.6))
        scenes.append(dict(kind=1, seed=tc.seed, octaves=octaves, scale=scale, amp=tc.amplitude,
                           step_factor=tc.step_factor, eps=tc.eps, tmax=tc.tmax,
                           max_steps=tc.max_steps, cam=tc.camera(), w=23, h=14, albedo=0.6))
    with rb.Batch(specs, max_depth=3, seed=5, mesh_bias=1e-4) as b:
        prim = torch.empty((b.total_pixels, 4), dtype=torch.int32, device="cuda")
        rad = b.render(primary=prim).cpu().numpy()
        g = np.arange(b.total_pixels, dtype=np.uint32)
        orad, oprim, _ = po.batch_path(scenes, b.offsets, g, 3, 5, 1e-4)
        assert np.array_equal(rad.view(np.uint32), orad.view(np.uint32))
        assert np.array_equal(prim.cpu().numpy()[:, :2], oprim[:, :2])


# the terrain tables past 16 seeds: words or bytes, by the blocks they leave an SM
# and the kind of most pixels
@pytest.mark.parametrize("meshes,terrains", [(0, 17), (0, 40), (3, 40), (0, 64), (40, 24)])
def test_many_seeds(cuda, meshes, terrains):
    from oracle import pyoracle as po

    cfg = rb.configs.SoupConfig(num_tris=2000)
    mesh = rb.KDScene.from_packed(cfg.packed(), cfg.kd_params())
    specs = [dict(mesh=mesh, camera=_cam(15, 12), width=15, height=12, albedo=0.7)] * meshes
    scenes = []
    for i in range(terrains):
        tc = rb.configs.TerrainConfig(seed=70 + i, octaves=5 + i % 4, width=11, height=7)
        specs = specs + [dict(terrain=tc.params(), camera=tc.camera(), width=11, height=7,
                              albedo=0.6)]
        scenes.append(dict(kind=1, seed=tc.seed, octaves=tc.octaves, scale=tc.scale,
                           amp=tc.amplitude, step_factor=tc.step_factor, eps=tc.eps, tmax=tc.tmax,
                           max_steps=tc.max_steps, cam=tc.camera(), w=11, h=7, albedo=0.6))
    with rb.Batch(specs, max_depth=3, seed=5, mesh_bias=1e-4) as b:
        rad = b.render().cpu().numpy()
        counts = b.counts()
        if not meshes:
            g = np.arange(b.total_pixels, dtype=np.uint32)
            orad, _, _ = po.batch_path(scenes, b.offsets, g, 3, 5, 1e-4)
            assert np.array_equal(rad.view(np.uint32), orad.view(np.uint32))
        for tuning in ((128, 8, 0, 8), (64, 32, 256, 64)):
            b.set_tuning(*tuning)
            assert np.array_equal(b.render(graph=True).cpu().numpy(), rad), tuning
            assert b.counts() == counts and b.stats()["error"] == 0
    mesh.close()
