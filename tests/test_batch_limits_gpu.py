"""The batched renderer at its limits: claims of waiting warps."""
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
