"""Voxel SDF on the GPU against the CPU oracle: bake, the three samplers
and the voxel sphere tracer, bit for bit; .rsdf round trip."""
import numpy as np
import pytest
import torch

import rayengine_b200 as rb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DIM, SP, ORG = (48, 24, 40), (0.5, 0.5, 0.5), (-12.0, -6.0, -4.0)


def _grid():
    tc = rb.configs.TerrainConfig()
    return tc, rb.VoxelGrid.bake(tc.params(), DIM, SP, ORG)


def test_bake_and_samplers_match_oracle(cuda):
    tc, g = _grid()
    got = g.data.cpu().numpy()
    want = po.voxel_bake(po.perm(tc.seed), tc.octaves, tc.scale, tc.amplitude, DIM, SP, ORG)
    assert np.array_equal(got, want)
    rng = np.random.default_rng(2)
    lo = np.array(ORG, np.float32) - 1.0
    hi = np.array(ORG, np.float32) + np.array(DIM, np.float32) * 0.5 + 1.0
    pts = rng.uniform(lo, hi, (20000, 3)).astype(np.float32)
    d = torch.from_numpy(pts).cuda()
    for q in (rb.VOXEL_LOW, rb.VOXEL_MEDIUM, rb.VOXEL_HIGH):
        s = g.sample(d, q).cpu().numpy()
        assert np.array_equal(s, po.voxel_sample(got, DIM, SP, ORG, q, pts)), q


def test_voxel_trace_matches_oracle_and_file_round_trip(cuda, tmp_path):
    tc, g = _grid()
    w, h = 80, 45
    cam = rb.build_camera((0.0, 6.0, -14.0), (0.0, 0.0, 6.0), (60.0, rb.vertical_fov(60.0, w, h)))
    march = rb.sdf_params(step_factor=0.6, eps=1e-3, tmax=100.0, max_steps=256)
    grid = g.data.cpu().numpy()
    for q in (rb.VOXEL_LOW, rb.VOXEL_MEDIUM, rb.VOXEL_HIGH):
        out = g.trace(q, march, cam, w, h).cpu().numpy()
        ref = po.voxel_trace(grid, DIM, SP, ORG, q, 0.6, 1e-3, 100.0, 256, cam, w, h)
        f = out.view(np.float32).reshape(-1, 8)
        u = out.view(np.uint32).reshape(-1, 8)
        assert np.array_equal(u[:, 7], ref["status"]), q
        assert np.array_equal(u[:, 6], ref["steps"]), q
        hit = ref["status"] == 1
        assert hit.mean() > 0.3
        assert np.array_equal(f[hit, 0:3], ref["pos"][hit])
        assert np.array_equal(f[hit, 3], ref["normal"][hit, 0])
        assert np.array_equal(f[hit, 4:6], ref["normal"][hit, 1:3])
    path = str(tmp_path / "terrain.rsdf")
    g.save(path)
    g2 = rb.VoxelGrid.load(path, origin=ORG)
    assert np.array_equal(g2.data.cpu().numpy(), grid)
    a = g.trace(rb.VOXEL_MEDIUM, march, cam, w, h).cpu().numpy()
    b = g2.trace(rb.VOXEL_MEDIUM, march, cam, w, h).cpu().numpy()
    assert np.array_equal(a, b)


def test_brush_edits_match_oracle(cuda):
    tc, g = _grid()
    grid = g.data.cpu().numpy()
    edits = [(rb.BRUSH_SPHERE_ADD, (0.0, 1.0, 4.0), 2.0, 3.0),
             (rb.BRUSH_SPHERE_SUBTRACT, (2.0, -0.5, 6.0), 1.5, 4.0),
             (rb.BRUSH_CUBE_ADD, (-4.0, 0.5, 8.0), (1.0, 2.0, 1.5), 5.0),
             (rb.BRUSH_CUBE_SUBTRACT, (3.0, 0.0, 2.0), (2.0, 1.0, 1.0), 6.0)]
    for kind, c, e, mat in edits:
        g.brush(kind, c, e, material=mat, smooth=0.1)
        grid = po.voxel_brush(grid, DIM, SP, ORG, kind, c, e, mat, 0.1)
        assert np.array_equal(g.data.cpu().numpy(), grid), kind
    # the edits changed the field
    assert not np.array_equal(grid, po.voxel_bake(po.perm(tc.seed), tc.octaves, tc.scale,
                                                  tc.amplitude, DIM, SP, ORG))


@pytest.mark.parametrize("quality", [rb.VOXEL_LOW, rb.VOXEL_MEDIUM, rb.VOXEL_HIGH])
@pytest.mark.parametrize("dim", [(2, 2, 2), (3, 5, 4), (4, 4, 4), (5, 4, 7), (33, 17, 9)])
def test_small_grids_and_ragged_frames(cuda, dim, quality):
    """Grids with no cell, one cell and a few whose neighbours all lie inside;
    points on voxels, across every face and far outside; frames from 2x2 to
    several ragged tiles.  Bit for bit against the oracle."""
    rng = np.random.default_rng(dim[0])
    sp, org = (0.5, 0.75, 0.4), (-1.0, 0.5, 2.0)
    nx, ny, nz = dim
    y = np.arange(ny, dtype=np.float32)[None, :, None] - 0.45 * ny
    data = np.zeros((nz, ny, nx, 2), np.float32)
    data[..., 0] = 0.5 * y + rng.normal(0, 0.1, (nz, ny, nx)).astype(np.float32)
    g = rb.VoxelGrid(dim, sp, org, data)
    grid = g.data.cpu().numpy()
    ext = np.array(dim, np.float64) * sp
    pts = rng.uniform(np.array(org) - 2.5, np.array(org) + ext + 2.5, (4000, 3))
    on = np.stack([rng.integers(-3, d + 3, 500) * np.float32(s) + np.float32(o)
                   for d, s, o in zip(dim, sp, org)], 1)
    pts = np.concatenate([pts, on, [[1e9, -1e9, 1e30]]]).astype(np.float32)
    got = g.sample(torch.from_numpy(pts).cuda(), quality).cpu().numpy()
    want = po.voxel_sample(grid, dim, sp, org, quality, pts)
    # the C oracle's conversion to int is defined below 2^31 only: the point
    # at z = 1e30 is looked up (a voxel of the grid) but has no oracle value
    fits = np.abs((pts.astype(np.float64) - org) / sp).max(1) < 2.0 ** 31 - 4.0
    assert np.array_equal(fits, np.arange(len(pts)) < len(pts) - 1)
    assert np.array_equal(got.view(np.uint32)[fits], want.view(np.uint32)[fits])
    assert np.isfinite(got).all()
    march = rb.sdf_params(step_factor=0.6, eps=1e-3, tmax=100.0, max_steps=64)
    mid = np.array(org) + 0.5 * ext
    for w, h in ((2, 2), (9, 5), (70, 43)):
        cam = rb.build_camera(tuple(mid + (0.3, 4.0, -5.0)), tuple(mid), (60.0, 45.0))
        u = g.trace(quality, march, cam, w, h).cpu().numpy().view(np.uint32).reshape(-1, 8)
        ref = po.voxel_trace(grid, dim, sp, org, quality, 0.6, 1e-3, 100.0, 64, cam, w, h)
        assert np.array_equal(u[:, 7], ref["status"])
        assert np.array_equal(u[:, 6], ref["steps"])
        hit = ref["status"] == 1
        assert np.array_equal(u[hit, 0:3], ref["pos"][hit].view(np.uint32))
        # a flat neighbourhood (nearest voxel) has no normal: NaN on both sides
        assert np.array_equal(u[hit, 3:6].view(np.float32), ref["normal"][hit], equal_nan=True)
        assert not u[~hit, 0:6].any()


@pytest.mark.parametrize("quality", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 1000])
def test_lookups_whatever_their_neighbours(cuda, quality, n):
    """A warp takes the path that suits all its points: each point's value is
    the one it has alone, inside the grid, across its faces and far outside."""
    rng = np.random.default_rng(4)
    dim, spacing, origin = (13, 9, 11), (0.5, 0.7, 0.6), (-3.0, -2.0, -1.0)
    grid = rb.VoxelGrid(dim, spacing, origin, rng.normal(size=(dim[0] * dim[1] * dim[2], 2)))
    pts = rng.uniform(-6.0, 8.0, (n, 3)).astype(np.float32)
    pts[::7] = rng.uniform(-1.0, 2.0, (len(pts[::7]), 3))
    pts[5::40] = 1e30
    d = torch.from_numpy(pts).cuda()
    got = grid.sample(d, quality).cpu().numpy()
    alone = np.array([float(grid.sample(d[i:i + 1].contiguous(), quality)) for i in range(min(n, 64))],
                     np.float32)
    assert np.array_equal(got[:64].view(np.uint32), alone.view(np.uint32))
    inner = grid.sample(d[::7].contiguous(), quality).cpu().numpy()
    assert np.array_equal(got[::7].view(np.uint32), inner.view(np.uint32))
