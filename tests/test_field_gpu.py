"""The field evaluated two octaves at a time against the CPU oracle, bit for
bit: octave counts around the pairs (odd ones end on half a pair), and
coordinates below, across and beyond the range of the paired form (the
largest |scale * p| times 2^octaves below 2^22) on both sides of zero."""
import numpy as np
import pytest
import torch

import rayengine_b200 as rb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

DIM = (37, 6, 11)


def _bake(octaves, scale, spacing, origin):
    field = rb.sdf_params(octaves=octaves, scale=scale, amplitude=3.0)
    got = rb.VoxelGrid.bake(field, DIM, spacing, origin).data.cpu().numpy()
    want = po.voxel_bake(po.perm(2016), octaves, scale, 3.0, DIM, spacing, origin)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert len(np.unique(got)) > DIM[1]


@pytest.mark.parametrize("octaves", [1, 2, 3, 7, 8, 9, 16])
def test_octave_counts(cuda, octaves):
    # about zero, lattice points (multiples of 4) among the samples
    _bake(octaves, 0.25, (0.5, 1.0, 0.37), (-9.0, -3.0, -2.0))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("octaves", [7, 8])
def test_across_the_paired_range(cuda, octaves, axis, sign):
    # |scale p| crosses 2^(22 - octaves) within the grid
    edge = 2.0 ** (22 - octaves) / 0.25
    origin = [-9.0, -3.0, -2.0]
    origin[axis] = sign * edge - 2.5
    _bake(octaves, 0.25, (0.5, 1.0, 0.5), tuple(origin))


def test_far_from_the_origin(cuda):
    _bake(8, 1.0, (3.0, 1024.0, 513.0), (3.0e6, -3.0, -7.0e8))


# pixels at and past 8 and 16 rays for each of 148 x 20 warps, where a frame's
# rays go from four lanes each to two and one, and frames of a few rays
@pytest.mark.parametrize("w,h,octaves", [(2, 2, 8), (37, 5, 9), (64, 36, 7), (160, 148, 8),
                                         (161, 148, 8), (320, 148, 8), (321, 148, 8)])
def test_frames_of_few_rays(cuda, w, h, octaves):
    cfg = rb.configs.TerrainConfig(width=w, height=h, octaves=octaves)
    shade = rb.sdf_shade_params()
    img, hits = rb.render_sdf_frame(cfg.params(), shade, cfg.camera(), w, h)
    plain = rb.sphere_trace(cfg.params(), cfg.camera(), w, h)
    assert torch.equal(plain, hits)
    ref = po.sdf_image(po.perm(cfg.seed), cfg.camera(), w, h, octaves=octaves)
    u = plain.cpu().numpy().view(np.uint32).reshape(-1, 8)
    assert np.array_equal(u[:, 6], ref["steps"])
    assert np.array_equal(u[:, 7], ref["status"])
    hit = ref["status"] == 1
    assert np.array_equal(u[hit, 0:3], ref["pos"][hit].view(np.uint32))
    assert np.array_equal(u[hit, 3:6], ref["normal"][hit].view(np.uint32))
    want = po.sdf_frame(po.perm(cfg.seed), cfg.camera(), w, h, cfg.params(), shade)
    assert np.array_equal(img.cpu().numpy().view(np.uint32), want)


# frames with some rays, most and all of them past the near form's range, odd
# and even octave counts, coordinates past 2^23 and up to the largest integers
# (beyond those the oracle's conversion is undefined in C)
@pytest.mark.parametrize("octaves,scale", [(16, 1.0), (17, 0.25), (32, 0.004), (8, 300.0),
                                           (3, 1e6), (8, 70000.0)])
def test_frames_past_the_near_range(cuda, octaves, scale):
    w, h = 67, 41
    cfg = rb.configs.TerrainConfig(width=w, height=h, octaves=octaves, scale=scale)
    got = rb.sphere_trace(cfg.params(), cfg.camera(), w, h).cpu().numpy().view(np.uint32)
    ref = po.sdf_image(po.perm(cfg.seed), cfg.camera(), w, h, octaves=octaves, scale=scale)
    u = got.reshape(-1, 8)
    assert np.array_equal(u[:, 6], ref["steps"])
    assert np.array_equal(u[:, 7], ref["status"])
    hit = ref["status"] == 1
    assert np.array_equal(u[hit, 0:3], ref["pos"][hit].view(np.uint32))
    normal, want = u[hit, 3:6].view(np.float32), ref["normal"][hit]
    nan = np.isnan(want)  # whose payload is not compared
    assert np.array_equal(np.isnan(normal), nan)
    assert np.array_equal(normal[~nan].view(np.uint32), want[~nan].view(np.uint32))


# the field's two forms (pairs on the rows, one octave at a time on copies) at
# the octave counts and sizes where kernels go from one to the other
@pytest.mark.parametrize("octaves,w,h", [(1, 64, 36), (2, 64, 36), (2, 512, 511), (2, 512, 512),
                                         (3, 128, 63), (3, 128, 64), (4, 64, 36)])
def test_forms_of_the_marches(cuda, octaves, w, h):
    cfg = rb.configs.TerrainConfig(width=w, height=h, octaves=octaves)
    shade = rb.sdf_shade_params(flags=1)
    pix = np.random.default_rng(1).choice(w * h, min(w * h, 5000), replace=False).astype(np.uint32)
    img, hits = rb.render_sdf_frame(cfg.params(), shade, cfg.camera(), w, h)
    u = hits.cpu().numpy().view(np.uint32).reshape(-1, 8)[pix]
    ref = po.sdf_image(po.perm(cfg.seed), cfg.camera(), w, h, octaves=octaves, pixels=pix)
    assert np.array_equal(u[:, 6], ref["steps"]) and np.array_equal(u[:, 7], ref["status"])
    hit = ref["status"] == 1
    assert np.array_equal(u[hit, 0:3], ref["pos"][hit].view(np.uint32))
    assert np.array_equal(u[hit, 3:6], ref["normal"][hit].view(np.uint32))
    if w * h < 10000:
        want = po.sdf_frame(po.perm(cfg.seed), cfg.camera(), w, h, cfg.params(), shade)
        assert np.array_equal(img.cpu().numpy().view(np.uint32), want)
    # the neural tracer's exact phase alone starts at the camera: the same
    # steps until a ray's crossing is bracketed, so the same hit or miss
    net = rb.NeuralSDF((-40.0, -6.0, -20.0), (40.0, 11.0, 60.0), 0.5, 1)
    for taps in (1, 4, 6):
        tp = rb.nsdf_trace_params(exact_only=True, normal_taps=taps, root_steps=4)
        out = net.trace(cfg.params(), tp, cfg.camera(), w, h).cpu().numpy()
        far = rb.nsdf_trace_params(exact_only=True, normal_taps=1, root_steps=4)
        base = net.trace(cfg.params(), far, cfg.camera(), w, h).cpu().numpy()
        assert np.array_equal(out[:, :3], base[:, :3]) and np.array_equal(out[:, 7], base[:, 7])
    net.close()


@pytest.mark.parametrize("octaves,dim", [(1, (64, 65, 64)), (2, (50, 63, 63)), (2, (50, 64, 63)),
                                         (8, (50, 64, 62)), (8, (50, 64, 63)), (3, (128, 129, 255)),
                                         (3, (128, 129, 257)), (7, (50, 64, 63))])
def test_forms_of_the_bake(cuda, octaves, dim):
    field = rb.sdf_params(octaves=octaves, scale=0.25, amplitude=3.0)
    sp, org = (0.2, 0.3, 0.25), (-9.0, -3.0, -2.0)
    got = rb.VoxelGrid.bake(field, dim, sp, org).data.cpu().numpy()
    want = po.voxel_bake(po.perm(2016), octaves, 0.25, 3.0, dim, sp, org)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
