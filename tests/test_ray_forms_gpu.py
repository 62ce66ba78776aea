"""The forms a ray pass takes by its number of rays and its tree (lanes per
ray, shared tests, one lane per ray), at the sizes where they change, bit for
bit: frames and closest-hit rays against the oracle, any-hit rays against the
lane-refill walk (the oracle's any-hit triangle may differ)."""
import numpy as np
import pytest
import torch

import rayengine_b200 as rb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _kd(sc):
    st = sc.stats()
    nodes, leaves, tris = sc.export()
    return st, po.KdTree(nodes, leaves, tris, st["bmin"], st["bmax"])


def _scene(long_leaves, **kw):
    cfg = rb.configs.SoupConfig(num_tris=6000)
    params = rb.kd_params(max_depth=24, leaf_size=8, **kw) if long_leaves else rb.kd_params(**kw)
    sc = rb.KDScene.from_packed(cfg.packed(), params)
    st = sc.stats()
    assert (st["num_refs"] >= 3 * st["num_leaves"]) == long_leaves
    return sc


def _rays(n):
    rng = np.random.default_rng(6)
    o = rng.uniform(-1.6, 1.6, (n, 3))
    d = rng.normal(size=(n, 3))
    d[: n // 10, 1:] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tmax = rng.choice([np.inf, 0.5, 1e20], n)
    return np.concatenate([o, tmax[:, None], d, np.zeros((n, 1))], 1).astype(np.float32)


# widths x heights at and just past 4096, 40,960 and 81,920 pixels, and the
# smallest frame
SIZES = [(2, 2), (64, 64), (241, 17), (256, 160), (283, 145), (320, 256), (331, 248)]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("long_leaves", [False, True])
def test_frames(cuda, long_leaves, mode):
    with _scene(long_leaves) as sc:
        st, kd = _kd(sc)
        for w, h in SIZES:
            cam = rb.build_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (60.0, 50.0))
            ref = po.primary_kd(kd, cam, w, h, mode=mode).view(np.int32).reshape(-1, 4)
            got = sc.trace_primary(cam, w, h, mode).cpu().numpy()
            assert np.array_equal(got, ref), (w, h)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("long_leaves", [False, True])
def test_caller_rays(cuda, long_leaves, mode):
    rays = _rays(50001)
    with _scene(long_leaves) as sc:
        st, kd = _kd(sc)
        ref = po.rays_kd(kd, rays, mode=mode).view(np.int32).reshape(-1, 4)
        dr = torch.from_numpy(rays).cuda()
        t = sc.tuning()
        any_hit = mode | rb.TRACE_ANY_HIT
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], 8)
        first = sc.trace_rays(dr, any_hit)
        assert np.array_equal(first[:, 0].cpu().numpy() >= 0, ref[:, 0] >= 0)
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], 32)
        for n in (1, 3, 33, 4096, 4097, 40960, 40961, 50001):
            part = dr[:n].contiguous()
            assert np.array_equal(sc.trace_rays(part, mode).cpu().numpy(), ref[:n]), n
            assert torch.equal(sc.trace_rays(part, any_hit), first[:n]), n


@pytest.mark.parametrize("n", [1000, 20000, 45000])
def test_visit_cap(cuda, n):
    """A walk stopped at the leaf-visit cap is counted once in every form."""
    rays = _rays(n)
    with _scene(True, max_leaf_visits=2) as sc:
        st, kd = _kd(sc)
        ref = po.rays_kd(kd, rays, max_visits=2).view(np.int32).reshape(-1, 4)
        dr = torch.from_numpy(rays).cuda()
        t = sc.tuning()
        got, cut = sc.trace_rays(dr).cpu().numpy(), sc.truncated()
        assert np.array_equal(got, ref)
        hit = sc.trace_rays(dr, rb.TRACE_ANY_HIT)
        any_cut = sc.truncated()
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], 8)
        assert np.array_equal(sc.trace_rays(dr).cpu().numpy(), ref)
        assert sc.truncated() == cut > n // 20
        assert torch.equal(sc.trace_rays(dr, rb.TRACE_ANY_HIT), hit)
        assert sc.truncated() == any_cut > 0


@pytest.mark.parametrize("long_leaves", [False, True])
def test_plain_walk(cuda, long_leaves):
    """The walk without refill or shared lanes, where the default chooses
    another form: the same hits."""
    rays = _rays(50001)
    with _scene(long_leaves) as sc:
        dr = torch.from_numpy(rays).cuda()
        cam = rb.build_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (60.0, 50.0))
        t = sc.tuning()
        want = [[sc.trace_primary(cam, w, h) for w, h in SIZES],
                [sc.trace_rays(dr[:n].contiguous(), f) for n in (1000, 20000, 50001)
                 for f in (0, rb.TRACE_ANY_HIT)]]
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], rb.RAY_NO_REFILL)
        got = [[sc.trace_primary(cam, w, h) for w, h in SIZES],
               [sc.trace_rays(dr[:n].contiguous(), f) for n in (1000, 20000, 50001)
                for f in (0, rb.TRACE_ANY_HIT)]]
        for a, b in zip(want[0] + want[1], got[0] + got[1]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("refill", [1, 8, 32])
@pytest.mark.parametrize("long_leaves", [False, True])
def test_ao_frames(cuda, long_leaves, refill):
    """The AO frame's passes bound their descents by the tree and the refill
    threshold: hits, masks and work counts as the oracle's."""
    cfg = rb.configs.SoupConfig(num_tris=6000)
    packed, light = cfg.packed(), rb.unit((0.3, 1.0, 0.2))
    w, h = 131, 67
    cam = rb.build_camera((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (60.0, 50.0))
    with _scene(long_leaves) as sc:
        st, kd = _kd(sc)
        sc.set_tuning(sc.tuning()["stage_nodes"], 0, refill)
        hits, mask, nsec = sc.render_ao(cam, w, h, light, 0.3, 1e-4, 5)
        rh, rm, rn = po.frame_ao(kd, packed, cam, w, h, light, 0.3, 1e-4, 5)
        assert np.array_equal(hits.cpu().numpy(), rh.view(np.int32).reshape(-1, 4))
        assert np.array_equal(mask.cpu().numpy().view(np.uint32), rm)
        assert int(nsec.item()) == rn > 0
        want = sc.render_ao_counts(cam, w, h, rb.ao_params(light, 0.3, 1e-4, 5))
        sc.set_tuning(0, 2, 8)
        assert sc.render_ao_counts(cam, w, h, rb.ao_params(light, 0.3, 1e-4, 5)) == want


def _camera_rows(w, h):
    """A camera's rays in row order, from (0, 0, 3) to the origin, 60 degrees
    wide."""
    t = np.tan(np.radians(30.0))
    x, y = np.meshgrid(np.linspace(-t, t, w), np.linspace(t, -t, h) * h / w)
    d = np.stack([x, y, -np.ones_like(x)], -1).reshape(-1, 3)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((w * h, 8), np.float32)
    rays[:, 2], rays[:, 3], rays[:, 4:7] = 3.0, 1e20, d
    return rays


# 1,500,000 rays: from here on their order decides between the forms
@pytest.mark.parametrize("n", [1499999, 1500000, 1500013])
@pytest.mark.parametrize("order", ["rows", "shuffled", "rows, then shuffled", "not finite"])
def test_many_caller_rays(cuda, order, n):
    rays = torch.from_numpy(_camera_rows(1600, 938)[:n]).cuda()
    g = torch.Generator(device="cuda").manual_seed(3)
    mixed = rays[torch.randperm(n, generator=g, device="cuda")]
    if order == "shuffled":
        rays = mixed
    elif order != "rows":
        rays = torch.cat([rays[: n // 2], mixed[n // 2:]])
    if order == "not finite":
        rays[::33, 4] = float("nan")
        rays[5::33, 0] = float("inf")
    rays = rays.contiguous()
    with _scene(True, max_leaf_visits=3) as sc:
        t = sc.tuning()
        for flags in (0, 1, rb.TRACE_ANY_HIT, 1 | rb.TRACE_ANY_HIT):
            got, cut = sc.trace_rays(rays, flags), sc.truncated()
            sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"],
                          rb.RAY_NO_REFILL)
            assert torch.equal(got, sc.trace_rays(rays, flags)), flags
            assert sc.truncated() == cut
            sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], 32)
        assert (got[:, 0] >= 0).sum() > n // 50


@pytest.mark.parametrize("flags", [0, 1, rb.TRACE_ANY_HIT])
def test_caller_rays_fill_the_gpu(cuda, flags):
    """At and past the numbers of rays that are resident at once with 8 and
    with 4 lanes each."""
    warps = 48 * torch.cuda.get_device_properties(0).multi_processor_count
    with _scene(False) as sc:
        dr = torch.from_numpy(_rays(8 * warps + 1)).cuda()
        t = sc.tuning()
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], rb.RAY_NO_REFILL)
        want = sc.trace_rays(dr, flags)
        sc.set_tuning(t["stage_nodes"], t["queue_kind_major"], t["refill_min"], 32)
        for n in (4 * warps, 4 * warps + 1, 8 * warps - 3, 8 * warps, 8 * warps + 1):
            assert torch.equal(sc.trace_rays(dr[:n].contiguous(), flags), want[:n]), n
