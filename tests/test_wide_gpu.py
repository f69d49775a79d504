"""The four-wide traversal on the GPU (trees converted by tt_bvh_upload) against the two-wide tree of variant 3,
bit for bit, over small and odd ray counts and rays with special values in every field."""
import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for, soup
from trenchanttracer_gb300 import BVHCompact, DeviceBVH, Renderer, Scene, make_camera_meta, render_meta, render_params, scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = np.float32


def deep():
    """A stack of copies that reaches the depth limit: the tree stays two-wide."""
    v = np.concatenate([np.random.default_rng(1).normal(size=(3, 3)).astype(F)] * 120)
    return Scene.from_arrays(v, np.ones_like(v), np.arange(360, dtype=np.int32).reshape(-1, 3)), 1e-5, 1, 3.0


ALL = dict(SCENES, deep=deep, wide_leaves=lambda: (soup(900, 9, 0.3, 2.0), 1e-5, 64, 3.0))


def hits(dbvh, rays, variant, closest, ext):
    dbvh.set_variant(variant)
    h = torch.full((rays.shape[0], 6 if ext else 2), 77, dtype=torch.int32, device="cuda")
    dbvh.intersect(rays, h, closest=closest, ext=ext)
    dbvh.check()
    return h.cpu().numpy()


@pytest.mark.parametrize("name", sorted(ALL))
def test_four_wide_equals_two_wide_on_the_gpu(name):
    sc, alpha, leaf, extent = ALL[name]()
    dbvh = DeviceBVH(BVHCompact.build(sc, alpha, 1, leaf))
    rays = torch.from_numpy(rays_for(extent, 3, 70001)).cuda()
    for n in (1, 7, 31, 32, 33, 999, 40000, 70001):
        r = rays[:n].contiguous()
        for closest in (True, False):
            for ext in (False, True):
                ref = hits(dbvh, r, DeviceBVH.VARIANT_DYNAMIC, closest, ext)
                for variant in DeviceBVH.DETERMINISTIC_VARIANTS if n in (33, 40000) else (DeviceBVH.VARIANT_SORTED,):
                    assert np.array_equal(hits(dbvh, r, variant, closest, ext), ref), (n, closest, ext, variant)


@pytest.mark.parametrize("n", [(1 << 20) - 1, 1 << 20, (1 << 20) + 37])
def test_ordered_ray_sets_around_the_threshold(n):
    """From 2^20 rays on the default variant traces them in sorted order; every hit is its own ray's."""
    sc, alpha, leaf, extent = SCENES["spheres"]()
    dbvh = DeviceBVH(BVHCompact.build(sc, alpha, 1, leaf))
    rays = torch.from_numpy(rays_for(extent, 5, n)).cuda()
    for closest, ext in ((True, False), (False, True)):
        ref = hits(dbvh, rays, DeviceBVH.VARIANT_DYNAMIC, closest, ext)
        for variant in (DeviceBVH.VARIANT_SORTED, DeviceBVH.VARIANT_SORTED_OCC):
            assert np.array_equal(hits(dbvh, rays, variant, closest, ext), ref), (closest, ext, variant)


@pytest.mark.parametrize("streamed", [0, 1])
def test_ordered_queues_give_the_unordered_image(streamed):
    """Queues of 2^22 rays and more are ordered: waves whose queues cross that length, and a streamed pool of
    more slots than that."""
    sc = Scene.from_mesh(scenes.multi_material(12, 3))
    sc.set_env(scenes.sky_env(64, 32, sun_radiance=5e2, sun_diameter_deg=10.0))
    r = Renderer(DeviceBVH(BVHCompact.build(sc, 1e-5, 1, 8)), sc)
    w, h = 2311, 1999
    cam = make_camera_meta(w, h, [0.0, 14.0, 34.0], [0.0, -12.0, -34.0], fov=(60.0, 53.0))
    params = render_params(spp=3 if streamed else 1, max_depth=5, rr_depth=3, seed=3)
    images = []
    for ordered in (0, 1):
        r.set_launch(128, 8, 6000000, ordered, streamed)
        acc = torch.zeros(3 * w * h, device="cuda")
        r.render_native(cam, params, acc)
        r.check()
        images.append(acc.cpu().numpy().view(np.uint32))
    assert np.array_equal(*images)


@pytest.mark.parametrize("w,h,samples", [(16, 16, 1), (48, 32, 3), (333, 77, 2), (640, 352, 1)])
def test_compat_frames_do_not_depend_on_overlap_or_size(w, h, samples):
    """tt_render_compat hands its pixels to the warps that are there: every pixel of the whole 16 x 16 blocks gets
    its value once a frame, and frames on two streams do not disturb each other."""
    sc = Scene.from_mesh(scenes.cornell(2))
    sc.set_env(np.ones((8, 16, 3), F))
    r = Renderer(DeviceBVH(BVHCompact.build(sc, 1e-5, 1, 8)), sc)
    away = make_camera_meta(w, h, [0.0, 0.0, 1.55], [0.0, 0.0, 1.0], fov=(45.0, 45.0))  # every ray meets the sky
    box = make_camera_meta(w, h, [0.0, 0.0, 1.55], [0.0, 0.0, -1.0], fov=(45.0, 45.0))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    accs = [torch.zeros(h, w, 3, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    for k in (0, 1):
        r.render_compat(box, render_meta(7, samples), accs[k], stream=streams[k].cuda_stream)
    torch.cuda.synchronize()
    r.render_compat(box, render_meta(7, samples), accs[2])
    for _ in range(2):
        r.render_compat(away, render_meta(7, samples), accs[3])
    r.check()
    a, b, c, sky = (x.cpu().numpy() for x in accs)
    assert np.array_equal(a, b) and np.array_equal(a, c)
    # rows count from the image's bottom; the blocks cover its top rows and left columns
    inside = np.zeros((h, w), bool)
    inside[h - h // 16 * 16:, :w // 16 * 16] = True
    assert not a[~inside].any() and not sky[~inside].any()
    one = F(0)
    for _ in range(samples):  # the samples' sum as the kernel rounds it; the sky counts twice
        one = F(np.float64(F(2.0)) * np.float64(F(1.0) / F(samples)) + np.float64(one))
    assert (sky[inside] == one + one).all()


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_page_locked_host_rays(offset):
    """Page-locked rays and hits go through the mapped buffers, rays and hits that start off a 16- or 8-byte
    boundary through staging; the hits are those of device rays either way."""
    sc, alpha, leaf, extent = SCENES["spheres"]()
    dbvh = DeviceBVH(BVHCompact.build(sc, alpha, 1, leaf))
    for n in (1, 33, 5000, 70001):
        rays = rays_for(extent, 21, n)
        h_rays = torch.empty(8 * n + 4).pin_memory().numpy()[offset:offset + 8 * n].reshape(n, 8)
        h_hits = torch.empty(2 * n + 4, dtype=torch.int32).pin_memory().numpy()[offset:offset + 2 * n].reshape(n, 2)
        h_rays[:] = rays
        for closest in (True, False):
            h_hits[:] = 77
            dbvh.intersect_host(h_rays, h_hits, closest=closest)
            want = hits(dbvh, torch.from_numpy(rays).cuda(), DeviceBVH.VARIANT_DYNAMIC, closest, False)
            dbvh.set_variant(DeviceBVH.VARIANT_SORTED)
            assert np.array_equal(h_hits, want), (n, closest)


@pytest.mark.parametrize("n", [33, 5000, (1 << 20) + 1])
def test_calls_captured_calls_and_streams_in_any_order(n):
    """Direct calls, replays of a captured call and calls on other streams use work counters of their own."""
    sc, alpha, leaf, extent = SCENES["spheres"]()
    dbvh = DeviceBVH(BVHCompact.build(sc, alpha, 1, leaf))
    rays = torch.from_numpy(rays_for(extent, 6, n)).cuda()
    few = rays[:17].contiguous()
    ref, ref_few = hits(dbvh, rays, DeviceBVH.VARIANT_DYNAMIC, True, False), hits(dbvh, few, DeviceBVH.VARIANT_DYNAMIC, True, False)
    dbvh.set_variant(DeviceBVH.VARIANT_SORTED)
    h, g, o = (torch.full((k, 2), 77, dtype=torch.int32, device="cuda") for k in (n, n, 17))
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    dbvh.intersect(rays, h)  # allocates what the call needs
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        dbvh.intersect(rays, g, stream=side.cuda_stream)
    for k in range(7):
        for t in (h, g, o):
            t.fill_(77)
        torch.cuda.synchronize()
        for _ in range(k % 3):
            dbvh.intersect(few, o)
        graph.replay()
        dbvh.intersect(rays, h)
        torch.cuda.synchronize()
        dbvh.intersect(few, o, stream=side.cuda_stream)
        side.synchronize()
        dbvh.check()
        assert np.array_equal(h.cpu().numpy(), ref) and np.array_equal(g.cpu().numpy(), ref), k
        assert np.array_equal(o.cpu().numpy(), ref_few), k
