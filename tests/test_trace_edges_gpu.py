"""Calls at the edges of what the trace entry points accept, on the GPU: files whose tree is no plain tree, calls on
several streams, host buffers in unusual places."""
import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for
from trenchanttracer_gb300 import (BVHCompact, DeviceBVH, Renderer, Scene, TTError, make_camera_meta, render_meta,
                                   render_params, scenes)

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = np.float32


def tree(name):
    sc, alpha, leaf, extent = SCENES[name]()
    return BVHCompact.build(sc, alpha, 1, leaf), extent


def trace(dbvh, rays, closest=True):
    h = torch.full((rays.shape[0], 2), 77, dtype=torch.int32, device="cuda")
    dbvh.intersect(rays, h, closest=closest)
    dbvh.check()
    return h.cpu().numpy()


def edited(bvh, path, edit):
    """The tree of bvh with its node and vertex words changed: bvh.cache written, edited and loaded."""
    bvh.save(path)
    raw = np.fromfile(path, np.int32)
    n, v = int(raw[0]), int(raw[3])
    words = list(np.split(raw, [7, 7 + 4 * n, 7 + 4 * n + 4 * v]))
    words[1] = edit(words[1].reshape(-1, 4)).reshape(-1)
    words[0][0] = len(words[1]) // 4
    np.concatenate(words).tofile(path)
    return BVHCompact.load(path)


def test_file_with_a_node_that_no_node_refers_to(tmp_path):
    bvh, extent = tree("terrain")
    odd = edited(bvh, tmp_path / "bvh.cache", lambda nodes: np.concatenate([nodes, nodes[-4:]]))
    rays = torch.from_numpy(rays_for(extent, 3, 20001)).cuda()
    ref, got = DeviceBVH(bvh), DeviceBVH(odd)
    for closest in (True, False):
        assert np.array_equal(trace(got, rays, closest), trace(ref, rays, closest))


@pytest.mark.parametrize("n", [1000, 40000, (1 << 20) + 1])
def test_calls_whose_streams_run_in_another_order_than_they_were_issued(n):
    """A call that waits in its stream while later calls on another stream come and go: each traces all its rays. The
    small set needs no counter; the larger ones' calls do not run at the same time."""
    bvh, extent = tree("spheres")
    dbvh = DeviceBVH(bvh)
    rays = torch.from_numpy(rays_for(extent, 6, n)).cuda()
    h_rays, h_hits = torch.empty(n, 8).pin_memory().numpy(), torch.empty(n, 2, dtype=torch.int32).pin_memory().numpy()
    h_rays[:] = rays.cpu().numpy()
    ref = trace(dbvh, rays)
    late, early = torch.cuda.Stream(), torch.cuda.Stream()
    waiting = torch.full((n, 2), -7, dtype=torch.int32, device="cuda")
    others = [torch.full((n, 2), -7, dtype=torch.int32, device="cuda") for _ in range(7)]
    for _ in range(5):
        trace(dbvh, rays)
    torch.cuda.synchronize()
    with torch.cuda.stream(late):
        torch.cuda._sleep(400_000_000)  # a fifth of a second
    dbvh.intersect(rays, waiting, stream=late.cuda_stream)
    for h in others:
        dbvh.intersect(rays, h, stream=early.cuda_stream)
    early.synchronize()
    h_hits[:] = -7
    dbvh.intersect_host(h_rays, h_hits, stream=early.cuda_stream)
    assert not late.query()  # (else the call came first and shows nothing)
    for h in others:
        assert np.array_equal(h.cpu().numpy(), ref)
    assert np.array_equal(h_hits, ref)
    late.synchronize()
    assert np.array_equal(waiting.cpu().numpy(), ref)
    dbvh.check()


@pytest.mark.parametrize("at", [0, 24])
@pytest.mark.parametrize("n", [100, 300000])
def test_host_hits_over_the_rays(n, at):
    """Hits written where the (page-locked) rays are, from their first byte or from the fourth part on: every ray is
    read before the first hit is written."""
    bvh, extent = tree("spheres")
    dbvh = DeviceBVH(bvh)
    rays = rays_for(extent, 9, n)
    ref = trace(dbvh, torch.from_numpy(rays).cuda())
    buf = torch.empty(8 * n).pin_memory().numpy()
    h_rays = buf.reshape(n, 8)
    h_rays[:] = rays
    first = at * n // 4 // 2 * 2
    h_hits = buf[first:first + 2 * n].view(np.int32).reshape(n, 2)
    dbvh.intersect_host(h_rays, h_hits)
    assert np.array_equal(h_hits, ref)


def test_upload_after_a_refused_call():
    """A call that fails leaves its error behind in the thread; the next upload is none of its business."""
    bvh, extent = tree("spheres")
    dbvh = DeviceBVH(bvh)
    n, runtime = 1000, torch.cuda.cudart()
    room = np.empty(8 * n + 2048, np.float32)
    h_rays = room[-room.ctypes.data % 4096 // 4:][:8 * n].reshape(n, 8)
    h_rays[:] = rays_for(extent, 12, n)
    h_hits = np.empty((n, 2), np.int32)
    assert int(runtime.cudaHostRegister(h_rays.ctypes.data, 16384, 0)) == 0
    try:
        with pytest.raises(TTError):  # half of the rays page-locked: no valid range to copy
            dbvh.intersect_host(h_rays, h_hits)
        again = DeviceBVH(bvh)
    finally:
        runtime.cudaHostUnregister(h_rays.ctypes.data)
    rays = torch.from_numpy(h_rays.copy()).cuda()
    assert np.array_equal(trace(again, rays), trace(dbvh, rays))


def test_host_rays_in_two_registrations():
    """Rays that span two page-locked registrations next to each other are traced; with one of the two gone, the call
    is refused (a copy of such a range is no valid one) and writes no hits."""
    bvh, extent = tree("spheres")
    dbvh = DeviceBVH(bvh)
    n = 100000
    room = np.empty(8 * n + 2048, np.float32)
    h_rays = room[-room.ctypes.data % 4096 // 4:][:8 * n].reshape(n, 8)
    h_rays[:] = rays_for(extent, 12, n)
    h_hits = torch.empty(n, 2, dtype=torch.int32).pin_memory().numpy()
    ref = trace(dbvh, torch.from_numpy(h_rays.copy()).cuda())
    first, half, runtime = h_rays.ctypes.data, 16 * n // 4096 * 4096, torch.cuda.cudart()
    assert int(runtime.cudaHostRegister(first, half, 0)) == 0
    try:
        assert int(runtime.cudaHostRegister(first + half, 32 * n - half, 0)) == 0
        h_hits[:] = -7
        try:
            dbvh.intersect_host(h_rays, h_hits)
        finally:
            runtime.cudaHostUnregister(first + half)
        assert np.array_equal(h_hits, ref)
        h_hits[:] = -7
        with pytest.raises(TTError):
            dbvh.intersect_host(h_rays, h_hits)
        assert (h_hits == -7).all()
    finally:
        runtime.cudaHostUnregister(first)
    dbvh.intersect_host(h_rays, h_hits)
    assert np.array_equal(h_hits, ref)


@pytest.mark.parametrize("share", [0.0, 0.01, 0.05, 0.5, 1.0])
@pytest.mark.parametrize("closest", [True, False])
def test_coherent_sets_with_rays_that_the_four_wide_loop_does_not_serve(share, closest):
    """Camera rays of which some start at a negative tmin: the probe sends a set with too many of them to the two-wide
    loop as a whole, and its decision must not outlast the call."""
    sc, alpha, leaf, _ = SCENES["spheres"]()
    dbvh = DeviceBVH(BVHCompact.build(sc, alpha, 1, leaf))
    side = 1100
    rays = torch.from_numpy(scenes.pinhole_rays(side, side, [0.0, 14.0, 34.0], [0.0, 2.0, 0.0], 0.45)).cuda()
    g = torch.Generator("cuda").manual_seed(3)
    rays[torch.rand(side * side, generator=g, device="cuda") < share, 6] = -1e-3
    dbvh.set_variant(DeviceBVH.VARIANT_DYNAMIC)
    ref = trace(dbvh, rays, closest)
    plain = rays.clone()
    plain[:, 6] = 1e-3
    ref_plain = trace(dbvh, plain, closest)
    for variant in (DeviceBVH.VARIANT_SORTED, DeviceBVH.VARIANT_SORTED_OCC):
        dbvh.set_variant(variant)
        assert np.array_equal(trace(dbvh, rays, closest), ref)
        assert np.array_equal(trace(dbvh, plain, closest), ref_plain)
        assert np.array_equal(trace(dbvh, rays[:40001].contiguous(), closest), ref[:40001])


def without_a_four_wide_form(bvh, path):
    """The same tree with one box plane of its last node far away: its two-wide hits are the same (the box only grows),
    and it has no four-wide form."""
    def grow(nodes):
        nodes.view(F)[-4, 1] = 1e15
        return nodes
    return edited(bvh, path, grow)


@pytest.mark.parametrize("streamed", [0, 1])
@pytest.mark.parametrize("shape", [(64, 0), (128, 8), (256, 16)])
def test_renders_on_a_tree_without_a_four_wide_form(tmp_path, shape, streamed):
    """Extension and shadow queues of a tree that stays two-wide, at every stack depth: the image of the four-wide
    tree."""
    sc = Scene.from_mesh(scenes.multi_material(6, 3))
    sc.set_env(scenes.sky_env(64, 32, sun_radiance=5e2, sun_diameter_deg=10.0))
    sc.set_geometries([{"type": "Sphere", "position": [0.0, 3.0, 9.0], "radius": 2.0, "material": 0}])
    bvh = BVHCompact.build(sc, 1e-5, 1, 8)
    images = []
    for b in (bvh, without_a_four_wide_form(bvh, tmp_path / "bvh.cache")):
        r = Renderer(DeviceBVH(b), sc)
        r.set_launch(*shape, 3001, 1, streamed)
        acc = torch.zeros(3 * 97 * 61, device="cuda")
        cam = make_camera_meta(97, 61, [0.0, 14.0, 34.0], [0.0, -12.0, -34.0], fov=(60.0, 40.0))
        r.render_native(cam, render_params(spp=3, max_depth=6, rr_depth=3, seed=3), acc)
        r.check()
        images.append(acc.cpu().numpy())
    assert images[0].any() and np.array_equal(*(i.view(np.uint32) for i in images))


@pytest.mark.parametrize("w,h,samples", [(16, 16, 1), (200, 133, 3)])
def test_compat_frames_on_a_tree_without_a_four_wide_form(tmp_path, w, h, samples):
    sc = Scene.from_mesh(scenes.cornell(3))
    sc.set_env(np.ones((8, 16, 3), F))
    bvh = BVHCompact.build(sc, 1e-5, 1, 8)
    images = []
    for b in (bvh, without_a_four_wide_form(bvh, tmp_path / "bvh.cache")):
        r = Renderer(DeviceBVH(b), sc)
        acc = torch.zeros(3 * w * h, device="cuda")
        cam = make_camera_meta(w, h, [0.0, 0.0, 1.55], [0.0, 0.0, -1.0], fov=(45.0, 45.0))
        r.render_compat(cam, render_meta(7, samples), acc)
        r.check()
        images.append(acc.cpu().numpy())
    assert images[0].any() and np.array_equal(*(i.view(np.uint32) for i in images))
