"""Calls at the edges of what the trace entry points accept, on the GPU: files whose tree is no plain tree, calls on
several streams, host buffers in unusual places."""
import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for
from trenchanttracer_gb300 import BVHCompact, DeviceBVH

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
