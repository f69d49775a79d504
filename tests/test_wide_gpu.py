"""The four-wide traversal on the GPU (trees converted by tt_bvh_upload) against the two-wide tree of variant 3,
bit for bit, over small and odd ray counts and rays with special values in every field."""
import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for, soup
from trenchanttracer_gb300 import BVHCompact, DeviceBVH, Scene

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
