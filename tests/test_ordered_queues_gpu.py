"""Renders whose extension and shadow queues are long enough to be ordered (2^22 rays): a room that few paths leave. The
orders are taken through an index, hits by place and back, so every image is that of the unordered queues."""
import numpy as np
import pytest

from trenchanttracer_gb300 import BVHCompact, DeviceBVH, Renderer, Scene, make_camera_meta, render_params, scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = np.float32
ORDERED_FROM = 1 << 22


def room():
    """Six inward walls about the origin, the ceiling with a window of a tenth of its area, and a bumpy ball. Every
    surface reflects and glows in a colour of its own."""
    quads, lo, hi = [], -2.0, 2.0
    corner = lambda k: np.array([[lo, hi][k & 1], [lo, hi][k >> 1 & 1], [lo, hi][k >> 2 & 1]])
    for q in ((0, 4, 5, 1), (0, 1, 3, 2), (4, 6, 7, 5), (0, 2, 6, 4), (1, 5, 7, 3)):  # all but the ceiling
        quads.append([corner(k) for k in q])
    w = 0.6  # half a window's side
    for x0, x1, z0, z1 in ((lo, hi, lo, -w), (lo, hi, w, hi), (lo, -w, -w, w), (w, hi, -w, w)):
        quads.append([np.array([x, hi, z]) for x, z in ((x0, z0), (x1, z0), (x1, z1), (x0, z1))])
    v, n, tri, mat = [], [], [], []
    for k, q in enumerate(quads):
        for t in ((0, 1, 2), (0, 2, 3)):
            p = [q[i] for i in t]
            nrm = np.cross(p[1] - p[0], p[2] - p[0])
            if nrm @ p[0] > 0:  # towards the origin
                p, nrm = [p[0], p[2], p[1]], -nrm
            tri.append(range(len(v), len(v) + 3))
            v += p
            n += [nrm / np.linalg.norm(nrm)] * 3
            mat.append(min(k, 5))
    bv, bt, bn = scenes.displaced_icosphere(4, 0.7, [0.3, -0.9, -0.2], 5, 0.1)
    tri = np.concatenate([np.array([list(t) for t in tri], np.int32), np.asarray(bt, np.int32) + len(v)])
    mat = np.array(mat + [6] * len(bt), np.uint32)
    g = np.random.default_rng(1)
    materials = [{"name": f"m{k}", "type": "Diff", "diffuseColor": list(g.uniform(0.4, 0.9, 3)),
                  "emission": list(g.uniform(0.0, 0.5, 3))} for k in range(7)]
    sc = Scene.from_arrays(np.concatenate([v, bv]).astype(F), np.concatenate([n, bn]).astype(F), tri, mat=mat)
    sc.set_materials(materials)
    sc.set_env(np.full((8, 16, 3), 3.0, F))
    return sc


@pytest.mark.parametrize("streamed", [0, 1])
def test_ordered_queues_give_the_unordered_image(streamed):
    sc = room()
    r = Renderer(DeviceBVH(BVHCompact.build(sc, 1e-5, 1, 8)), sc)
    w, h, depth = 4096, 2560, 4
    pool = 9 << 20 if streamed else 1 << 24
    cam = make_camera_meta(w, h, [-1.0, 0.4, 1.5], [0.5, -0.3, -1.0], fov=(80.0, 55.0))
    params = render_params(spp=1, max_depth=depth, rr_depth=99, seed=4)
    images = []
    for ordered in (0, 1):
        r.set_launch(128, 8, pool, ordered, streamed)
        acc = torch.zeros(3 * w * h, device="cuda")
        r.stats(reset=True)
        r.render_native(cam, params, acc)
        r.check()
        images.append(acc.view(torch.int32))
        s = r.stats()
    assert s["paths"] == w * h
    # rays that leave the room, and those that end at the depth, are all that a queue loses
    if not streamed:  # the last extension queue; the longest shadow queue
        assert s["extension_rays"] - (depth - 1) * w * h >= ORDERED_FROM
        assert s["shadow_rays"] / depth >= ORDERED_FROM
    else:  # the first queues hold the pool and its survivors
        assert s["extension_rays"] / (w * h * depth) * pool >= ORDERED_FROM
        assert s["shadow_rays"] / (w * h * depth) * pool >= ORDERED_FROM
    assert acc.any() and torch.equal(*images)
