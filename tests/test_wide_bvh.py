"""The four-wide traversal against the two-wide one, ray by ray and bit by bit, on the CPU: both loops of the
device headers built with plain C++ (tests/wide_host.cpp). Every form of ray the entry points take is among
the inputs: any origin, direction, tmin and tmax, finite or not."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from trenchanttracer_gb300 import BVHCompact, Scene, scenes

ROOT = Path(__file__).resolve().parents[1]
F = np.float32


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = tmp_path_factory.mktemp("wide") / "wide_host.so"
    csrc = ROOT / "trenchanttracer_gb300" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{csrc}",
                    f"-I{ROOT / 'include'}", str(ROOT / "tests" / "wide_host.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.wide_host_trace.restype = C.c_longlong
    return lib


def trace(lib, arrays, rays, closest, wide):
    n = rays.shape[0]
    addr, tuv = np.empty(n, np.int32), np.empty((n, 3), F)
    err, flags, regular = C.c_uint(0), C.c_uint(0), np.empty(n, np.int32)
    p = lambda a: C.c_void_p(a.ctypes.data)
    nodes, verts = np.ascontiguousarray(arrays["nodes"]), np.ascontiguousarray(arrays["vertices"])
    count = lib.wide_host_trace(p(nodes), C.c_longlong(len(nodes)), p(verts), C.c_longlong(len(verts)), p(rays),
                                C.c_longlong(n), C.c_int(closest), C.c_int(wide), p(addr), p(tuv), C.byref(err),
                                p(regular), C.byref(flags))
    return count, addr, tuv.view(np.uint32), err.value, regular, flags.value


def soup(n, seed, spread, extent):
    g = np.random.default_rng(seed)
    c = g.uniform(-extent, extent, (n, 1, 3))
    v = (c + g.normal(size=(n, 3, 3)) * spread).astype(F).reshape(-1, 3)
    return Scene.from_arrays(v, np.ones_like(v), np.arange(3 * n, dtype=np.int32).reshape(-1, 3))


def zero_planes(seed):
    """Axis-aligned quads in the planes at +0.0 and -0.0 and around them."""
    g = np.random.default_rng(seed)
    quads = []
    for k in range(60):
        axis = k % 3
        p = g.uniform(-1, 1, 3).astype(F)
        p[axis] = [F(0.0), F(-0.0), F(0.25), F(-0.5)][k % 4]
        a, b = np.zeros(3, F), np.zeros(3, F)
        a[(axis + 1) % 3], b[(axis + 2) % 3] = g.uniform(0.1, 0.6), g.uniform(0.1, 0.6)
        if k % 2:
            a, b = b, a
        q = np.stack([p, p + a, p + b])
        q[:, axis] = p[axis]
        quads.append(q)
    v = np.concatenate(quads).astype(F)
    return Scene.from_arrays(v, np.ones_like(v), np.arange(len(v), dtype=np.int32).reshape(-1, 3))


SCENES = {
    "terrain": lambda: (Scene.from_mesh(scenes.terrain(48, 8.0)), 1e-5, 8, 8.0),
    "spheres": lambda: (Scene.from_mesh(scenes.multi_material(8, 3)), 1e-5, 8, 20.0),
    "cornell": lambda: (Scene.from_mesh(scenes.cornell(2)), 1e-5, 4, 0.6),
    "splits": lambda: (soup(3000, 1, 0.5, 3.0), 1.0, 3, 4.0),
    "needles": lambda: (soup(400, 2, 8.0, 3.0), 1e-5, 1, 10.0),
    "zero_planes": lambda: (zero_planes(3), 1e-5, 1, 1.2),
    "one_leaf_each": lambda: (soup(2, 4, 1.0, 3.0), 1e-5, 1, 4.0),
}


def rays_for(extent, seed, n):
    """Ordinary rays, and rays with special values in every field."""
    g = np.random.default_rng(seed)
    r = np.empty((n, 8), F)
    r[:, 0:3] = g.uniform(-extent, extent, (n, 3))
    d = g.normal(size=(n, 3))
    r[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 6] = g.choice(np.array([0.0, 0.0, 1e-3, 0.01], F), n)
    r[:, 7] = g.choice(np.array([1e20, 1e20, np.inf, 1.0], F), n)
    odd = np.array([0.0, -0.0, 1e-30, -1e-30, 1.0, -1.0, 2e-24, 1e12, -3e11, 1e30, np.inf, -np.inf, np.nan], F)
    for col in range(8):
        pick = g.random(n) < (0.12 if col < 6 else 0.06)
        few = odd[:6] if col < 6 else np.concatenate([odd, np.array([-5.0, 0.5, 3e38], F)])
        vals = np.where(g.random(n) < 0.85, g.choice(few, n), g.choice(odd, n))
        r[pick, col] = vals[pick]
    return r


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("closest", [1, 0])
def test_four_wide_equals_two_wide(host, name, closest):
    sc, alpha, leaf, extent = SCENES[name]()
    arrays = BVHCompact.build(sc, alpha, 1, leaf).arrays()
    rays = rays_for(extent, 11, 60000)
    count, addr, tuv, err, regular, flags = trace(host, arrays, rays, closest, 1)
    _, ref_addr, ref_tuv, ref_err, _, _ = trace(host, arrays, rays, closest, 0)
    assert count > 0 and err == ref_err
    assert 0.4 < regular.mean() < 0.95  # both routes are taken
    assert np.array_equal(addr, ref_addr)
    assert np.array_equal(tuv, ref_tuv)
    assert (ref_addr[regular == 1] >= 0).any()
    assert name != "zero_planes" or flags & 1


def test_trees_without_a_four_wide_form(host):
    """A tree that shares a node, a box or vertex beyond the bounds and a tree as deep as the depth limit are
    traced two-wide, with the two-wide results."""
    rays = rays_for(3.0, 5, 4000)
    base = BVHCompact.build(soup(60, 7, 0.5, 2.0), 1e-5, 1, 1).arrays()
    shared = {k: v.copy() for k, v in base.items()}
    inner = np.nonzero(shared["nodes"][3::4, 0] >= 0)[0]
    shared["nodes"][4 * inner[1] + 3, 0] = shared["nodes"][4 * inner[0] + 3, 0]
    huge = {k: v.copy() for k, v in base.items()}
    huge["nodes"].view(F)[0, 1] = F(1e15)
    g = np.random.default_rng(1)
    tri = g.normal(size=(3, 3)).astype(F)
    stack = np.concatenate([tri] * 120)
    deep = BVHCompact.build(Scene.from_arrays(stack, np.ones_like(stack), np.arange(360, dtype=np.int32).reshape(-1, 3)),
                            1e-5, 1, 1).arrays()
    for arrays in (huge, deep):
        for closest in (1, 0):
            count, addr, tuv, err, _, _ = trace(host, arrays, rays, closest, 1)
            _, ref_addr, ref_tuv, ref_err, _, _ = trace(host, arrays, rays, closest, 0)
            assert count == 0 and err == ref_err
            assert np.array_equal(addr, ref_addr) and np.array_equal(tuv, ref_tuv)
    assert trace(host, shared, rays[:1], 1, 0)[0] == 0
