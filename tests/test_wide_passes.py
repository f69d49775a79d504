"""The device passes that make the four-wide tree at upload, run on the CPU (tests/wide_passes_host.cpp): what they make
of a tree gives the two-wide traversal's hits, and trees they must leave two-wide are refused before a pass that
relies on what they lack."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for, soup
from trenchanttracer_gb300 import BVHCompact, build

ROOT = Path(__file__).resolve().parents[1]
F = np.float32


def host_library(tmp_path_factory, source, *flags):
    so = tmp_path_factory.mktemp("host") / (source + ".so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", *flags, f"-I{ROOT / 'tests'}",
                    f"-I{ROOT / 'trenchanttracer_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    f"-I{build._cuda_home() / 'include'}", str(ROOT / "tests" / source), "-o", str(so)], check=True)
    return C.CDLL(str(so))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = host_library(tmp_path_factory, "wide_passes_host.cpp")
    lib.wide_passes_trace.restype = C.c_longlong
    return lib


def convert(lib, arrays, rays, closest=1, two_wide=0, top=50):
    """(wide nodes, stage of refusal, hit slots, t u v as words, error word)"""
    n = rays.shape[0]
    addr, tuv = np.empty(n, np.int32), np.empty((n, 3), F)
    err, stage = C.c_uint(0), C.c_int(0)
    p = lambda a: C.c_void_p(a.ctypes.data)
    nodes, verts = np.ascontiguousarray(arrays["nodes"]), np.ascontiguousarray(arrays["vertices"])
    wide = lib.wide_passes_trace(p(nodes), C.c_longlong(len(nodes)), p(verts), C.c_longlong(len(verts)),
                                 C.c_longlong(top), p(rays), C.c_longlong(n), C.c_int(closest), C.c_int(two_wide),
                                 p(addr), p(tuv), C.byref(err), C.byref(stage))
    return wide, stage.value, addr, tuv.view(np.uint32), err.value


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("top", [1, 50, 1 << 20])
def test_converted_trees_give_the_two_wide_hits(host, name, top):
    sc, alpha, leaf, extent = SCENES[name]()
    arrays = BVHCompact.build(sc, alpha, 1, leaf).arrays()
    rays = rays_for(extent, 17, 5000)
    for closest in (1, 0):
        wide, stage, *got = convert(host, arrays, rays, closest, 0, top)
        *_, a, b, c = convert(host, arrays, rays, closest, 1)
        assert wide > 0 and stage == 0
        assert np.array_equal(got[0], a) and np.array_equal(got[1], b) and got[2] == c


def with_node(arrays, left, right):
    """The tree with one node more, that no other node refers to."""
    out = {k: v.copy() for k, v in arrays.items()}
    node = out["nodes"][-4:].copy()
    node[3, 0], node[3, 1] = left, right
    out["nodes"] = np.concatenate([out["nodes"], node])
    return out


def test_trees_with_a_node_that_no_node_refers_to_stay_two_wide(host):
    """Alone, with leaves or with one more such node below it: the passes that follow a node's links to the root
    must not run."""
    rays = rays_for(3.0, 5, 2000)
    base = BVHCompact.build(soup(60, 7, 0.5, 2.0), 1e-5, 1, 1).arrays()
    leaf = int(base["nodes"][-1, 0]) if base["nodes"][-1, 0] < 0 else ~0
    n = len(base["nodes"])
    two = BVHCompact.build(soup(2, 4, 1.0, 3.0), 1e-5, 1, 1).arrays()  # one inner node
    small = with_node(two, int(two["nodes"][3, 0]), int(two["nodes"][3, 1]))
    alone = with_node(base, leaf, leaf)
    over_a_leaf_node = with_node(alone, n, leaf)          # refers to the node that `alone` added
    ring = with_node(base, n, leaf)                       # refers to itself
    for arrays in (small, alone, over_a_leaf_node, ring):
        wide, stage, *got = convert(host, arrays, rays)
        assert wide == 0 and stage in (1, 2)
        *_, a, b, c = convert(host, arrays, rays, 1, 1)
        assert np.array_equal(got[0], a) and np.array_equal(got[1], b) and got[2] == c


def run_of(triangles, g):
    """`triangles` triangles behind one another and the terminator, as vertex words."""
    v = np.zeros((3 * triangles + 1, 4), np.int32)
    v[:-1, :3] = g.normal(size=(3 * triangles, 3)).astype(F).view(np.int32)
    v[-1, 0] = -2**31
    return v


@pytest.mark.parametrize("leaves,triangles", [(2, 1), (2, 40), (300, 2000)])
def test_trees_whose_leaves_overlap_stay_two_wide(host, leaves, triangles):
    """Leaf addresses of a file may point into one another's triangles. A pass that walked each from its address to
    its end would take leaves times triangles steps, so the first triangle met twice ends it."""
    g = np.random.default_rng(3)
    base = BVHCompact.build(soup(leaves, 7, 0.5, 2.0), 1e-5, 1, 1).arrays()
    child = base["nodes"][3::4, :2]  # a view: the children's addresses
    at = np.arange((child < 0).sum(), dtype=np.int32)
    base["vertices"] = run_of(triangles, g)
    child[child < 0] = ~(3 * (at % triangles))
    base["nodes"] = base["nodes"].copy()
    rays = rays_for(3.0, 5, 200)
    wide, stage, *got = convert(host, base, rays)
    assert wide == 0 and stage == 3
    *_, a, b, c = convert(host, base, rays, 1, 1)
    assert np.array_equal(got[0], a) and np.array_equal(got[1], b) and got[2] == c


@pytest.mark.parametrize("triangles,accepted", [(8192, True), (8193, False)])
def test_a_leaf_of_very_many_triangles_stays_two_wide(host, triangles, accepted):
    """One thread walks a leaf, so its length is bounded."""
    g = np.random.default_rng(4)
    base = BVHCompact.build(soup(2, 4, 1.0, 3.0), 1e-5, 1, 1).arrays()
    base["vertices"] = np.concatenate([run_of(triangles, g), run_of(1, g)])
    base["nodes"][3, :2] = [~0, ~(3 * triangles + 1)]
    rays = rays_for(3.0, 5, 50)
    wide, stage, *got = convert(host, base, rays)
    assert (wide > 0 and stage == 0) if accepted else (wide == 0 and stage == 3)
    *_, a, b, c = convert(host, base, rays, 1, 1)
    assert np.array_equal(got[0], a) and np.array_equal(got[1], b) and got[2] == c


def test_the_walk_up_a_chain_of_nodes_is_bounded(host):
    """A file may hold one long chain of nodes, which one thread walks up. A tree that deep needs more stack than the
    four-wide loop has, so the walk ends where that is certain."""
    base = BVHCompact.build(soup(2, 4, 1.0, 3.0), 1e-5, 1, 1).arrays()
    n = 5000
    nodes = np.tile(base["nodes"][:4], (n, 1))
    lo, hi = F(-9.0), F(9.0)
    nodes.view(F)[0::4] = nodes.view(F)[1::4] = nodes.view(F)[2::4] = [lo, hi, lo, hi]
    leaf = int(base["nodes"][3, 0])
    nodes[3::4, 0] = leaf
    nodes[3::4, 1] = 4 * np.arange(1, n + 1)
    nodes[-1, 1] = int(base["nodes"][3, 1])
    verts = np.ascontiguousarray(base["vertices"])
    out, size, flags, done = (C.c_void_p * 2)(), (C.c_longlong * 2)(), C.c_uint(0), C.c_uint(0)
    host.wide_passes_form.restype = C.c_longlong
    wide = host.wide_passes_form(C.c_void_p(nodes.ctypes.data), C.c_longlong(len(nodes)), C.c_void_p(verts.ctypes.data),
                                 C.c_longlong(len(verts)), C.c_longlong(50), out, size, C.byref(flags), C.byref(done))
    assert wide == 0 and done.value <= 150
