"""The trace kernels on the CPU, run on emulated warps (tests/warp_host.h): the queue loop that every kernel over the
four-wide tree uses, and what a kernel does with an order that holds anything."""
import ctypes as C

import numpy as np
import pytest

from tests.test_wide_bvh import SCENES, rays_for
from tests.test_wide_passes import host_library
from trenchanttracer_gb300 import BVHCompact

F = np.float32
ORDERED, LOCAL, HOST, TWO_WIDE, DYNAMIC = range(5)
ERR_ORDER = 4


class Tree:
    def __init__(self, passes, name):
        sc, alpha, leaf, self.extent = SCENES[name]()
        a = BVHCompact.build(sc, alpha, 1, leaf).arrays()
        self.nodes, self.verts = np.ascontiguousarray(a["nodes"]), np.ascontiguousarray(a["vertices"])
        self.tri = np.ascontiguousarray(a["tri_indices"])
        size, flags = (C.c_longlong * 2)(), C.c_uint(0)
        raw = (C.c_void_p * 2)()
        wide = passes.wide_passes_form(ptr(self.nodes), C.c_longlong(len(self.nodes)), ptr(self.verts),
                                       C.c_longlong(len(self.verts)), C.c_longlong(50), raw, size, C.byref(flags),
                                       C.byref(C.c_uint(0)))
        assert wide > 0
        # 32-byte aligned copies, as the kernels' loads want them
        self.wide = [aligned(np.frombuffer(C.string_at(raw[k], size[k]), np.uint8)) for k in (0, 1)]
        self.flags = flags.value


def ptr(a):
    return C.c_void_p(None if a is None else a.ctypes.data)


def aligned(a):
    buf = np.empty(a.nbytes + 32, np.uint8)
    at = -buf.ctypes.data % 32
    buf[at:at + a.nbytes] = a
    return buf[at:at + a.nbytes]


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    lib = host_library(tmp_path_factory, "trace_kernel_host.cpp", "-fvisibility=hidden", "-ffunction-sections",
                       "-fdata-sections", "-Wl,--gc-sections", "-Wl,--no-undefined", "-Wno-attributes")
    lib.trace_kernel_host.restype = C.c_uint
    passes = host_library(tmp_path_factory, "wide_passes_host.cpp")
    passes.wide_passes_form.restype = C.c_longlong
    return lib, passes


def trace(lib, tree, kernel, rays, closest, order=None, wide=True, blocks=2, spare=0, share=0, decision=0):
    """Hits of the first len(rays) - spare rays; the spare ones and their hits lie behind the buffers' ends."""
    n = rays.shape[0] - spare
    hits = np.full((rays.shape[0], 2), -7, np.int32)
    nodes, pairs = tree.wide if wide else (None, None)
    err = lib.trace_kernel_host(kernel, blocks, ptr(tree.nodes), ptr(tree.verts), ptr(tree.tri), ptr(nodes), ptr(pairs),
                                tree.flags if wide else 0, ptr(rays), C.c_longlong(n), int(closest), ptr(order),
                                C.c_uint(share), decision or int(order is not None), ptr(hits))
    return hits, err


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("closest", [1, 0])
def test_queue_kernels_give_the_two_wide_hits(kernels, name, closest):
    lib, passes = kernels
    tree = Tree(passes, name)
    rays = rays_for(tree.extent, 23, 1500)
    ref, err = trace(lib, tree, DYNAMIC, rays, closest)
    order = np.random.default_rng(1).permutation(len(rays)).astype(np.int32)
    assert err == 0 and not (ref[:, 0] == -7).any()
    for kernel, o, wide in ((ORDERED, None, True), (ORDERED, order, True), (ORDERED, order, False), (LOCAL, None, True),
                            (HOST, None, True), (TWO_WIDE, order, False)):
        got, err = trace(lib, tree, kernel, rays, closest, o, wide)
        assert err == 0 and np.array_equal(got, ref), (kernel, wide)
    for n in (1, 2, 31, 32, 33, 63, 65):
        got, err = trace(lib, tree, ORDERED, rays[:n], closest)
        assert err == 0 and np.array_equal(got, ref[:n]), n


@pytest.mark.parametrize("name", ["spheres", "zero_planes", "needles"])
def test_the_probe_may_send_a_set_to_the_two_wide_loop(kernels, name):
    """The default kernel over a set of which the probe found too many rays that the four-wide loop does not serve."""
    lib, passes = kernels
    tree = Tree(passes, name)
    for n in (1, 33, 1000):
        rays = rays_for(tree.extent, 37, n)
        for closest in (1, 0):
            ref, _ = trace(lib, tree, DYNAMIC, rays, closest)
            got, err = trace(lib, tree, ORDERED, rays, closest, decision=2)
            assert err == 0 and np.array_equal(got, ref), (n, closest)


@pytest.mark.parametrize("n,warps", [(1, 4), (3, 4), (4, 4), (5, 4), (13, 4), (16, 4), (253, 64), (256, 64)])
def test_shares_dealt_without_a_counter_cover_every_ray(kernels, n, warps):
    """Small sets: at most four rays to a warp, dealt out in ray order; the last warps may have fewer or none."""
    lib, passes = kernels
    tree = Tree(passes, "spheres")
    rays = rays_for(tree.extent, 31, n)
    for closest in (1, 0):
        ref, _ = trace(lib, tree, DYNAMIC, rays, closest)
        for kernel in (ORDERED, HOST):
            got, err = trace(lib, tree, kernel, rays, closest, blocks=warps, share=-(-n // warps))
            assert err == 0 and np.array_equal(got, ref), kernel


@pytest.mark.parametrize("kernel", [ORDERED, TWO_WIDE])
@pytest.mark.parametrize("beyond", ["just", "far"])
def test_an_order_with_slots_out_of_range_is_reported(kernels, kernel, beyond):
    """Two overlapping calls share the ordering's scratch, so a place of the order can hold anything: no ray or hit
    beyond the caller's buffers is touched, the error word says so, and the other rays' hits are right."""
    lib, passes = kernels
    tree = Tree(passes, "spheres")
    n, spare = 700, 200
    rays = rays_for(tree.extent, 29, n + spare)
    ref, _ = trace(lib, tree, DYNAMIC, rays[:n], 1)
    order = np.random.default_rng(2).permutation(n).astype(np.int32)
    lost = order[::7].copy()
    bad = np.array([n, n + 1, n + spare - 1] if beyond == "just" else [-1, -2**31, 2**31 - 1, n + spare], np.int32)
    order[::7] = np.resize(bad, len(lost))
    got, err = trace(lib, tree, kernel, rays, 1, order, kernel == ORDERED, spare=spare)
    assert (got[n:] == -7).all() and err & ERR_ORDER
    kept = np.setdiff1d(np.arange(n), lost)
    assert np.array_equal(got[kept], ref[kept])
    unwritten = (got[lost] == -7).all(axis=1)
    assert np.array_equal(got[lost][~unwritten], ref[lost][~unwritten])
