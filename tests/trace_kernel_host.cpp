// Host build of the trace kernels (trenchanttracer_gb300/csrc/tt_trace.cu) on the warps of warp_host.h.
#include "warp_host.h"

#define fmaxf dev_max
#define fminf dev_min
#include "tt_trace.cu"

using namespace tt;

template <bool kClosest>
static void trace(int kernel, unsigned blocks, const TraceArgs &a) {
    warp_host::run(blocks, [&] {
        if (kernel == 0) trace_wide_kernel<kClosest, false, 8, true, 8>(a);
        else if (kernel == 1) trace_wide_kernel<kClosest, false, 0, false, 1>(a);
        else if (kernel == 2) trace_wide_kernel<kClosest, false, 8, false, 8, true>(a);
        else if (kernel == 3) trace_warp_kernel<kClosest, false, false, 16, true>(a);
        else trace_dynamic_kernel<kClosest, false, 16>(a);
    });
}

extern "C" {
// Traces n rays by a kernel (0: the default, 1: without shared stack, 2: over host rays, 3: two-wide in the
// default's place, 4: two-wide with per-lane claims) in a grid of `blocks` warps, over a two-wide tree and,
// unless wide_nodes is null, its four-wide form. order: the ray in each place, or null. share: the places dealt
// to each warp (0: claimed from a counter). decision: of the ordering's probe (1 with an order, 2: two-wide).
// Returns the error word.
__attribute__((visibility("default"))) unsigned trace_kernel_host(
    int kernel, unsigned blocks, const float *nodes, const float *verts, const int *tri_idx, const char *wide_nodes,
    const char *wide_pairs, unsigned wide_flags, const float *rays, long long n, int closest, const int *order, unsigned share,
    int decision, int *hits) {
    unsigned err = 0;
    unsigned long long counter = 0, state[5] = {0, 0, 0, (unsigned long long)decision, 0};
    TraceArgs a{};
    a.bvh.nodes = reinterpret_cast<const float4 *>(nodes);
    a.bvh.verts = reinterpret_cast<const float4 *>(verts);
    a.bvh.tri_idx = tri_idx;
    a.bvh.wide_nodes = wide_nodes;
    a.bvh.wide_pairs = wide_pairs;
    a.bvh.wide_flags = wide_flags;
    a.rays = reinterpret_cast<const float4 *>(rays);
    a.n = n;
    a.hits = hits;
    a.counter = &counter;
    a.share = share;
    a.err = &err;
    a.order_src = order;
    a.order_state = decision ? state : nullptr;
    if (closest) trace<true>(kernel, blocks, a);
    else trace<false>(kernel, blocks, a);
    return err;
}
}
