// Traversal stages of the native wavefront path tracer: closest hit of every queued path
// (extend) and any hit of every queued shadow ray (shadow).
//
// Both are persistent grids in which each warp claims consecutive queue slots, as many as it has
// finished rays, and traces them with the per-ray traversal of tt_wide.cuh, so the result of a ray never
// depends on the other rays of its warp. Each is built for every block size and shared-memory
// stack depth in kBlockShapes x kStackShapes; the renderer's autotuner picks one.
#include <cuda_runtime.h>

#include "tt_launch.cuh"
#include "tt_native.cuh"
#include "tt_wide.cuh"

namespace tt {

using namespace pt;

// trace_queue's lanes at inner nodes below which a warp turns to leaves and new rays: the Cornell box at
// 512 x 512 x 16 takes 3.39 ms with 8, 3.33 with 10, 3.30 with 12; 12 views of a terrain 2.59, 2.58 and 2.65.
constexpr int kQueueInner = 10;

// Compiled for 1,024 threads per SM (64 registers): with both loops in the kernel the compiler takes 70, which
// leaves one block less (the Cornell box 3.35 ms instead of 3.24 with another way to hold both loops). A tree without a four-wide form goes through
// two_wide_queue: tracing each ray where trace_queue meets it, the box took 6.91 ms, so 5.35.
// kPrefix: the ordering covers only the queue's first *n_sorted slots (a streamed render's
// survivors); the rest is traced in place. Without it an ordered queue is ordered whole.
template <int kBlock, int kSh, bool kPrefix>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) k_extend(NativeArgs a, int cur) {
    chain_begin();
    __shared__ uint2 sh_stack[(kSh > 0 ? kSh : 1) * kBlock];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.ps.counts[cur ^ 1] = 0;
        a.ps.counts[2] = 0;
        a.ps.counts[4] = 0;
    }
    const int n = a.ps.counts[cur];
    const int lane = threadIdx.x & 31;
    WideStackOf<kSh, kBlock, true> stack;
    stack.sh = sh_stack + threadIdx.x;
    WideRays<0> rays;
    uint32_t err = 0;
    // an ordered queue prefix: hits by place, moved back by k_order_gather_hits
    const bool ordered = a.order.src && order_built(a.order.state);
    const int n_sorted = ordered ? (kPrefix ? *a.order.n_sorted : n) : 0;
    const auto claim = [&](bool, unsigned &count) {
        int base = 0;
        if (lane == 0) base = atomicAdd(a.ps.counts + 3, (int)count);
        return (unsigned)__shfl_sync(0xffffffffu, base, 0);
    };
    const auto at = [&](unsigned place) {
        const bool srt = kPrefix ? (int)place < n_sorted : ordered;
        return srt ? ordered_slot(a.order.src, place, (unsigned)n_sorted, err) : place;
    };
    const auto fetch = [&](unsigned q, float4 &r0, float4 &r1) {
        r0 = a.ps.ray[cur][2 * (size_t)q];
        r1 = a.ps.ray[cur][2 * (size_t)q + 1];
    };
    const auto store = [&](unsigned lanes, unsigned q, const TraceResult &tr) {
        float t = tr.t, hu = tr.u, hv = tr.v;
        int prim = tr.addr;
        if (a.num_geoms) {
            const float4 r0 = a.ps.ray[cur][2 * (size_t)q], r1 = a.ps.ray[cur][2 * (size_t)q + 1];
            analytic_hit(a, lanes, true, V3(r0.x, r0.y, r0.z), V3(r0.w, r1.x, r1.y), r1.z, t, prim, hu, hv, false);
        }
        const float4 h = make_float4(t, hu, hv, __int_as_float(prim));
        if (kPrefix ? (int)q < n_sorted : ordered) {
            const int p = a.order.pos[q];
            // (k_order_gather_hits lets a path whose place is out of range miss)
            if ((unsigned)p < (unsigned)n_sorted) a.order.hits[p] = h;
            else err |= kErrOrder;
        } else {
            a.ps.hit[q] = h;
        }
    };
    if (a.bvh.wide_nodes)
        trace_queue<true, kQueueInner>(stack, rays, a.bvh, (unsigned)n, err, claim, at, fetch, store);
    else
        two_wide_queue<true, 2 * kSh, kBlock>(reinterpret_cast<int *>(sh_stack) + threadIdx.x, a.bvh, (unsigned)n, err,
                                              claim, at, fetch, store);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.stats + 0, (unsigned long long)n);
    if (err) atomicOr(a.err, err);
}

template <int kBlock, int kSh>
__global__ void __launch_bounds__(kBlock, 1024 / kBlock) k_shadow(NativeArgs a) {
    chain_begin();
    __shared__ uint32_t sh_stack[(kSh > 0 ? kSh : 1) * kBlock];
    if (blockIdx.x == 0 && threadIdx.x == 0) a.ps.counts[3] = 0;  // the next extend's work counter
    const int n = a.ps.counts[2];
    const int lane = threadIdx.x & 31;
    WideStackOf<kSh, kBlock, false> stack;
    stack.sh = sh_stack + threadIdx.x;
    WideRays<0> rays;
    uint32_t err = 0;
    const bool ordered = a.shadow_order.src && order_built(a.shadow_order.state);
    const auto claim = [&](bool, unsigned &count) {
        int base = 0;
        if (lane == 0) base = atomicAdd(a.ps.counts + 4, (int)count);
        return (unsigned)__shfl_sync(0xffffffffu, base, 0);
    };
    const auto at = [&](unsigned place) {
        return ordered ? ordered_slot(a.shadow_order.src, place, (unsigned)n, err) : place;
    };
    const auto fetch = [&](unsigned j, float4 &r0, float4 &r1) {
        r0 = a.ps.shadow_ray[2 * (size_t)j];
        r1 = a.ps.shadow_ray[2 * (size_t)j + 1];
    };
    const auto store = [&](unsigned lanes, unsigned j, const TraceResult &tr) {
        bool blocked = tr.addr >= 0;
        if (a.num_geoms) {
            const float4 r0 = a.ps.shadow_ray[2 * (size_t)j], r1 = a.ps.shadow_ray[2 * (size_t)j + 1];
            float t = r1.w, hu, hv;
            int prim = -1;
            analytic_hit(a, lanes, !blocked, V3(r0.x, r0.y, r0.z), V3(r0.w, r1.x, r1.y), r1.z, t, prim, hu, hv,
                         true);
            blocked = blocked || prim != -1;
        }
        if (!blocked) {
            // a path's radiance: state slot t for t >= 0, else (an ended path of a streamed
            // render) ring entry -1 - t
            const int t = a.ps.shadow_path[j];
            const float *c = a.ps.shadow_val + 3ll * j;
            if (t >= 0) {
                float4 L = a.ps.lf[t];
                L.x = PT_ADD(L.x, c[0]);
                L.y = PT_ADD(L.y, c[1]);
                L.z = PT_ADD(L.z, c[2]);
                a.ps.lf[t] = L;
            } else {
                float *L = a.stream.ring + 3ll * (-1ll - t);
                L[0] = PT_ADD(L[0], c[0]);
                L[1] = PT_ADD(L[1], c[1]);
                L[2] = PT_ADD(L[2], c[2]);
            }
        }
    };
    if (a.bvh.wide_nodes)
        trace_queue<false, kQueueInner>(stack, rays, a.bvh, (unsigned)n, err, claim, at, fetch, store);
    else
        two_wide_queue<false, kSh, kBlock>(reinterpret_cast<int *>(sh_stack) + threadIdx.x, a.bvh, (unsigned)n, err, claim,
                                           at, fetch, store);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.stats + 1, (unsigned long long)n);
    if (err) atomicOr(a.err, err);
}

__global__ void __launch_bounds__(256) k_order_gather_hits(NativeArgs a, int cur) {
    chain_begin();
    if (!a.order.src || !order_built(a.order.state)) return;
    const int n = *a.order.n_sorted;
    unsigned bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = __ldcs(a.order.pos + i);
        if ((unsigned)p < (unsigned)n) {
            a.ps.hit[i] = a.order.hits[p];
        } else {  // not reachable with a consistent ordering: report, and let the path miss
            a.ps.hit[i] = make_float4(1e20f, 0.0f, 0.0f, __int_as_float(-1));
            bad = 1;
        }
    }
    if (bad) atomicOr(a.err, kErrOrder);
}

template <int kBlock, int kSh>
static TraceKernels kernels_of() {
    TraceKernels k;
    k.extend = k_extend<kBlock, kSh, false>;
    k.extend_prefix = k_extend<kBlock, kSh, true>;
    k.shadow = k_shadow<kBlock, kSh>;
    return k;
}

template <int kBlock>
static TraceKernels kernels_of_block(int sh) {
    switch (sh) {
        case 0: return kernels_of<kBlock, 0>();
        case 8: return kernels_of<kBlock, 8>();
        case 16: return kernels_of<kBlock, 16>();
        default: return TraceKernels{nullptr, nullptr, nullptr};
    }
}

TraceKernels trace_kernels(int block, int stack_shared) {
    switch (block) {
        case 64: return kernels_of_block<64>(stack_shared);
        case 128: return kernels_of_block<128>(stack_shared);
        case 256: return kernels_of_block<256>(stack_shared);
        default: return TraceKernels{nullptr, nullptr, nullptr};
    }
}

}  // namespace tt
