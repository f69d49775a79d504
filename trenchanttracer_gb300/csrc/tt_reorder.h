// Ray ordering before traversal (tt_reorder.cu); internal to libtt.so.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <cstdint>

#include "../../include/tt.h"

namespace tt {

// the origin's cell (up to 13 bits: Morton-like code of a grid over the scene bounds whose bits go
// to the longest remaining cell side first; fewer bits for fewer rays, about 2^(origin bits + 9)
// rays each) above the direction's cell (8 bits: 16 x 16 octahedral grid)
constexpr int kOrderDirBits = 8;
constexpr int kOrderOriginBits = 13;
constexpr int kOrderMinOriginBits = 6;
constexpr int kOrderBits = kOrderDirBits + kOrderOriginBits;  // the largest key
static_assert(kOrderDirBits % 2 == 0 && kOrderBits <= 21, "direction cells square; counts for 2^21 keys at most");
// Fewer rays than this are traced in their own order. One line for closest and any hit, between the counts where
// ordering starts to pay for either: at 1M it still costs cosine bounces up to 7 % or gains 3 %, and gains
// shadow rays 3 to 8 %. Measured on hashed cosine bounces and shadow rays, ordered against not, in us: on a
// 2,097,152-triangle terrain 287 / 269 at 1M, 451 / 457 at 2M, 790 / 835 at 4M (shadow rays 371 / 382
// and 1,166 / 1,310 at 1M and 4M); on 400 spheres of 5,120 triangles 201 / 179 at 300K, 395 / 407 at 1M,
// 1,215 / 1,398 at 4M (shadow rays 342 / 370 and 1,092 / 1,284).
constexpr int64_t kOrderMinRays = 1 << 20;
// The same for the queues of a render. They follow the image, so neighbours start close together
// and go less far astray: with queues from 1M rays on ordered, 12 uneven views of a terrain (4M-slot
// pool, whose queues never reach 4M) take 3.35 ms, from 2M on 2.88, with none 2.65; 960 x 540 x 16 samples of 400
// spheres 15.5, 15.2 and 15.2 ms. Above the line it depends on the scene: in pools of 16M and 64M slots the
// 8.2M-triangle multi-material view takes 164.8 and 163.7 ms unordered, 161.5 and 159.9 ordered, 16 views of
// the terrain from 16M slots 32.7 unordered, 35.0 ordered. In a pool that cannot reach the line `ordered` only costs
// its passes' launches (4M slots: 178.5 ms unordered, 185.0 ordered).
constexpr int64_t kOrderMinQueue = 1 << 22;
// Error-word bit: a slot of the order came out of range (see ordered_slot, and k_order_scatter).
constexpr uint32_t kErrOrder = 4u;

// The origin grid: q_k = clamp((o_k - lo_k) * scale_k, 0, cells_k - 1), and bit j of q_k goes to
// the j-th lowest set bit of mask_k in the origin code.
struct OrderGrid {
    float3 lo, scale, qmax;
    unsigned mask[3];
    int origin_bits;
};

__host__ __device__ inline unsigned deposit(unsigned q, unsigned mask) {
    unsigned r = 0;
    for (unsigned m = mask; m; m &= m - 1u) {
        if (q & 1u) r |= m & (0u - m);
        q >>= 1;
    }
    return r;
}

__host__ __device__ inline unsigned order_key(const float4 r0, const float4 r1, const OrderGrid &g) {
    // direction: octahedral map (x, z over |x| + |y| + |z|, the lower hemisphere folded out),
    // kOrderDirBits / 2 bits per map axis, interleaved; non-finite or zero directions go to cell 0
    const float dx = r0.w, dy = r1.x, dz = r1.y;
    const float s = fabsf(dx) + fabsf(dy) + fabsf(dz);
    unsigned dcell = 0;
    if (s > 0.0f && s < INFINITY) {
        float u = dx / s, v = dz / s;
        if (dy < 0.0f) {
            const float fu = (1.0f - fabsf(v)) * (u < 0.0f ? -1.0f : 1.0f);
            v = (1.0f - fabsf(u)) * (v < 0.0f ? -1.0f : 1.0f);
            u = fu;
        }
        constexpr float kCells = (float)(1 << (kOrderDirBits / 2));  // per map axis
        constexpr unsigned kMask = (1u << kOrderDirBits) - 1u;
        const unsigned qu = (unsigned)fminf(fmaxf((u + 1.0f) * (0.5f * kCells), 0.0f), kCells - 1.0f);
        const unsigned qv = (unsigned)fminf(fmaxf((v + 1.0f) * (0.5f * kCells), 0.0f), kCells - 1.0f);
        dcell = deposit(qu, 0xAAAAAAAAu & kMask) | deposit(qv, 0x55555555u & kMask);
    }
    // origin (NaN coordinates clamp to cell 0: fmaxf returns the non-NaN operand)
    const unsigned qx = (unsigned)fminf(fmaxf((r0.x - g.lo.x) * g.scale.x, 0.0f), g.qmax.x);
    const unsigned qy = (unsigned)fminf(fmaxf((r0.y - g.lo.y) * g.scale.y, 0.0f), g.qmax.y);
    const unsigned qz = (unsigned)fminf(fmaxf((r0.z - g.lo.z) * g.scale.z, 0.0f), g.qmax.z);
    const unsigned ocell = deposit(qx, g.mask[0]) | deposit(qy, g.mask[1]) | deposit(qz, g.mask[2]);
    return (ocell << kOrderDirBits) | dcell;
}

// Origin bits of the key for n rays, and the grid they index (host).
int order_origin_bits(int64_t n);
OrderGrid order_grid(const float lo[3], const float hi[3], int origin_bits);

// Device scratch for ordering n rays: key + rank, the ray of each sorted slot, the sorted slot of
// each ray, 16 B per ray for a caller's hits in sorted order, 2^21 counts, the scan's chunk totals and
// the 256-byte state block (which must be zero when the scratch is new).
size_t reorder_scratch_bytes(int64_t n);
// Byte offset of the state block inside the scratch (to clear it on allocation).
size_t reorder_state_offset(int64_t n);

struct OrderOut {
    const int *src;                   // ray of each sorted slot
    const int *pos;                   // sorted slot of each ray (with_pos)
    void *hits;                       // 16 B per ray
    const unsigned long long *state;  // order_built(state): whether src / pos were built
};

// Launches (on stream s) the ordering of n rays (or of min(*n_dev, n) when n_dev is set: a count
// that lives on the device) within scene bounds lo < hi per axis. The scratch holds at least
// reorder_scratch_bytes(n); its 256-byte state block sits at byte state_at, zeroed when the
// scratch was made and fixed for its life (reorder_state_offset of the size it was made for).
// Calls on one scratch must be ordered (one stream). Launches only, no allocation, so a call can
// be captured in a CUDA graph. Fewer than min_rays rays keep their own order. Device-side errors go
// to *err as kErrOrder. with_pos: also the inverse permutation. clear: a word that the first pass sets to 0 (the work
// counter of the kernel that follows). wide_flags >= 0, a tree's BvhView::wide_flags: coherent rays are also looked
// at for those that its four-wide form does not serve (order_two_wide).
//
// The rays themselves stay where they are and a trace kernel reads them through src. A copy in
// sorted order, undone for the hits by a last pass, cost more than the scattered sectors do in a trace
// that takes 3 % of the memory bandwidth: 4M terrain bounces 840 us with the copy, 790 without.
tt_status reorder_rays(const float4 *rays, int64_t n, const int *n_dev, const float lo[3], const float hi[3],
                       void *scratch, size_t state_at, int64_t min_rays, unsigned *err, cudaStream_t s, OrderOut *out,
                       bool with_pos = false, unsigned long long *clear = nullptr, int64_t wide_flags = -1);

// Whether this call's rays were ordered: false when more than half of the sampled warps held 32
// equal keys (the rays are coherent already: camera rays share one origin cell and neighbouring
// pixels one direction cell) or too few rays came; they are then traced in their own order.
__device__ __forceinline__ bool order_built(const unsigned long long *state) { return state[3] == 1ull; }

// Whether this call's rays are coherent and hold so many that the four-wide loop does not serve that the two-wide
// one takes less for all: more than one of a sampled warp's 32. Each such ray holds up its warp while one lane
// runs the two-wide loop. 4M camera rays on the 2,097,152-triangle terrain, two-wide 660 us: with none
// such 489, a hundredth 604, a fiftieth 670, a twentieth 814, half 1,203. On terrains, spheres and the Cornell box, 1M
// and 4M camera rays, closest and any hit, two-wide takes 0.84 to 1.13 of the time with a fiftieth of them, 0.69
// to 0.99 with a twentieth. Incoherent sets are faster four-wide whatever the share (4M bounces, two-wide
// 1,165 us: 891 with a twentieth, 898 with half).
__device__ __forceinline__ bool order_two_wide(const unsigned long long *state) { return state[3] == 2ull; }

// The ray in a place of the order of rays 0 .. n - 1, for the kernels that take their rays through it. An order
// that is no permutation (two calls that overlap on one scratch make one, and places that the scatter left out
// hold what was there) is reported, and such a place keeps its own ray: a ray it leaves out has its hit
// unwritten, and no access goes beyond the caller's buffers.
__host__ __device__ inline unsigned ordered_slot(const int *src, unsigned place, unsigned n, uint32_t &err) {
    const unsigned i = (unsigned)src[place];
    if (i < n) return i;
    err |= kErrOrder;
    return place;
}

}  // namespace tt
