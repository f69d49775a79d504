// Two-wide compact SBVH to the four-wide device form (layout in tt_wide.h), on the device. No
// counterpart in the reference, which traverses the compact arrays as they are
// (src/bvh/BVHCompact.cpp:88-192).
//
// Which children a node takes in is chosen by expected visits: with A(n) the surface area of n's
// box, a wide node at n costs A(n) plus, for each of its two children, the cheaper of keeping the
// child as a wide node of its own or taking in its two children. The choice is made bottom up, so
// the tree's bottom fills up too: on a 512 x 512-cell terrain (188,814 two-wide nodes) it leaves
// 83,515 wide nodes where taking in every child top down leaves 89,942, a third of them with just
// two leaves.
//
// Passes over the two-wide nodes, one thread each: links to the parents (a node met twice: not a
// tree) and the bounds of tt_wide.h; costs from the bottom up, the second child to arrive going on
// with the parent; which nodes are wide nodes, their depth and their triangle pairs; their places,
// the tree's top levels first and breadth first, the rest in about the file's depth-first order;
// the records. The host reads the totals once, then allocates the records. Everything
// moves at memory speed: uploading the 2,097,152-triangle terrain (765,188 two-wide nodes), arrays and
// conversion, takes 3.0 ms (a conversion on one host thread took 59 ms by itself).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "tt_launch.cuh"
#include "tt_wide.cuh"
#include "tt_wide_build.h"

namespace tt {
namespace {

constexpr uint32_t kNoParent = 0xffffffffu;
// A scene of some thousand nodes meets more SMs than with 256 (uploading 20,492 triangles, one read-back
// less as well: 368 to 344 us; 131,072 triangles 550 to 513; 64: 353 and 533).
constexpr int kBuildBlock = 128;
constexpr uint32_t kLeafTriangles = 8192;  // of a leaf; a tree with a longer one stays two-wide
constexpr int kDepths = 128;  // depth buckets; deeper trees stay two-wide anyway (kWideStack)

struct Totals {
    uint32_t bad;       // not a tree, or outside the bounds
    uint32_t neg_zero;  // a box plane at -0.0
    uint32_t done;      // nodes whose cost is known and which are the root or have a parent
    uint32_t need;      // stack entries the root's traversal may need
    unsigned long long pairs;
    uint32_t depth[kDepths];   // wide nodes by depth
    uint32_t cursor[kDepths];  // places given out, by bucket
    uint32_t pair_cursor;
};

// No fault found and every node met, below the stack's depth.
__host__ __device__ inline bool convertible(const Totals &t, uint32_t count) {
    return !t.bad && t.done == count && t.need <= (uint32_t)kWideStack;
}

struct Build {
    const float4 *nodes, *verts;
    uint32_t count, num_verts;
    uint32_t *parent;  // 2 * parent + side
    float *cost;
    uint32_t *arrived, *index;
    uint8_t *take, *depth;
    uint16_t *need;
    uint32_t *met;  // a bit per vertex slot: the triangle that starts there is in a leaf already
    Totals *tot;
};
__host__ __device__ inline size_t leaf_words(uint32_t num_verts) { return (size_t)num_verts / 32 + 1; }

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ void load_node(const float4 *n, Box b[2], int32_t ch[2]) {
    const float4 a = n[0], c = n[1], z = n[2], r = n[3];
    b[0] = Box{{a.x, a.z, z.x}, {a.y, a.w, z.y}};
    b[1] = Box{{c.x, c.z, z.z}, {c.y, c.w, z.w}};
    ch[0] = __float_as_int(r.x);
    ch[1] = __float_as_int(r.y);
}

__device__ __forceinline__ float area(const Box &a, const Box &b) {
    float e[3];
    for (int k = 0; k < 3; k++) e[k] = fmaxf(a.hi[k], b.hi[k]) - fminf(a.lo[k], b.lo[k]);
    return e[0] * e[1] + e[1] * e[2] + e[2] * e[0];
}

// (1) parents; bounds of the planes
__global__ void __launch_bounds__(kBuildBlock) k_wide_parents(Build b) {
    bool bad = false, neg = false;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < b.count; n += gridDim.x * blockDim.x) {
        Box box[2];
        int32_t ch[2];
        load_node(b.nodes + 4 * (size_t)n, box, ch);
        for (int k = 0; k < 2; k++) {
            for (int a = 0; a < 3; a++) {
                for (float p : {box[k].lo[a], box[k].hi[a]}) {
                    const float m = fabsf(p);
                    bad |= !(m <= kWideCoordMax) || (m != 0.0f && m < kWidePlaneMin);  // also NaN
                    neg |= __float_as_uint(p) == 0x80000000u;
                }
                bad |= !(box[k].lo[a] <= box[k].hi[a]);
            }
            if (ch[k] < 0) {
                bad |= (uint32_t)~ch[k] >= b.num_verts;
                continue;
            }
            const uint32_t c = (uint32_t)ch[k] / 4;
            if (ch[k] % 4 || c >= b.count || c == 0) bad = true;
            else bad |= atomicExch(b.parent + c, 2 * n + k) != kNoParent;
        }
    }
    if (bad) b.tot->bad = 1;
    if (neg) b.tot->neg_zero = 1;
}

// (2) costs, from the nodes without inner children up
__global__ void __launch_bounds__(kBuildBlock) k_wide_costs(Build b) {
    if (b.tot->bad) return;
    uint32_t done = 0;
    for (uint32_t start = blockIdx.x * blockDim.x + threadIdx.x; start < b.count; start += gridDim.x * blockDim.x) {
        uint32_t n = start;
        Box box[2];
        int32_t ch[2];
        load_node(b.nodes + 4 * (size_t)n, box, ch);
        if (ch[0] >= 0 || ch[1] >= 0) continue;
        // Every node is reached once: each pass goes one level up a finite tree. A node of 2 h levels needs h stack
        // entries at least (a wide node holds two levels and keeps one or more of its slots for later).
        for (int level = 0;; level++) {
            if (level > 2 * kWideStack) {
                b.tot->bad = 1;
                break;
            }
            float total = area(box[0], box[1]);
            uint8_t taken = 0;
            uint32_t slots = 2, below = 0;
            bool sticks_out = false;
            for (int k = 0; k < 2; k++) {
                if (ch[k] < 0) continue;
                const uint32_t c = (uint32_t)ch[k] / 4;
                Box kb[2];
                int32_t g[2];
                load_node(b.nodes + ch[k], kb, g);
                float split = 0.0f;
                uint32_t deep = 0;
                for (int j = 0; j < 2; j++)
                    if (g[j] >= 0) {
                        split += __ldcg(b.cost + g[j] / 4);
                        deep = max(deep, (uint32_t)__ldcg(b.need + g[j] / 4));
                    }
                bool whole = true;  // the child's box is the union of its children's
                for (int a = 0; a < 3; a++) {
                    const float lo = fminf(kb[0].lo[a], kb[1].lo[a]), hi = fmaxf(kb[0].hi[a], kb[1].hi[a]);
                    whole &= lo == box[k].lo[a] && hi == box[k].hi[a];
                    sticks_out |= lo < box[k].lo[a] || hi > box[k].hi[a];
                }
                const float own = __ldcg(b.cost + c);
                if (whole && split <= own) {
                    taken |= (uint8_t)(1 << k);
                    total += split;
                    below = max(below, deep);
                    slots++;
                } else {
                    total += own;
                    below = max(below, (uint32_t)__ldcg(b.need + c));
                }
            }
            if (sticks_out) b.tot->bad = 1;
            b.cost[n] = total;
            b.take[n] = taken;
            const uint32_t need = min(below + slots - 1, 60000u);
            b.need[n] = (uint16_t)need;
            if (n == 0) {
                done++;
                b.tot->need = need;
                break;
            }
            // A node that no node refers to does not count, so the tree is refused before the passes that
            // follow every node's links up to the root. (Nodes in a ring never get here: each waits for
            // the next.)
            const uint32_t up = b.parent[n];
            if (up == kNoParent) break;
            done++;
            n = up / 2;
            load_node(b.nodes + 4 * (size_t)n, box, ch);
            if (ch[0] >= 0 && ch[1] >= 0) {
                __threadfence();
                if (atomicAdd(b.arrived + n, 1u) == 0) break;  // the other child goes on
                __threadfence();
            }
        }
    }
    if (done) atomicAdd(&b.tot->done, done);
}

__device__ __forceinline__ bool is_terminator(const float4 &v) { return __float_as_uint(v.x) == 0x80000000u; }

// Pairs of the leaf at slot `slot`; 0 for one that is not closed or outside the bounds, and, first time round,
// for one that shares a triangle with another leaf or is longer than one thread should walk. Leaves of
// a file may overlap: without the marks the walks would take leaves times triangles steps.
template <bool kFirst>
__device__ uint32_t leaf_pairs(const Build &b, uint32_t slot) {
    uint32_t tris = 0;
    for (; slot < b.num_verts; slot += 3, tris++) {
        const float4 v0 = b.verts[slot];
        if (is_terminator(v0)) return max(1u, (tris + 1) / 2);
        if (kFirst && tris == kLeafTriangles) return 0;
        if (slot + 3 >= b.num_verts) return 0;
        const float4 v1 = b.verts[slot + 1], v2 = b.verts[slot + 2];
        for (float c : {v0.x, v0.y, v0.z, v1.x, v1.y, v1.z, v2.x, v2.y, v2.z})
            if (!(fabsf(c) <= kWideCoordMax)) return 0;
        if (kFirst && (atomicOr(b.met + slot / 32, 1u << slot % 32) >> slot % 32 & 1u)) return 0;
    }
    return 0;
}

// The four slots of the wide node at two-wide node n: child address (kEmptySlot: none) and box.
constexpr int32_t kEmptySlot = 1;  // addresses of inner nodes are multiples of 4
__device__ __forceinline__ void wide_slots(const Build &b, uint32_t n, int32_t ref[4], Box box[4]) {
    const float inf = __int_as_float(0x7f800000);
    Box own[2];
    int32_t ch[2];
    load_node(b.nodes + 4 * (size_t)n, own, ch);
    for (int k = 0; k < 2; k++) {
        if (b.take[n] >> k & 1) {
            load_node(b.nodes + ch[k], box + 2 * k, ref + 2 * k);
        } else {
            ref[2 * k] = ch[k];
            box[2 * k] = own[k];
            ref[2 * k + 1] = kEmptySlot;
            box[2 * k + 1] = Box{{inf, inf, inf}, {-inf, -inf, -inf}};
        }
    }
}

// (3) wide nodes, their depths and pairs. index: 1 for a wide node, else 0. A node is taken in when
// its parent is a wide node and takes it; up a chain of taken links wide nodes alternate.
__global__ void __launch_bounds__(kBuildBlock) k_wide_roots(Build b) {
    __shared__ uint32_t s_depth[kDepths];
    if (!convertible(*b.tot, b.count)) return;
    for (int d = threadIdx.x; d < kDepths; d += blockDim.x) s_depth[d] = 0;
    __syncthreads();
    unsigned long long pairs = 0;
    bool bad = false;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < b.count; n += gridDim.x * blockDim.x) {
        uint32_t depth = 0, links = 0;
        bool chain = true;
        for (uint32_t x = n; x != 0 && depth < kDepths - 1; depth++) {
            const uint32_t up = b.parent[x];
            x = up / 2;
            chain = chain && (b.take[x] >> (up & 1) & 1);
            if (chain) links++;
        }
        const bool wide = (links & 1) == 0;
        b.index[n] = wide;
        b.depth[n] = (uint8_t)depth;
        if (!wide) continue;
        atomicAdd(s_depth + depth, 1u);
        int32_t ref[4];
        Box box[4];
        wide_slots(b, n, ref, box);
        for (int s = 0; s < 4; s++)
            if (ref[s] < 0) {
                const uint32_t p = leaf_pairs<true>(b, (uint32_t)~ref[s]);
                bad |= p == 0;
                pairs += p;
            }
    }
    if (bad) b.tot->bad = 1;
    if (pairs) atomicAdd(&b.tot->pairs, pairs);
    __syncthreads();
    for (int d = threadIdx.x; d < kDepths; d += blockDim.x)
        if (s_depth[d]) atomicAdd(b.tot->depth + d, s_depth[d]);
}

struct Buckets {
    uint32_t first[kDepths];   // place of the first wide node of each bucket
    uint32_t bucket[kDepths];  // bucket of each depth
};

// Buckets: every depth its own while they fit in top_nodes, then one for all the rest. The number of wide
// nodes.
inline size_t plan_places(const Totals &t, size_t top_nodes, Buckets &k) {
    k = Buckets{};
    size_t wide = 0;
    int rest = -1;
    for (int d = 0; d < kDepths; d++) {
        if (rest < 0 && wide + t.depth[d] > top_nodes) {
            rest = d;
            k.first[d] = (uint32_t)wide;
        }
        k.bucket[d] = (uint32_t)(rest < 0 ? d : rest);
        if (rest < 0) k.first[d] = (uint32_t)wide;
        wide += t.depth[d];
    }
    return wide;
}

// (4) places
__global__ void __launch_bounds__(kBuildBlock) k_wide_places(Build b, Buckets k) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < b.count; n += gridDim.x * blockDim.x) {
        if (!b.index[n]) continue;
        const uint32_t q = k.bucket[b.depth[n]];
        // one atomic per bucket among the warp's converged lanes, in lane order
        const unsigned peers = __match_any_sync(__activemask(), q);
        const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(b.tot->cursor + q, (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        b.index[n] = 1 + k.first[q] + base + __popc(peers & ((1u << lane) - 1u));
    }
}

// (5) records; the leaves' pairs in the order the threads ask for them
__global__ void __launch_bounds__(kBuildBlock) k_wide_records(Build b, char *nodes, uint32_t num_nodes, char *pairs,
                                                      uint32_t num_pairs) {
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < b.count; n += gridDim.x * blockDim.x) {
        const uint32_t place = b.index[n];
        if (!place || place > num_nodes) continue;
        int32_t ref[4];
        Box box[4];
        wide_slots(b, n, ref, box);
        float *w = reinterpret_cast<float *>(nodes + (size_t)(place - 1) * kWideNodeBytes);
        uint32_t own[4], sum = 0;
        for (int s = 0; s < 4; s++) {
            own[s] = ref[s] < 0 ? leaf_pairs<false>(b, (uint32_t)~ref[s]) : 0u;
            sum += own[s];
        }
        uint32_t first = sum ? atomicAdd(&b.tot->pair_cursor, sum) : 0u;
        for (int s = 0; s < 4; s++) {
            for (int c = 0; c < 4; c++) {
                w[8 * c + 2 * s] = c & 1 ? box[s].hi[0] : box[s].lo[0];
                w[8 * c + 2 * s + 1] = c & 2 ? box[s].hi[1] : box[s].lo[1];
                w[32 + 4 * c + s] = c == 0 || c == 3 ? box[s].lo[2] : box[s].hi[2];
            }
            uint32_t r = kWideEmpty;
            if (ref[s] < 0) {
                r = kWideLeaf | first;
                if (first + own[s] <= num_pairs)
                    wide_fill_pairs(b.verts, (uint32_t)~ref[s],
                                    reinterpret_cast<float *>(pairs + (size_t)first * kWidePairBytes));
                first += own[s];
            } else if (ref[s] != kEmptySlot) {
                r = b.index[ref[s] / 4] - 1;
            }
            w[48 + s] = __uint_as_float(r);
            w[52 + s] = 0.0f;
        }
    }
}

}  // namespace

#if defined(__CUDACC__)  // the passes above also build as plain C++, for the tests that run them on the CPU
cudaError_t build_wide(const BvhView &two, uint32_t num_nodes, uint32_t num_verts, size_t top_bytes, int num_sms,
                       WideBVH &out) {
    out = WideBVH();
    Build b{};
    b.nodes = two.nodes;
    b.verts = two.verts;
    b.count = num_nodes / 4;
    b.num_verts = num_verts;
    if (b.count == 0 || num_nodes % 4 || b.count > kWideIndex) return cudaSuccess;
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t n = b.count, words = align(4 * n), met = align(4 * leaf_words(num_verts));
    char *work = nullptr;
    cudaError_t e = cudaMalloc(&work, 4 * words + 2 * align(n) + align(2 * n) + met + align(sizeof(Totals)));
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();  // no room for the conversion: two-wide
    if (e != cudaSuccess) return e == cudaErrorMemoryAllocation ? cudaSuccess : e;
    char *p = work;
    auto take = [&p](size_t bytes) {
        char *q = p;
        p += bytes;
        return q;
    };
    b.parent = reinterpret_cast<uint32_t *>(take(words));
    b.arrived = reinterpret_cast<uint32_t *>(take(words));
    b.met = reinterpret_cast<uint32_t *>(take(met));  // (cleared together with arrived and tot)
    b.tot = reinterpret_cast<Totals *>(take(align(sizeof(Totals))));
    b.cost = reinterpret_cast<float *>(take(words));
    b.index = reinterpret_cast<uint32_t *>(take(words));
    b.take = reinterpret_cast<uint8_t *>(take(align(n)));
    b.depth = reinterpret_cast<uint8_t *>(take(align(n)));
    b.need = reinterpret_cast<uint16_t *>(take(align(2 * n)));
    const unsigned grid = (unsigned)std::min<size_t>((n + kBuildBlock - 1) / kBuildBlock, (size_t)num_sms * 2048 / kBuildBlock);
    Totals t;
    auto run = [&]() -> cudaError_t {
        cudaError_t c = cudaMemsetAsync(b.parent, 0xff, words, nullptr);
        if (c == cudaSuccess) c = cudaMemsetAsync(b.arrived, 0, words + met + align(sizeof(Totals)), nullptr);
        if (c == cudaSuccess) c = launch_plain(k_wide_parents, grid, kBuildBlock, 0, nullptr, b);
        if (c == cudaSuccess) c = launch_plain(k_wide_costs, grid, kBuildBlock, 0, nullptr, b);
        if (c == cudaSuccess) c = launch_plain(k_wide_roots, grid, kBuildBlock, 0, nullptr, b);
        if (c == cudaSuccess) c = cudaMemcpy(&t, b.tot, sizeof t, cudaMemcpyDeviceToHost);
        if (c != cudaSuccess) return c;
        if (!convertible(t, b.count)) return cudaSuccess;  // stays two-wide
        // (pairs: at most one per vertex slot, with every triangle in one leaf)
        if (t.pairs > num_verts || t.pairs > kWideIndex || t.depth[kDepths - 1]) return cudaSuccess;
        const size_t top_nodes = std::max<size_t>(1, top_bytes / kWideNodeBytes);
        Buckets k;
        const size_t wide = plan_places(t, top_nodes, k);
        const size_t nb = align(wide * kWideNodeBytes), pb = (size_t)t.pairs * kWidePairBytes;
        c = cudaMalloc(&out.base, nb + pb);
        if (c != cudaSuccess) return c;
        char *nodes = static_cast<char *>(out.base), *pairs = nodes + nb;
        c = launch_plain(k_wide_places, grid, kBuildBlock, 0, nullptr, b, k);
        if (c == cudaSuccess)
            c = launch_plain(k_wide_records, grid, kBuildBlock, 0, nullptr, b, nodes, wide, pairs, t.pairs);
        if (c == cudaSuccess) c = cudaStreamSynchronize(nullptr);
        if (c != cudaSuccess) return c;
        out.nodes = nodes;
        out.pairs = pairs;
        out.flags = t.neg_zero ? kWideNegZero : 0u;
        out.top_bytes = kWideNodeBytes * std::min(wide, top_nodes);
        return cudaSuccess;
    };
    e = run();
    cudaFree(work);
    if (e != cudaSuccess && out.base) {
        cudaFree(out.base);
        out = WideBVH();
    }
    if (e == cudaErrorMemoryAllocation) {  // no room for a second form: two-wide, as before
        cudaGetLastError();
        e = cudaSuccess;
    }
    return e;
}
#endif

}  // namespace tt
