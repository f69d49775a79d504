// Host build of the four-wide traversal (trenchanttracer_gb300/csrc/tt_wide.cuh), for the CPU tests:
// the device header with plain C++ in the place of the CUDA intrinsics it uses.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#define __device__
#define __forceinline__ inline
#define __noinline__
struct float4 { float x, y, z, w; };
struct uint4 { uint32_t x, y, z, w; };
struct uint2 { uint32_t x, y; };
static inline float4 make_float4(float a, float b, float c, float d) { return float4{a, b, c, d}; }
static inline uint2 make_uint2(uint32_t a, uint32_t b) { return uint2{a, b}; }
template <class T> static inline T __ldg(const T *p) { return *p; }
static inline int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static inline float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static inline unsigned __float_as_uint(float f) { return (unsigned)__float_as_int(f); }
static inline float __uint_as_float(unsigned u) { return __int_as_float((int)u); }
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }
static inline int __popc(unsigned x) { return __builtin_popcount(x); }
static inline unsigned __activemask() { return 1u; }
static inline unsigned __ballot_sync(unsigned, bool p) { return p; }
// the device's maximum and minimum: a NaN loses, +0 is above -0
static inline float dev_max(float a, float b) {
    if (a == b) return std::signbit(a) ? b : a;
    return std::fmax(a, b);
}
static inline float dev_min(float a, float b) {
    if (a == b) return std::signbit(a) ? a : b;
    return std::fmin(a, b);
}
#define fmaxf dev_max
#define fminf dev_min

#include "tt_wide.cuh"
#include "tt_internal.h"

#undef fmaxf
#undef fminf
#include <algorithm>
#include <limits>

namespace tt {
namespace {

struct Box {
    float lo[3], hi[3];
};

Box child_box(const I4 *n, int k) {
    float f[12];
    std::memcpy(f, n, sizeof f);
    Box b;
    b.lo[0] = f[4 * k];
    b.hi[0] = f[4 * k + 1];
    b.lo[1] = f[4 * k + 2];
    b.hi[1] = f[4 * k + 3];
    b.lo[2] = f[8 + 2 * k];
    b.hi[2] = f[9 + 2 * k];
    return b;
}

float area(const Box &b) {
    const float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
    return x * y + y * z + z * x;
}

Box unite(const Box &a, const Box &b) {
    Box u;
    for (int k = 0; k < 3; k++) {
        u.lo[k] = std::min(a.lo[k], b.lo[k]);
        u.hi[k] = std::max(a.hi[k], b.hi[k]);
    }
    return u;
}

bool same_planes(const Box &a, const Box &b) {
    for (int k = 0; k < 3; k++)
        if (!(a.lo[k] == b.lo[k] && a.hi[k] == b.hi[k])) return false;
    return true;
}

bool inside(const Box &a, const Box &b) {
    for (int k = 0; k < 3; k++)
        if (!(a.lo[k] >= b.lo[k] && a.hi[k] <= b.hi[k])) return false;
    return true;
}

bool plane_ok(float p, uint32_t &flags) {
    const float m = std::fabs(p);
    if (!(m <= kWideCoordMax)) return false;  // also NaN
    if (m == 0.0f) {
        if (std::signbit(p)) flags |= kWideNegZero;
        return true;
    }
    return m >= kWidePlaneMin;
}

bool vertex_ok(const I4 &v) {
    float f[3];
    std::memcpy(f, &v, sizeof f);
    return std::fabs(f[0]) <= kWideCoordMax && std::fabs(f[1]) <= kWideCoordMax && std::fabs(f[2]) <= kWideCoordMax;
}

}  // namespace

struct WideBVH {
    std::vector<uint32_t> nodes;   // kWideNodeBytes / 4 words per node, root first
    std::vector<uint32_t> leaves;  // per leaf: its float4 slot in the vertex array, its first pair
    size_t pairs = 0;
    uint32_t flags = 0;
};

// The four-wide form, by the rules of tt_wide_build.cu; false when the tree must stay two-wide.
static bool build_wide(const CompactBVH &b, size_t top_bytes, WideBVH &out) {
    out = WideBVH();
    const size_t count = b.nodes.size() / 4;
    if (count == 0 || b.nodes.size() % 4 || count > kWideIndex) return false;
    const I4 *N = b.nodes.data();
    // depth-first order, every node once (a node met twice: not a tree)
    std::vector<uint32_t> order;
    order.reserve(count);
    {
        std::vector<uint8_t> seen(count, 0);
        std::vector<uint32_t> todo{0};
        seen[0] = 1;
        while (!todo.empty()) {
            const uint32_t n = todo.back();
            todo.pop_back();
            order.push_back(n);
            const I4 &c = N[4 * (size_t)n + 3];
            for (int32_t a : {c.y, c.x}) {
                if (a < 0) continue;
                if (a % 4 || (size_t)a / 4 >= count || seen[a / 4]) return false;
                seen[a / 4] = 1;
                todo.push_back((uint32_t)(a / 4));
            }
        }
    }
    // bottom up: which children a wide node at n takes in, and what that costs
    std::vector<float> cost(count);
    std::vector<uint8_t> take(count);
    std::vector<uint16_t> need(count);
    for (size_t i = order.size(); i-- > 0;) {
        const uint32_t n = order[i];
        const I4 *node = N + 4 * (size_t)n;
        const int32_t ch[2] = {node[3].x, node[3].y};
        const Box box[2] = {child_box(node, 0), child_box(node, 1)};
        float total = area(unite(box[0], box[1]));
        uint8_t taken = 0;
        int slots = 0;
        unsigned below = 0;
        for (int k = 0; k < 2; k++) {
            for (int a = 0; a < 3; a++)
                if (!plane_ok(box[k].lo[a], out.flags) || !plane_ok(box[k].hi[a], out.flags) ||
                    !(box[k].lo[a] <= box[k].hi[a]))
                    return false;
            if (ch[k] < 0) {
                slots++;
                continue;
            }
            const uint32_t c = (uint32_t)(ch[k] / 4);
            const I4 *kid = N + 4 * (size_t)c;
            const Box kb[2] = {child_box(kid, 0), child_box(kid, 1)};
            if (!inside(kb[0], box[k]) || !inside(kb[1], box[k])) return false;
            float split = 0.0f;
            unsigned deep = 0;
            for (int32_t g : {kid[3].x, kid[3].y})
                if (g >= 0) {
                    split += cost[g / 4];
                    deep = std::max<unsigned>(deep, need[g / 4]);
                }
            if (same_planes(unite(kb[0], kb[1]), box[k]) && split <= cost[c]) {
                taken |= (uint8_t)(1 << k);
                total += split;
                below = std::max(below, deep);
                slots += 2;
            } else {
                total += cost[c];
                below = std::max<unsigned>(below, need[c]);
                slots++;
            }
        }
        cost[n] = total;
        take[n] = taken;
        need[n] = (uint16_t)std::min<unsigned>(below + (unsigned)slots - 1u, 60000u);
    }
    if (need[0] > (unsigned)kWideStack) return false;
    // the wide nodes: breadth first from the root until top_bytes, then depth first
    struct Item {
        uint32_t n, at;
    };
    auto slots_of = [&](uint32_t n, int32_t ref[4], Box box[4]) {
        const I4 *node = N + 4 * (size_t)n;
        const int32_t ch[2] = {node[3].x, node[3].y};
        for (int k = 0; k < 2; k++) {
            if (take[n] >> k & 1) {
                const I4 *kid = N + ch[k];
                ref[2 * k] = kid[3].x;
                ref[2 * k + 1] = kid[3].y;
                box[2 * k] = child_box(kid, 0);
                box[2 * k + 1] = child_box(kid, 1);
            } else {
                ref[2 * k] = ch[k];
                box[2 * k] = child_box(node, k);
                ref[2 * k + 1] = 1;  // empty (addresses of inner nodes are multiples of 4)
                const float inf = std::numeric_limits<float>::infinity();
                box[2 * k + 1] = Box{{inf, inf, inf}, {-inf, -inf, -inf}};
            }
        }
    };
    constexpr size_t kWords = kWideNodeBytes / 4;
    out.nodes.reserve(kWords * (count / 2 + 1));
    size_t wide = 1;
    const size_t top_nodes = std::max<size_t>(1, top_bytes / kWideNodeBytes);
    size_t pairs = 0;
    bool ok = true;
    // writes the wide node of item `it`, appending its inner slots to `next` (with their places)
    auto emit = [&](const Item &it, std::vector<Item> &next) {
        int32_t ref[4];
        Box box[4];
        slots_of(it.n, ref, box);
        if (out.nodes.size() < kWords * (it.at + 1)) out.nodes.resize(kWords * (it.at + 1));
        uint32_t *w = out.nodes.data() + kWords * it.at;
        for (int s = 0; s < 4; s++) {
            for (int c = 0; c < 4; c++) {
                std::memcpy(w + 8 * c + 2 * s, c & 1 ? &box[s].hi[0] : &box[s].lo[0], 4);
                std::memcpy(w + 8 * c + 2 * s + 1, c & 2 ? &box[s].hi[1] : &box[s].lo[1], 4);
            }
            for (int c = 0; c < 4; c++) std::memcpy(w + 32 + 4 * c + s, c == 0 || c == 3 ? &box[s].lo[2] : &box[s].hi[2], 4);
            uint32_t r;
            if (ref[s] == 1) {
                r = kWideEmpty;
            } else if (ref[s] >= 0) {
                r = (uint32_t)wide++;
                next.push_back({(uint32_t)(ref[s] / 4), r});
            } else {
                const size_t slot = (size_t)~ref[s];
                size_t tris = 0;
                for (size_t v = slot; v < b.vertices.size() && (uint32_t)b.vertices[v].x != 0x80000000u; v += 3) {
                    if (v + 3 >= b.vertices.size() || !vertex_ok(b.vertices[v]) || !vertex_ok(b.vertices[v + 1]) ||
                        !vertex_ok(b.vertices[v + 2])) {
                        ok = false;
                        return;
                    }
                    tris++;
                }
                out.leaves.push_back((uint32_t)slot);
                out.leaves.push_back((uint32_t)pairs);
                r = kWideLeaf | (uint32_t)pairs;
                pairs += std::max<size_t>(1, (tris + 1) / 2);
                // leaves shared by several nodes could multiply the triangles
                if (slot >= b.vertices.size() || pairs > b.vertices.size() || pairs >= kWideIndex) {
                    ok = false;
                    return;
                }
            }
            w[48 + s] = r;
        }
        for (int s = 52; s < 56; s++) w[s] = 0;
    };
    std::vector<Item> level{{0, 0}}, next;
    size_t placed = 0;
    while (!level.empty() && placed + level.size() <= top_nodes && ok) {
        next.clear();
        for (const Item &it : level) {
            emit(it, next);
            if (!ok) return false;
        }
        placed += level.size();
        level.swap(next);
    }
    std::vector<Item> todo(level.rbegin(), level.rend());
    while (!todo.empty()) {
        const Item it = todo.back();
        todo.pop_back();
        next.clear();
        emit(it, next);
        if (!ok) return false;
        todo.insert(todo.end(), next.rbegin(), next.rend());
    }
    if (out.nodes.size() != kWords * wide || wide > kWideIndex) return false;
    out.pairs = pairs;
    return true;
}

}  // namespace tt

using namespace tt;

template <bool kClosest>
static void trace(const BvhView &v, const float *rays, long long n, int *addr, float *tuv, unsigned *err, int *regular,
                  bool wide) {
    for (long long i = 0; i < n; i++) {
        const float *r = rays + 8 * i;
        const float4 r0{r[0], r[1], r[2], r[3]}, r1{r[4], r[5], r[6], r[7]};
        TraceResult res;
        if (wide) {
            WideStackOf<8, 1, kClosest> stack;
            typename WideEntry<kClosest>::type shared[8];
            stack.sh = shared;
            res = traverse_wide<kClosest>(stack, v, r0, r1, *err);
        } else {
            res = traverse<kClosest>(v, r0, r1, *err);
        }
        TravStack<0, 1> tmp;
        TravState s;
        trav_init(s, tmp, r0, r1);
        regular[i] = wide_regular(r0, r1, s.idirx, s.idiry, s.idirz, s.oodx, s.oody, s.oodz, v.wide_flags);
        addr[i] = res.addr;
        tuv[3 * i] = res.t;
        tuv[3 * i + 1] = res.u;
        tuv[3 * i + 2] = res.v;
    }
}

extern "C" {
// Traces n rays through a compact tree (float4 nodes and vertices), two-wide or four-wide. Returns
// the number of four-wide nodes (0: the tree has no four-wide form), -1 on bad input.
long long wide_host_trace(const int32_t *nodes, long long num_nodes, const int32_t *verts, long long num_verts,
                          const float *rays, long long n, int closest, int wide, int *addr, float *tuv, unsigned *err,
                          int *regular, unsigned *flags) {
    CompactBVH b;
    b.nodes.resize((size_t)num_nodes);
    b.vertices.resize((size_t)num_verts);
    memcpy(b.nodes.data(), nodes, 16 * (size_t)num_nodes);
    memcpy(b.vertices.data(), verts, 16 * (size_t)num_verts);
    WideBVH w;
    const bool have = build_wide(b, 1 << 16, w);
    std::vector<char> pairs(kWidePairBytes * (have ? w.pairs : 0));
    BvhView v{};
    v.nodes = reinterpret_cast<const float4 *>(b.nodes.data());
    v.verts = reinterpret_cast<const float4 *>(b.vertices.data());
    if (have) {
        for (size_t k = 0; k < w.leaves.size(); k += 2)
            wide_fill_pairs(v.verts, w.leaves[k],
                            reinterpret_cast<float *>(pairs.data() + (size_t)kWidePairBytes * w.leaves[k + 1]));
        v.wide_nodes = reinterpret_cast<const char *>(w.nodes.data());
        v.wide_pairs = pairs.data();
        v.wide_flags = w.flags;
    }
    *flags = w.flags;
    if (closest) trace<true>(v, rays, n, addr, tuv, err, regular, wide != 0);
    else trace<false>(v, rays, n, addr, tuv, err, regular, wide != 0);
    return have ? (long long)(w.nodes.size() * 4 / kWideNodeBytes) : 0;
}
}
