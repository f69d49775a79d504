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
