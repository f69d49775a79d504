// Host build of the device passes that make the four-wide tree (trenchanttracer_gb300/csrc/tt_wide_build.cu), for
// the CPU tests: the passes themselves, one thread to a block and one block after another.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#undef __noinline__
#undef __launch_bounds__
#define __noinline__
#define __launch_bounds__(...)
template <class T> static inline T __ldg(const T *p) { return *p; }
template <class T> static inline T __ldcg(const T *p) { return *p; }
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
static inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static inline unsigned __activemask() { return 1u; }
static inline unsigned __ballot_sync(unsigned, bool p) { return p; }
static inline unsigned __match_any_sync(unsigned, unsigned) { return 1u; }
template <class T> static inline T __shfl_sync(unsigned, T v, int) { return v; }
static inline void __syncthreads() {}
static inline void __threadfence() {}
template <class T, class U> static inline T atomicAdd(T *p, U v) { const T old = *p; *p += (T)v; return old; }
template <class T> static inline T atomicExch(T *p, T v) { const T old = *p; *p = v; return old; }
template <class T> static inline T atomicOr(T *p, T v) { const T old = *p; *p |= v; return old; }
static uint3 blockIdx;
static const uint3 threadIdx{0, 0, 0};
static dim3 gridDim;
static const dim3 blockDim(1);
static inline uint32_t max(uint32_t a, uint32_t b) { return a < b ? b : a; }
static inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
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

#include "tt_wide_build.cu"

using namespace tt;

template <class Pass>
static void run(unsigned blocks, Pass pass) {
    gridDim = dim3(blocks);
    for (blockIdx.x = 0; blockIdx.x < blocks; blockIdx.x++) pass();
}

template <bool kClosest>
static void trace(const BvhView &v, const float *rays, long long n, int *addr, float *tuv, unsigned *err) {
    for (long long i = 0; i < n; i++) {
        const float *r = rays + 8 * i;
        const float4 r0 = make_float4(r[0], r[1], r[2], r[3]), r1 = make_float4(r[4], r[5], r[6], r[7]);
        WideStackOf<8, 1, kClosest> stack;
        typename WideEntry<kClosest>::type shared[8];
        stack.sh = shared;
        const TraceResult res =
            v.wide_nodes ? traverse_wide<kClosest>(stack, v, r0, r1, *err) : traverse<kClosest>(v, r0, r1, *err);
        addr[i] = res.addr;
        tuv[3 * i] = res.t;
        tuv[3 * i + 1] = res.u;
        tuv[3 * i + 2] = res.v;
    }
}

struct Form {
    std::vector<char> nodes, pairs;
    uint32_t flags = 0;
    long long wide = 0;  // nodes; 0: refused after pass `stage`; -1: see below
    int stage = 0;
    uint32_t done = 0;  // nodes whose cost the second pass knows
};

static Form convert(const float *nodes, long long num_nodes, const float *verts, long long num_verts,
                    long long top_nodes) {
    Form f;
    Build b{};
    b.nodes = reinterpret_cast<const float4 *>(nodes);
    b.verts = reinterpret_cast<const float4 *>(verts);
    b.count = (uint32_t)(num_nodes / 4);
    b.num_verts = (uint32_t)num_verts;
    std::vector<uint32_t> parent(b.count, 0xffffffffu), arrived(b.count, 0), index(b.count, 0xabababab);
    std::vector<float> cost(b.count, -1.0f);
    std::vector<uint8_t> take(b.count, 0xee), depth(b.count, 0xee);
    std::vector<uint16_t> need(b.count, 0xeeee);
    std::vector<uint32_t> met(leaf_words(b.num_verts), 0);
    Totals t{};
    b.parent = parent.data();
    b.arrived = arrived.data();
    b.index = index.data();
    b.cost = cost.data();
    b.take = take.data();
    b.depth = depth.data();
    b.need = need.data();
    b.met = met.data();
    b.tot = &t;
    const unsigned blocks = 7;
    run(blocks, [&] { k_wide_parents(b); });
    f.stage = 1;
    if (t.bad) return f;
    run(blocks, [&] { k_wide_costs(b); });
    f.stage = 2;
    f.done = t.done;
    if (!convertible(t, b.count)) return f;
    for (uint32_t k = 1; k < b.count; k++)  // the third pass follows every node's links up to the root
        if (parent[k] / 2 >= b.count) {
            f.wide = -1;
            return f;
        }
    run(blocks, [&] { k_wide_roots(b); });
    f.stage = 3;
    if (t.bad || t.pairs > b.num_verts || t.depth[kDepths - 1]) return f;
    Buckets k;
    f.wide = (long long)plan_places(t, (size_t)top_nodes, k);
    f.nodes.resize((size_t)f.wide * kWideNodeBytes);
    f.pairs.resize((size_t)t.pairs * kWidePairBytes);
    run(blocks, [&] { k_wide_places(b, k); });
    run(blocks, [&] { k_wide_records(b, f.nodes.data(), (uint32_t)f.wide, f.pairs.data(), (uint32_t)t.pairs); });
    f.stage = t.pair_cursor == t.pairs ? 0 : 5;
    f.flags = t.neg_zero ? kWideNegZero : 0u;
    return f;
}

extern "C" {
// Converts a compact tree (float4 nodes and vertices) and traces n rays through what the passes made, or
// through the two-wide tree. Returns the number of four-wide nodes, 0 when the tree must stay
// two-wide, -1 when the passes let one through whose later passes would read out of range. stage: the pass
// (1 to 5) after which a tree was refused, 0 for none.
long long wide_passes_trace(const float *nodes, long long num_nodes, const float *verts, long long num_verts,
                            long long top_nodes, const float *rays, long long n, int closest, int two_wide, int *addr,
                            float *tuv, unsigned *err, int *stage) {
    Form f;
    if (!two_wide) f = convert(nodes, num_nodes, verts, num_verts, top_nodes);
    *stage = f.stage;
    if (f.wide < 0) return f.wide;
    BvhView v{};
    v.nodes = reinterpret_cast<const float4 *>(nodes);
    v.verts = reinterpret_cast<const float4 *>(verts);
    if (f.wide) {
        v.wide_nodes = f.nodes.data();
        v.wide_pairs = f.pairs.data();
        v.wide_flags = f.flags;
    }
    if (closest) trace<true>(v, rays, n, addr, tuv, err);
    else trace<false>(v, rays, n, addr, tuv, err);
    return f.wide;
}

// The four-wide form alone; out[0] nodes, out[1] pairs (kept until the next call), sizes in bytes, flags; done: the
// nodes whose cost the second pass found.
long long wide_passes_form(const float *nodes, long long num_nodes, const float *verts, long long num_verts,
                           long long top_nodes, const char **out, long long *bytes, unsigned *flags, unsigned *done) {
    static Form f;
    f = convert(nodes, num_nodes, verts, num_verts, top_nodes);
    out[0] = f.nodes.data();
    out[1] = f.pairs.data();
    bytes[0] = (long long)f.nodes.size();
    bytes[1] = (long long)f.pairs.size();
    *flags = f.flags;
    *done = f.done;
    return f.wide;
}
}
