// Traversal of the four-wide tree (layout in tt_wide.h), with the result of the two-wide one
// (tt_traverse.cuh) bit for bit.
//
// Why it is faster: the two-wide loop is bound by issue, by load sectors and by latency. An
// incoherent terrain ray takes 24 dependent node steps of some 75 instructions and 4 load sectors.
// A four-wide step does the work of two: one round trip to the cache instead of two, the planes
// of four boxes in three 32-byte loads, two planes per packed float instruction, and no per-axis
// minima and maxima, because the signs of the direction pick the entered and the left planes by
// address. Leaves hold their triangles in pairs, so one pass of the packed instructions tests two.
// 4M rays on the 2,097,152-triangle terrain, two-wide to four-wide (both sets through the ordering):
// camera rays 0.64 to 0.49 ms, cosine bounces 1.18 to 0.83 ms.
//
// Why the result is the same. The two-wide loop at a node A tests A's children B and C against the
// current hit distance t, goes to the one with the smaller entry distance (B when equal) and
// pushes the other, which it visits later without another test; leaves are tested in that order.
//   - Near side. The near child is visited next, with t unchanged, so testing its children
//     together with A's is what the two-wide loop does. Its own test needs no instruction: a box is
//     taken apart only when it is the union of its children's, the slab value fma(plane, idir, -ood)
//     is monotone in the plane, so whenever a child passes the parent does too, and a parent none
//     of whose children passes has no effect.
//   - Order. A group's entry distance comes from the minima of its slots' near planes, which are
//     the near planes of the union.
//   - Far side. Its children are tested when they are popped, by then against a smaller t. A box
//     that passed with an earlier t passes with a smaller t >= 0 exactly when its entry distance is
//     at most t (the entry does not depend on t and the exit only through min(exit, t)), so the
//     entry goes on the stack as the key and is compared at the pop. The two-wide loop tests both
//     children of the far node at one moment, when the first of them is reached: if the second
//     is a leaf, the first one's entry carries kWideMark, and its pop settles the second's test
//     too. A leaf whose test was settled has key 0. For inner nodes a late test is harmless: an
//     inner node with entry > t has no child with entry <= t.
//   - Any hit never changes t, so nothing is tested at the pop and the keys are not kept.
// The box test's signed-integer min / max equals the float one when the begin operand tmin is
// not negative (a negative value never wins the entry, and an exit below zero fails either way)
// except for an exit of exactly -0.0 beside a more negative one when the entry is 0, which takes a
// plane at zero: wide_regular sends rays that could meet it, and rays outside the bounds of
// tt_wide.h, to the two-wide loop. Within those bounds no value overflows or is NaN, so a
// triangle's division can wait until the test's signs have not already refused it (below).
#pragma once

#include "tt_traverse.cuh"
#include "tt_wide.h"

namespace tt {

// ---- two floats in one 64-bit register pair ------------------------------------------------------
typedef unsigned long long f32x2;

#if defined(__CUDACC__)
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
#else  // the same on the host, for the tests that compare the two loops there
inline f32x2 pack2(float a, float b) {
    return (f32x2)(uint32_t)__float_as_int(a) | (f32x2)(uint32_t)__float_as_int(b) << 32;
}
inline void unpack2(f32x2 v, float &a, float &b) {
    a = __int_as_float((int)(uint32_t)v);
    b = __int_as_float((int)(uint32_t)(v >> 32));
}
inline f32x2 fma2(f32x2 x, f32x2 y, f32x2 z) {
    float a, b, c, d, e, f;
    unpack2(x, a, b);
    unpack2(y, c, d);
    unpack2(z, e, f);
    return pack2(__fmaf_rn(a, c, e), __fmaf_rn(b, d, f));
}
inline f32x2 mul2(f32x2 x, f32x2 y) {
    float a, b, c, d;
    unpack2(x, a, b);
    unpack2(y, c, d);
    return pack2(__fmul_rn(a, c), __fmul_rn(b, d));
}
inline f32x2 add2(f32x2 x, f32x2 y) {
    float a, b, c, d;
    unpack2(x, a, b);
    unpack2(y, c, d);
    return pack2(__fadd_rn(a, c), __fadd_rn(b, d));
}
#endif
__device__ __forceinline__ f32x2 neg2(f32x2 v) {
    float a, b;
    unpack2(v, a, b);
    return pack2(-a, -b);
}
// a.y*b.z - a.z*b.y and a.x*b.x + a.y*b.y + a.z*b.z of two triangles, contracted as cross_c and dot_c;
// naz = -a.z (negating a factor negates the product)
__device__ __forceinline__ f32x2 cross2(f32x2 ay, f32x2 bz, f32x2 naz, f32x2 by) {
    return fma2(ay, bz, mul2(naz, by));
}
__device__ __forceinline__ f32x2 dot2(f32x2 ax, f32x2 ay, f32x2 az, f32x2 bx, f32x2 by, f32x2 bz) {
    return fma2(az, bz, fma2(ax, bx, mul2(ay, by)));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
#if defined(__CUDACC__)
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
__device__ __forceinline__ float min3(float a, float b, float c) {
#if defined(__CUDACC__)
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fminf(fminf(a, b), c);
#endif
}

struct Sector {  // 32 bytes: four packed pairs
    f32x2 a, b, c, d;
};
__device__ __forceinline__ Sector ldg_sector(const char *p) {
    Sector r;
#if defined(__CUDACC__)
    asm("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(r.a), "=l"(r.b), "=l"(r.c), "=l"(r.d) : "l"(p));
#else
    memcpy(&r, p, sizeof r);
#endif
    return r;
}

// ---- traversal stack --------------------------------------------------------------------------
// Entry: .x the reference, .y the key's bits (closest hit; any hit keeps the reference alone).
// The lowest kSh entries lie in shared memory at sh[i * kStride], the rest in local memory.
template <int kSh, int kStride, bool kKeys>
struct WideStackOf;
template <int kSh, int kStride>
struct WideStackOf<kSh, kStride, true> {
    static constexpr int kShared = kSh;
    uint2 *sh;
    uint2 loc[kWideStack - kSh];
    __device__ __forceinline__ uint2 get(int i) const {
        if (kSh > 0 && i < kSh) return sh[i * kStride];
        return loc[i - kSh];
    }
    __device__ __forceinline__ void set(int i, uint32_t ref, float key) {
        const uint2 e = make_uint2(ref, __float_as_uint(key));
        if (kSh > 0 && i < kSh) sh[i * kStride] = e;
        else loc[i - kSh] = e;
    }
    // onto the shared part, which has room
    __device__ __forceinline__ void push_if(bool p, int &i, uint32_t ref, float key) {
        if (p) sh[i * kStride] = make_uint2(ref, __float_as_uint(key));
        i += p;
    }
};
template <int kSh, int kStride>
struct WideStackOf<kSh, kStride, false> {
    static constexpr int kShared = kSh;
    uint32_t *sh;
    uint32_t loc[kWideStack - kSh];
    __device__ __forceinline__ uint2 get(int i) const {
        if (kSh > 0 && i < kSh) return make_uint2(sh[i * kStride], 0u);
        return make_uint2(loc[i - kSh], 0u);
    }
    __device__ __forceinline__ void set(int i, uint32_t ref, float) {
        if (kSh > 0 && i < kSh) sh[i * kStride] = ref;
        else loc[i - kSh] = ref;
    }
    __device__ __forceinline__ void push_if(bool p, int &i, uint32_t ref, float) {
        if (p) sh[i * kStride] = ref;
        i += p;
    }
};

// The word of shared memory an entry takes.
template <bool kKeys>
struct WideEntry {
    typedef uint2 type;
};
template <>
struct WideEntry<false> {
    typedef uint32_t type;
};

// Whether the four-wide loop serves this ray (see the head of this file). idir and ood as
// trav_init forms them.
__device__ __forceinline__ bool wide_regular(float4 r0, float4 r1, float idx, float idy, float idz, float oodx,
                                             float oody, float oodz, uint32_t flags) {
    const bool in_bounds = fabsf(r0.x) <= kWideCoordMax && fabsf(r0.y) <= kWideCoordMax &&
                           fabsf(r0.z) <= kWideCoordMax && fabsf(r0.w) <= kWideDirMax &&
                           fabsf(r1.x) <= kWideDirMax && fabsf(r1.y) <= kWideDirMax;
    // tmin: sign bit clear, finite; tmax: positive, not NaN
    const unsigned tmin = __float_as_uint(r1.z);
    bool ok = in_bounds && tmin < 0x7f800000u && r1.w > 0.0f;
    if (tmin == 0u) {  // an exit of -0.0: ood = +0 and either idir < 0 or a plane at -0.0
        const bool neg = (flags & kWideNegZero) != 0;
        if (__float_as_uint(oodx) == 0u && (idx < 0.0f || neg)) ok = false;
        if (__float_as_uint(oody) == 0u && (idy < 0.0f || neg)) ok = false;
        if (__float_as_uint(oodz) == 0u && (idz < 0.0f || neg)) ok = false;
    }
    return ok;
}

// The same from the ray alone.
__device__ __forceinline__ bool wide_serves(float4 r0, float4 r1, uint32_t flags) {
    const float ooeps = 8.27180612553027674871e-25f;  // as in wide_start
    const float idx = __frcp_rn(fabsf(r0.w) > ooeps ? r0.w : copysignf(ooeps, r0.w));
    const float idy = __frcp_rn(fabsf(r1.x) > ooeps ? r1.x : copysignf(ooeps, r1.x));
    const float idz = __frcp_rn(fabsf(r1.y) > ooeps ? r1.y : copysignf(ooeps, r1.y));
    return wide_regular(r0, r1, idx, idy, idz, __fmul_rn(r0.x, idx), __fmul_rn(r0.y, idy), __fmul_rn(r0.z, idz), flags);
}

// The two-wide loop, kept out of line for the few rays (or trees) the four-wide one does not serve.
template <bool kClosest>
__device__ __noinline__ TraceResult traverse_two_wide(const BvhView &bvh, float4 r0, float4 r1, uint32_t &err) {
    return traverse<kClosest>(bvh, r0, r1, err);
}

// Where the leaf step takes its ray from. kStride > 0: shared memory, word k of thread t at k *
// kStride + t, for rays that lie in host memory: reading them again for every leaf would double the
// traffic over the link (4M camera rays 1.20 ms, kept in shared memory 0.72). 0: the ray buffer; in
// device memory the reads cost nothing that shows (in registers the ray would cost resident warps).
template <int kStride>
struct WideRays {
    float *sh;
    __device__ __forceinline__ void put(float4 r0, float4 r1) {
        sh[0 * kStride] = r0.x;
        sh[1 * kStride] = r0.y;
        sh[2 * kStride] = r0.z;
        sh[3 * kStride] = r0.w;
        sh[4 * kStride] = r1.x;
        sh[5 * kStride] = r1.y;
    }
    template <class Fetch>
    __device__ __forceinline__ void get(Fetch, unsigned, float4 &r0, float4 &r1) const {
        r0 = make_float4(sh[0 * kStride], sh[1 * kStride], sh[2 * kStride], sh[3 * kStride]);
        r1 = make_float4(sh[4 * kStride], sh[5 * kStride], 0.0f, 0.0f);
    }
};
template <>
struct WideRays<0> {
    float *sh;
    __device__ __forceinline__ void put(float4, float4) {}
    template <class Fetch>
    __device__ __forceinline__ void get(Fetch fetch, unsigned slot, float4 &r0, float4 &r1) const {
        fetch(slot, r0, r1);
    }
};

// What a lane is about to do, besides visiting an inner node (reference < kWideMark) or a leaf
// (bit 31 set).
constexpr uint32_t kWidePop = 0x7ffffffeu;   // take the next stack entry
constexpr uint32_t kWideDone = 0x7ffffffdu;  // its ray is finished
constexpr uint32_t kWideIdle = 0x7ffffffcu;  // it has no ray

// One lane's traversal. The ray's origin and direction are kept elsewhere (WideRays): the leaf test is
// the rarer step.
struct WideState {
    f32x2 ixy, iz;  // inverse direction: x and y, z twice
    f32x2 mxy, mz;  // -origin * inverse direction, alike
    uint32_t sxy, sz;  // byte offsets of the near x and y planes (the far ones: ^ 96) and of the z planes
    float tmin, t, u, v;
    int addr;
    uint32_t ref;
    int sp;
};

// A ray's start; false when the two-wide loop must trace it.
__device__ __forceinline__ bool wide_start(WideState &s, const BvhView &bvh, float4 r0, float4 r1) {
    const float ooeps = 8.27180612553027674871e-25f;  // exp2f(-80), exact
    const float dx = r0.w, dy = r1.x, dz = r1.y;
    const float idx = __frcp_rn(fabsf(dx) > ooeps ? dx : copysignf(ooeps, dx));
    const float idy = __frcp_rn(fabsf(dy) > ooeps ? dy : copysignf(ooeps, dy));
    const float idz = __frcp_rn(fabsf(dz) > ooeps ? dz : copysignf(ooeps, dz));
    const float oodx = __fmul_rn(r0.x, idx), oody = __fmul_rn(r0.y, idy), oodz = __fmul_rn(r0.z, idz);
    s.ixy = pack2(idx, idy);
    s.iz = pack2(idz, idz);
    s.mxy = pack2(-oodx, -oody);
    s.mz = pack2(-oodz, -oodz);
    s.sxy = (idx < 0.0f ? 32u : 0u) | (idy < 0.0f ? 64u : 0u);
    s.sz = idz < 0.0f ? 160u : 128u;
    s.tmin = r1.z;
    s.t = r1.w;
    s.u = 0.0f;
    s.v = 0.0f;
    s.addr = -1;
    s.ref = 0;
    s.sp = 0;
    return bvh.wide_nodes && wide_regular(r0, r1, idx, idy, idz, oodx, oody, oodz, bvh.wide_flags);
}

// The next stack entry whose box is still passed.
template <bool kClosest, class Stack>
__device__ __forceinline__ void wide_pop(WideState &s, Stack &stack) {
    while (s.ref == kWidePop) {
        if (s.sp == 0) {
            s.ref = kWideDone;
            break;
        }
        const uint2 e = stack.get(--s.sp);
        if (!kClosest) {
            s.ref = e.x;
        } else if (__uint_as_float(e.y) <= s.t) {
            s.ref = e.x;
            if (e.x & kWideMark) {
                s.ref = e.x & ~kWideMark;
                const uint2 below = stack.get(s.sp - 1);
                if (__uint_as_float(below.y) <= s.t) stack.set(s.sp - 1, below.x, 0.0f);
            }
        }
    }
}

// Visits inner node s.ref: pushes what is passed but the nearest, and goes to that.
template <bool kClosest, class Stack>
__device__ __forceinline__ void wide_node(WideState &s, Stack &stack, const BvhView &bvh) {
    const float kNone = __int_as_float(0x7f800000);
    const char *node = bvh.wide_nodes + (uint64_t)s.ref * kWideNodeBytes;
    const Sector near = ldg_sector(node + s.sxy), far = ldg_sector(node + (s.sxy ^ 96u));
    const Sector both = ldg_sector(node + s.sz);
    const uint4 refs = __ldg(reinterpret_cast<const uint4 *>(node + 192));
    const float tcull = fminf(s.t, 1e20f);
    float ax0, ax1, ax2, ax3, ay0, ay1, ay2, ay3, az0, az1, az2, az3;
    unpack2(fma2(near.a, s.ixy, s.mxy), ax0, ay0);
    unpack2(fma2(near.b, s.ixy, s.mxy), ax1, ay1);
    unpack2(fma2(near.c, s.ixy, s.mxy), ax2, ay2);
    unpack2(fma2(near.d, s.ixy, s.mxy), ax3, ay3);
    unpack2(fma2(both.a, s.iz, s.mz), az0, az1);
    unpack2(fma2(both.b, s.iz, s.mz), az2, az3);
    float bx0, bx1, bx2, bx3, by0, by1, by2, by3, bz0, bz1, bz2, bz3;
    unpack2(fma2(far.a, s.ixy, s.mxy), bx0, by0);
    unpack2(fma2(far.b, s.ixy, s.mxy), bx1, by1);
    unpack2(fma2(far.c, s.ixy, s.mxy), bx2, by2);
    unpack2(fma2(far.d, s.ixy, s.mxy), bx3, by3);
    unpack2(fma2(both.c, s.iz, s.mz), bz0, bz1);
    unpack2(fma2(both.d, s.iz, s.mz), bz2, bz3);
    // entries, kNone where the box is not passed
    float e0 = max3(ax0, ay0, fmaxf(az0, s.tmin)), e1 = max3(ax1, ay1, fmaxf(az1, s.tmin));
    float e2 = max3(ax2, ay2, fmaxf(az2, s.tmin)), e3 = max3(ax3, ay3, fmaxf(az3, s.tmin));
    e0 = e0 <= min3(bx0, by0, fminf(bz0, tcull)) ? e0 : kNone;
    e1 = e1 <= min3(bx1, by1, fminf(bz1, tcull)) ? e1 : kNone;
    e2 = e2 <= min3(bx2, by2, fminf(bz2, tcull)) ? e2 : kNone;
    e3 = e3 <= min3(bx3, by3, fminf(bz3, tcull)) ? e3 : kNone;
    // entries of the two groups' own boxes, kNone where no slot is passed
    float ga = max3(fminf(ax0, ax1), fminf(ay0, ay1), fmaxf(fminf(az0, az1), s.tmin));
    float gb = max3(fminf(ax2, ax3), fminf(ay2, ay3), fmaxf(fminf(az2, az3), s.tmin));
    // order inside each group
    const bool sa = e1 < e0, sb = e3 < e2;
    float a0 = fminf(e0, e1), a1 = fmaxf(e0, e1), b0 = fminf(e2, e3), b1 = fmaxf(e2, e3);
    const uint32_t qa0 = sa ? refs.y : refs.x, qa1 = sa ? refs.x : refs.y;
    const uint32_t qb0 = sb ? refs.w : refs.z, qb1 = sb ? refs.z : refs.w;
    ga = a0 < kNone ? ga : kNone;
    gb = b0 < kNone ? gb : kNone;
    // the groups: n near, f far
    const bool sg = gb < ga;
    const float n0 = sg ? b0 : a0, n1 = sg ? b1 : a1, f1 = sg ? a1 : b1;
    float f0 = sg ? a0 : b0;
    const uint32_t qn0 = sg ? qb0 : qa0, qn1 = sg ? qb1 : qa1, qf1 = sg ? qa1 : qb1;
    uint32_t qf0 = sg ? qa0 : qb0;
    if (kClosest) {
        if (f1 < kNone && (int)qf1 < 0) qf0 |= kWideMark;
        // a leaf that is the far child itself was tested just now, for good
        if (qf1 == kWideEmpty && (int)qf0 < 0) f0 = f0 < kNone ? 0.0f : kNone;
    }
    if (s.sp + 3 <= Stack::kShared) {  // all in shared memory: no branch per entry
        stack.push_if(f1 < kNone, s.sp, qf1, f1);
        stack.push_if(f0 < kNone, s.sp, qf0, f0);
        stack.push_if(n1 < kNone, s.sp, qn1, (int)qn1 < 0 ? 0.0f : n1);
    } else {
        if (f1 < kNone) stack.set(s.sp++, qf1, f1);
        if (f0 < kNone) stack.set(s.sp++, qf0, f0);
        if (n1 < kNone) stack.set(s.sp++, qn1, (int)qn1 < 0 ? 0.0f : n1);
    }
    s.ref = n0 < kNone ? qn0 : kWidePop;
}

// The rest of trav_leaf_phase's test, for a triangle whose cheap tests did not refuse it.
__device__ __forceinline__ bool accept_triangle(float det, float un, float vn, float tn, float tmin, float tcur,
                                                float &u, float &v, float &t) {
    const float inv_det = __frcp_rn(det);
    u = __fmul_rn(un, inv_det);
    v = __fmul_rn(vn, inv_det);
    t = __fmul_rn(tn, inv_det);
    return !(u < 0.0f || u > 1.0f || v < 0.0f || __fadd_rn(u, v) > 1.0f) && tmin < t && t < tcur;
}

// Tests the triangles of leaf s.ref.
template <bool kClosest>
__device__ __forceinline__ void wide_leaf(WideState &s, const BvhView &bvh, float4 r0, float4 r1) {
    const f32x2 dx2 = pack2(r0.w, r0.w), dy2 = pack2(r1.x, r1.x), dz2 = pack2(r1.y, r1.y);
    const f32x2 ndx2 = pack2(-r0.w, -r0.w), ndy2 = pack2(-r1.x, -r1.x), ndz2 = pack2(-r1.y, -r1.y);
    const f32x2 ox2 = pack2(r0.x, r0.x), oy2 = pack2(r0.y, r0.y), oz2 = pack2(r0.z, r0.z);
    const char *rec = bvh.wide_pairs + (uint64_t)(s.ref & kWideIndex) * kWidePairBytes;
    s.ref = kWidePop;
    for (;; rec += kWidePairBytes) {
        const Sector w0 = ldg_sector(rec), w1 = ldg_sector(rec + 32), w2 = ldg_sector(rec + 64);
        const f32x2 e1x = w0.d, e1y = w1.a, e1z = w1.b, e2x = w1.c, e2y = w1.d, e2z = w2.a;
        const f32x2 tvx = add2(ox2, w0.a), tvy = add2(oy2, w0.b), tvz = add2(oz2, w0.c);
        const f32x2 px = cross2(dy2, e2z, ndz2, e2y);
        const f32x2 py = cross2(dz2, e2x, ndx2, e2z);
        const f32x2 pz = cross2(dx2, e2y, ndy2, e2x);
        const f32x2 qx = cross2(tvy, e1z, neg2(tvz), e1y);
        const f32x2 qy = cross2(tvz, e1x, neg2(tvx), e1z);
        const f32x2 qz = cross2(tvx, e1y, neg2(tvy), e1x);
        const f32x2 det = dot2(e1x, e1y, e1z, px, py, pz), un = dot2(tvx, tvy, tvz, px, py, pz);
        const f32x2 vn = dot2(dx2, dy2, dz2, qx, qy, qz), tn = dot2(e2x, e2y, e2z, qx, qy, qz);
        const int slot = (int)(uint32_t)w2.b;
        const uint32_t flags = (uint32_t)(w2.b >> 32);
        // Signs first: with det > 0 and un < -1e-37 det the quotient u rounds to a negative number,
        // and so for v, and with un + vn > 1.00001 det u or u + v rounds above 1; in between the
        // division decides. (Most triangles end here; so does the padding of an odd leaf, det = 0.)
        float det0, det1, un0, un1, vn0, vn1, lo0, lo1, hi0, hi1, sum0, sum1;
        unpack2(det, det0, det1);
        unpack2(un, un0, un1);
        unpack2(vn, vn0, vn1);
        unpack2(mul2(det, pack2(-1e-37f, -1e-37f)), lo0, lo1);
        unpack2(mul2(det, pack2(1.00001f, 1.00001f)), hi0, hi1);
        unpack2(add2(un, vn), sum0, sum1);
        const bool m0 = det0 > 0.00001f && fminf(un0, vn0) >= lo0 && sum0 <= hi0;
        const bool m1 = det1 > 0.00001f && fminf(un1, vn1) >= lo1 && sum1 <= hi1;
        bool more = m0 || m1, first = m0;
        while (more) {  // one pass unless both are left
            float tn0, tn1, u, v, t;
            unpack2(tn, tn0, tn1);
            const bool hit = accept_triangle(first ? det0 : det1, first ? un0 : un1, first ? vn0 : vn1,
                                             first ? tn0 : tn1, s.tmin, s.t, u, v, t);
            if (hit) {
                s.t = t;
                s.u = u;
                s.v = v;
                s.addr = slot + (first ? 0 : 3);
                if (!kClosest) {
                    s.ref = kWideDone;
                    return;
                }
            }
            more = first && m1;
            first = false;
        }
        if (flags & kPairLast) return;
    }
}

__device__ __forceinline__ TraceResult wide_result(const WideState &s) {
    TraceResult res;
    res.addr = s.addr;
    res.t = s.t;
    res.u = s.u;
    res.v = s.v;
    return res;
}

// One ray through the tree, start to finish, on the given stack: the steps without the queue, which the CPU tests compare
// with the two-wide loop ray by ray (the kernels use trace_queue).
template <bool kClosest, class Stack>
__device__ __forceinline__ TraceResult traverse_wide(Stack &stack, const BvhView &bvh, float4 r0, float4 r1,
                                                     uint32_t &err) {
    WideState s;
    if (!wide_start(s, bvh, r0, r1)) return traverse_two_wide<kClosest>(bvh, r0, r1, err);
    while (s.ref != kWideDone) {
        while (s.ref < kWideMark) {
            wide_node<kClosest>(s, stack, bvh);
            wide_pop<kClosest>(s, stack);
        }
        if ((int)s.ref < 0) {
            wide_leaf<kClosest>(s, bvh, r0, r1);
            wide_pop<kClosest>(s, stack);
        }
    }
    return wide_result(s);
}

#if defined(__CUDACC__) || defined(TT_WARP_ON_HOST)  // (tests run it on emulated warps)
// Lanes at inner nodes below which a warp turns to its leaves and to new rays: 4M camera rays / 4M
// bounces on the 2,097,152-triangle terrain take 0.52 / 0.98 ms with 2, 0.50 / 0.90 with 4, 0.49 / 0.86
// with 8, 0.50 / 0.86 with 10, 0.53 / 0.89 with 16.
constexpr int kWideInner = 8;

// A warp's share of a ray queue. Every lane keeps a ray of its own. While at least kInner lanes
// stand at inner nodes they step on; then the lanes that wait at leaves test their triangles
// together, and where none does, the lanes whose rays are finished store them and take the queue's
// next ones (one claim; consecutive slots, so an ordered queue's neighbours start together).
// claim(first, count): the first of the `count` queue places that come to the warp (it may take fewer off them,
// by lowering count), all lanes taking part; places from n on do not exist; first: the warp's first
// claim. at(place): the slot in that place; fetch(slot, r0, r1): a slot's ray; store(lanes, slot,
// result): the lanes of `lanes` store together.
//
// Measured on 4M rays over a 2,097,152-triangle terrain against one warp-wide loop per 32 rays (each
// lane runs its own ray to its end): cosine bounces 0.86 against 1.05 ms, camera rays 0.49 against
// 0.54 ms; 18 of 32 lanes busy instead of 10.
template <bool kClosest, int kInner, class Stack, class Rays, class Claim, class At, class Fetch, class Store>
__device__ __forceinline__ void trace_queue(Stack &stack, Rays &rays, const BvhView &bvh, unsigned n, uint32_t &err,
                                            Claim claim, At at, Fetch fetch, Store store) {
    WideState s;
    s.ref = kWideIdle;
    unsigned slot = 0;
    unsigned left = n;  // rays that the queue may still have
    const unsigned warps = gridDim.x * blockDim.x / 32, few = min(n / warps, 3u);
    for (;;) {
        const unsigned inner = __ballot_sync(0xffffffffu, s.ref < kWideMark);
        if (__popc(inner) < kInner) {
            if (__any_sync(0xffffffffu, (int)s.ref < 0)) {
                if ((int)s.ref < 0) {
                    float4 r0, r1;
                    rays.get(fetch, slot, r0, r1);
                    wide_leaf<kClosest>(s, bvh, r0, r1);
                    wide_pop<kClosest>(s, stack);
                }
                continue;
            }
            const unsigned done = __ballot_sync(0xffffffffu, s.ref == kWideDone);
            if (s.ref == kWideDone) {
                store(done, slot, wide_result(s));
                s.ref = kWideIdle;
            }
            __syncwarp();
            if (left) {
                // no more than the warp's share of what is left, but a few
                const unsigned want = ~inner;
                unsigned count = min((unsigned)__popc(want), max(left / warps, few) + 1u);
                const unsigned base = claim(left == n, count);
                left = base < n && n - base > count ? n - base - count : 0;
                if (s.ref == kWideIdle) {
                    const unsigned off = __popc(want & ((1u << (threadIdx.x & 31)) - 1u));
                    if (off < count && base < n && off < n - base) {
                        slot = at(base + off);
                        float4 r0, r1;
                        fetch(slot, r0, r1);
                        rays.put(r0, r1);
                        if (!wide_start(s, bvh, r0, r1)) {
                            const TraceResult tr = traverse_two_wide<kClosest>(bvh, r0, r1, err);
                            s.t = tr.t;
                            s.u = tr.u;
                            s.v = tr.v;
                            s.addr = tr.addr;
                            s.ref = kWideDone;
                        }
                    }
                }
                continue;
            }
            if (!inner) break;
        }
        if (s.ref < kWideMark) {
            wide_node<kClosest>(s, stack, bvh);
            wide_pop<kClosest>(s, stack);
        }
    }
}
#endif

#if defined(__CUDACC__) || defined(TT_WARP_ON_HOST)
// A warp's share of a ray queue over the two-wide tree: 32 places at a time, a ray to a lane. For sets whose rays
// the four-wide loop mostly does not serve, and for trees without a four-wide form. sh: the lane's column of
// shared memory, kSh words at a stride of kStride; the rest as in trace_queue.
// The lanes meet at every pass of the outer loop: without that vote the compiler lets them part for longer (4M camera
// rays on the 2,097,152-triangle terrain 0.84 ms instead of 0.66; trace_warp_kernel alone takes 0.64).
template <bool kClosest, int kSh, int kStride, class Claim, class At, class Fetch, class Store>
__device__ __forceinline__ void two_wide_queue(int *sh, const BvhView &bvh, unsigned n, uint32_t &err, Claim claim, At at,
                                               Fetch fetch, Store store) {
    TravStack<kSh, kStride> stack;
    stack.sh = sh;
    for (bool first = true;; first = false) {
        unsigned count = 32;
        const unsigned base = claim(first, count), place = base + (threadIdx.x & 31);
        if (base >= n) break;
        const unsigned slot = place < n && place - base < count ? at(place) : n;
        const unsigned lanes = __ballot_sync(0xffffffffu, slot < n);
        TravState s;
        bool done = true;
        float4 r0{}, r1{};
        if (slot < n) {
            fetch(slot, r0, r1);
            trav_init(s, stack, r0, r1);
            done = false;
        }
        while (__any_sync(0xffffffffu, !done))
            if (!done) done = trav_iterate<kClosest, false>(s, stack, bvh, err, r1.w);
        if (slot < n) {
            TraceResult tr;
            tr.addr = s.addr;
            tr.t = s.t;
            tr.u = s.u;
            tr.v = s.v;
            store(lanes, slot, tr);
        }
        __syncwarp();
    }
}
#endif

// The pairs of the leaf whose triangles start at float4 slot `slot` of the compact vertex array.
// The edges are the differences trav_leaf_phase forms.
__device__ __forceinline__ void wide_fill_pairs(const float4 *verts, uint32_t slot, float *out) {
    for (bool last = false; !last; slot += 6, out += kWidePairBytes / 4) {
        float f[18];
        for (int i = 0; i < 18; i++) f[i] = 0.0f;
        float4 head = verts[slot];
        for (int k = 0; k < 2; k++) {
            if (__float_as_int(head.x) == (int)0x80000000) break;  // terminator: an empty leaf or second
            const float4 v1 = verts[slot + 3 * k + 1], v2 = verts[slot + 3 * k + 2];
            f[k] = -head.x;
            f[2 + k] = -head.y;
            f[4 + k] = -head.z;
            f[6 + k] = __fsub_rn(v1.x, head.x);
            f[8 + k] = __fsub_rn(v1.y, head.y);
            f[10 + k] = __fsub_rn(v1.z, head.z);
            f[12 + k] = __fsub_rn(v2.x, head.x);
            f[14 + k] = __fsub_rn(v2.y, head.y);
            f[16 + k] = __fsub_rn(v2.z, head.z);
            head = verts[slot + 3 * k + 3];
        }
        last = __float_as_int(head.x) == (int)0x80000000;
        for (int i = 0; i < 18; i++) out[i] = f[i];
        for (int i = 20; i < 24; i++) out[i] = 0.0f;
        out[18] = __int_as_float((int)slot);
        out[19] = __int_as_float(last ? (int)kPairLast : 0);
    }
}

}  // namespace tt
