// Plain C++ in the place of the CUDA intrinsics that the trace kernels use, so that the CPU tests can run the kernels
// themselves: a warp is 32 contexts that take turns, each running to its next warp-wide operation. Blocks are one
// warp and run one after another. Every warp-wide operation here is one of the whole warp.
#pragma once

#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#undef __noinline__
#undef __launch_bounds__
#undef __shared__
#define __noinline__
#define __launch_bounds__(...)
#define __shared__ static
#define TT_WARP_ON_HOST 1

static uint3 threadIdx, blockIdx;
static dim3 blockDim(32), gridDim(1);

namespace warp_host {
struct Lane {
    ucontext_t at;
    std::vector<char> stack;
    bool ended = false;
};
static Lane lanes[32];
static ucontext_t scheduler;
static uint32_t words[2][32];  // what each lane brought to this operation and to the last
static int phase[32];
static std::function<void()> body;

inline void entry() {
    body();
    lanes[threadIdx.x].ended = true;
}
// one value of every lane
inline const uint32_t *exchange(uint32_t mine) {
    const int lane = (int)threadIdx.x, p = phase[lane];
    words[p][lane] = mine;
    phase[lane] ^= 1;
    swapcontext(&lanes[lane].at, &scheduler);
    return words[p];
}
// a block of one warp
inline void run_warp() {
    for (int i = 0; i < 32; i++) {
        Lane &l = lanes[i];
        l.stack.resize(1 << 18);
        l.ended = false;
        phase[i] = 0;
        getcontext(&l.at);
        l.at.uc_stack.ss_sp = l.stack.data();
        l.at.uc_stack.ss_size = l.stack.size();
        l.at.uc_link = &scheduler;
        makecontext(&l.at, entry, 0);
    }
    for (int left = 32; left > 0;) {
        int ends = 0;
        for (int i = 0; i < 32; i++) {
            threadIdx.x = (unsigned)i;
            swapcontext(&scheduler, &lanes[i].at);
            ends += lanes[i].ended;
        }
        if (ends && ends != 32) {  // the lanes of a warp-wide operation did not all come to it
            fprintf(stderr, "warp_host: lanes parted\n");
            abort();
        }
        left -= ends;
    }
}
inline void run(unsigned blocks, std::function<void()> kernel) {
    body = kernel;
    gridDim = dim3(blocks);
    for (blockIdx.x = 0; blockIdx.x < blocks; blockIdx.x++) run_warp();
}
}  // namespace warp_host

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
static inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static inline unsigned __activemask() { return 0xffffffffu; }
static inline unsigned __ballot_sync(unsigned, bool p) {
    const uint32_t *w = warp_host::exchange(p);
    unsigned m = 0;
    for (int i = 0; i < 32; i++) m |= w[i] << i;
    return m;
}
static inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
static inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == 0xffffffffu; }
static inline void __syncwarp(unsigned = 0xffffffffu) { warp_host::exchange(0); }
template <class T> static inline T __shfl_sync(unsigned, T v, int from) {
    static_assert(std::is_integral<T>::value, "whole numbers");
    const uint32_t lo = warp_host::exchange((uint32_t)(uint64_t)v)[from];
    if (sizeof(T) == 4) return (T)lo;
    const uint32_t hi = warp_host::exchange((uint32_t)((uint64_t)v >> 32))[from];
    return (T)((uint64_t)hi << 32 | lo);
}
template <class T, class U> static inline T atomicAdd(T *p, U v) { const T old = *p; *p += (T)v; return old; }
template <class T> static inline T atomicOr(T *p, T v) { const T old = *p; *p |= v; return old; }
static inline unsigned max(unsigned a, unsigned b) { return a < b ? b : a; }
static inline unsigned min(unsigned a, unsigned b) { return a < b ? a : b; }
// the device's maximum and minimum: a NaN loses, +0 is above -0
static inline float dev_max(float a, float b) {
    if (a == b) return std::signbit(a) ? b : a;
    return std::fmax(a, b);
}
static inline float dev_min(float a, float b) {
    if (a == b) return std::signbit(a) ? a : b;
    return std::fmin(a, b);
}
