// Chained launches: a kernel of a fixed sequence may be set up while its predecessor still drains.
//
// A render is a chain of short dependent kernels (960 x 540 x 16 samples of a deep scene: 726 launches), and
// between two plain launches of a stream the SMs stand idle for the launch's latency. With the
// programmatic-serialization attribute a kernel's blocks take the places the predecessor's blocks
// leave and wait in chain_begin() until the predecessor has completed and its writes are visible
// (512 x 512 x 16 samples of the Cornell box, 27 launches: 3.46 to 3.40 ms; letting the blocks in before
// the predecessor's end gives nothing more).
// Every kernel launched this way calls chain_begin() first, in every thread and before any return, so
// completion stays transitive along the chain. Data a predecessor wrote is read with plain loads (not
// through the read-only path, which gives no such promise).
#pragma once

#include <cuda_runtime.h>

namespace tt {

__device__ __forceinline__ void chain_begin() {
#if defined(__CUDACC__)
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// A plain launch that returns its own error (cudaGetLastError would also return what an earlier call of the
// caller's thread had left there).
template <class... P, class... A>
inline cudaError_t launch_plain(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace tt
