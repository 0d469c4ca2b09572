// chain.cuh -- launches of a sequence of dependent kernels.
//
// Programmatic dependent launch: a kernel launched with chain() is made ready
// while the kernel before it in the stream still runs and waits in
// chain_begin() until that kernel is complete and its writes are visible, so
// that the gap between two launches is hidden.  The kernels do not let their
// successors onto the chip any earlier (a trigger at their start): the waiting
// CTAs then spread unevenly over the SMs, and strackw at W = 224 takes 28.7 ms
// instead of 27.4 (27.7 with plain launches).  The cull of 119 x 124 cells, 21
// launches, goes from 315 to 270 us, the 256 x 512 pair at window 32 from 251
// to 225, the 1024 x 2048 pair through strackw at W = 64 from 1.58 to 1.44 ms.
//
// Every kernel launched this way calls chain_begin() first, in every thread, so
// nothing is read or written before the earlier kernels are done.  What the
// kernel before it writes must not be promised to be read-only (__ldg, const
// __restrict__ kernel parameters): the promise holds for a kernel's lifetime,
// which begins before that write is done, and lets a load move above
// chain_begin().  Tables, images and what older kernels wrote are read-only for
// it.
// Where the operation before a launch is a copy, a memset or an event, full
// stream order applies with or without the attribute.  The plan, the records'
// first values, the stage selections and the complex stage always come after
// one and are launched plainly.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace sbk {

__device__ __forceinline__ void chain_begin() { cudaGridDependencySynchronize(); }

template <typename... P, typename... A>
inline cudaError_t chain(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args)
{
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace sbk
