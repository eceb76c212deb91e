// launch.cuh -- kernel launches on the library stream, each started as soon as the kernel before it
// ends.
//
// A kernel launched this way is set up while the one before it still runs (programmatic stream
// serialisation); its pdl_wait() holds it until that kernel has completed and its writes are visible,
// so the order of work is a plain stream's.  Every kernel launched through launch() calls pdl_wait()
// first, in every thread: a kernel that ended without it could end before its predecessor and let its
// successor start too early.  pdl_wait() returns a zero that the compiler cannot see through; kernels
// add it to the block index their addresses come from, so that no load of read-only data (__ldg, const
// __restrict__), which may move across the wait as far as the compiler knows, can be issued before it.
// No kernel lets its successor start before its own end: tried, the
// waiting blocks slowed the step at 11,000-30,000 atoms (mixed 14.6 -> 17.1 us at 27,436).
//
// Measured, us a step with its share of rebuilds, plain launches -> these: LJ mixed 256 atoms 9.5 -> 7.2,
// 16,384 14.1 -> 11.9, 131,072 37.1 -> 34.7; FP64 2,048 10.3 -> 8.0, 131,072 47.6 -> 44.7, half lists
// 90.8 -> 84.3 (three launches a step); contact DEM FP64 4,000 grains 21.8 -> 17.3, 260,800 58.7 -> 52.5
// (two launches a step).
#pragma once

#include <cuda_runtime.h>

#include "md_state.h"

namespace tmd {

__device__ __forceinline__ int pdl_wait() {
    int zero;
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero)::"memory");
    return zero;
}

template <class... P, class... A>
inline void launch(const State& s, unsigned grid, unsigned block, size_t shared, void (*kernel)(P...), A&&... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = shared;
    c.stream = s.stream;
    c.attrs = &at;
    // the default streams, by NULL or by their handles, keep plain launches
    c.numAttrs = s.stream && s.stream != cudaStreamLegacy && s.stream != cudaStreamPerThread ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace tmd
