// Launches that may start while the kernel before them in the stream drains
// (programmatic dependent launch): the grid is set up and its CTAs take the
// slots the last wave leaves free, then stop at pdl_wait() until every kernel
// before has completed and its writes are visible.  A kernel launched this way
// calls pdl_trigger() first (the next launch may be set up) and pdl_wait()
// before it touches anything another kernel writes or reads; chains of them
// stay ordered because each waits for the one before.  Between two launches of
// a few microseconds the launch itself is a third of the time (the 64^3 FP64
// step, some twenty launches: AAA us with plain launches, BBB so).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace x3d {

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                              A &&...args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace x3d
