// Launches that may start while the kernel before them in the stream drains
// (programmatic dependent launch): the grid is set up and its CTAs take the
// slots the last wave leaves free, then stop at pdl_wait() until every kernel
// before has completed and its writes are visible.  A kernel launched this way
// calls pdl_trigger() first (the next launch may be set up) and pdl_wait()
// before it touches anything another kernel writes or reads; chains of them
// stay ordered because each waits for the one before.  Between two launches of
// a few microseconds the launch itself is a third of the time (the 64^3 FP64
// step, some twenty launches: 147 us with plain launches, 128 so).
//
// Launches of kPdlTiles tiles or more are plain: there the start is nothing, and
// CTAs of the next kernel that sit in the slots of the last ones cost about a
// hundredth (the 512^3 FP32 sweep 2277 us plain, 2301 so).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace x3d {

constexpr long kPdlTiles = 8192;

// tiles: the tiles of the launch's work, its CTAs unless it is persistent.
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kern)(P...), long tiles, unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
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
    cfg.numAttrs = tiles < kPdlTiles ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace x3d
