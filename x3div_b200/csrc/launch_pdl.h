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
// Launches of kPdlTiles tiles or more are plain.  Both ways measured, plain and
// dependent, in us: six y operators 128^3 FP32 17.5 and 14.6 (1024 tiles), 256^3
// 97.9 and 93.9 (4096), 384^3 315 and 316 (9216), 512^3 728 and 779 (16384: CTAs
// of the next kernel sit in slots that the last ones' would take); walls along y
// 128 x 129 x 128 FP32 16.7 and 13.2 (512), 512 x 257 x 512 303 and 299 (8192);
// the two updates of a step 112^3 FP32 13.0 and 12.1 (5488), 128^3 16.7 and 18.5
// (8192), FP64 112^3 20.7 and 17.7, 120^3 24.8 and 25.6; the pressure solve 128^3
// 51 and 47, 256^3 289 and 283, 512^3 2146 and 2139 (65536).  On odd rows one
// direction after another gains 2 to 25 % up to the line (FP64 y 129^3 24.8 and
// 18.9, 335^3 456 and 452); y, z and x by turns on a field about the size of L2
// lose by it what the order of the tiles leaves there (FP64 255^3 191 and 212, but
// 209^3 121 and 113, 271^3 423 and 417).
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
