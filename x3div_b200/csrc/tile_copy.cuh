// Copies of line tiles into shared memory by all threads of a CTA (cp.async),
// for fields that TMA boxes and bulk copies cannot move: any extent, any
// element-aligned address.  16-byte copies where the caller knows rows and
// addresses are whole 16-byte units.  The index arithmetic is pointer steps:
// with an index and a wrap test computed per element, the copy of a tile cost
// as many instructions as one operator's solve.
#pragma once

#include "ptx.cuh"

namespace x3d {

// Points 0 .. n-1 of `cols` <= W x-adjacent lines (src: the first line's first
// point, stride elements between points) to rows of W elements from dst.
template <int W, typename U>
__device__ __forceinline__ void copy_columns(U *dst, const U *src, size_t stride, int n, int cols, bool vec)
{
    constexpr int V = 16 / sizeof(U);
    const int t = threadIdx.x, nt = blockDim.x;
    if (vec) {
        constexpr int TPR = W / V;
        const int x = t % TPR * V, r0 = t / TPR, step = nt / TPR;
        if (x >= cols) return;
        const U *s = src + (size_t)r0 * stride + x;
        U *d = dst + r0 * W + x;
        const size_t ds = (size_t)step * stride;
#pragma unroll 4
        for (int r = r0; r < n; r += step, s += ds, d += step * W) cp_async<16>(d, s);
    } else {
        const int x = t % W, r0 = t / W, step = nt / W;
        if (x >= cols) return;
        const U *s = src + (size_t)r0 * stride + x;
        U *d = dst + r0 * W + x;
        const size_t ds = (size_t)step * stride;
#pragma unroll 4
        for (int r = r0; r < n; r += step, s += ds, d += step * W) cp_async<sizeof(U)>(d, s);
    }
}

// Rows of n consecutive points (src_pitch elements apart) to rows of dst_pitch.
template <typename U>
__device__ __forceinline__ void copy_rows(U *dst, int dst_pitch, const U *src, size_t src_pitch, int n, int rows,
                                          bool vec)
{
    constexpr int V = 16 / sizeof(U);
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int rr = threadIdx.x >> 5; rr < rows; rr += nw) {
        const U *s = src + (size_t)rr * src_pitch;
        U *d = dst + (size_t)rr * dst_pitch;
        if (vec) {
#pragma unroll 4
            for (int i = lane * V; i < n; i += 32 * V) cp_async<16>(d + i, s + i);
        } else {
#pragma unroll 4
            for (int i = lane; i < n; i += 32) cp_async<sizeof(U)>(d + i, s + i);
        }
    }
}

}  // namespace x3d
