// Boundary rows of the non-periodic first derivatives, shared by the
// one-thread-per-line kernels (linesolve.cu) and the chunked ones
// (linesolve_walls.cu).
#pragma once

#include "x3d_internal.h"

namespace x3d {

// Right-hand side at the first two and last two points of a non-periodic
// first-derivative line (der?_ij, src/x3d_derive.f90:171-210): v is the same
// 9-point window (v[k] = u_{i-4+k}; entries past the line's ends are never
// used here).  Free slip (ncl = 1) mirrors the field (npaire = 1: even, so
// the derivative vanishes at the wall; npaire = 0: odd); Dirichlet (ncl = 2)
// uses the one-sided closures.  Other points keep the interior stencil r.
template <typename T>
__device__ __forceinline__ T der_closure(int i, int n, const T *v, const LineOp<T> &op, T r)
{
    const T a = op.a, b = op.b;
    if (i == 0) {
        if (op.ncl1 == 1) return op.npaire == 1 ? T(0) : a * (v[5] + v[5]) + b * (v[6] + v[6]);
        return op.cl[0] * v[4] + op.cl[1] * v[5] + op.cl[2] * v[6];
    }
    if (i == 1) {
        if (op.ncl1 == 1)
            return op.npaire == 1 ? a * (v[5] - v[3]) + b * (v[6] - v[4]) : a * (v[5] - v[3]) + b * (v[6] + v[4]);
        return op.cl[3] * (v[5] - v[3]);
    }
    if (i == n - 2) {
        if (op.ncln == 1)
            return op.npaire == 1 ? a * (v[5] - v[3]) + b * (v[4] - v[2]) : a * (v[5] - v[3]) + b * ((-v[4]) - v[2]);
        return op.cl[4] * (v[5] - v[3]);
    }
    if (i == n - 1) {
        if (op.ncln == 1) return op.npaire == 1 ? T(0) : a * ((-v[3]) - v[3]) + b * ((-v[2]) - v[2]);
        return -op.cl[5] * v[4] - op.cl[6] * v[3] - op.cl[7] * v[2];
    }
    return r;
}

}  // namespace x3d
