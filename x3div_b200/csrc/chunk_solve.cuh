// Device code of the chunked line solves shared by the stage kernels
// (linesolve_chunk.cu and linesolve_batch.cu: TMA and bulk-copied tiles; linesolve_any.cu: tiles of
// any extent and alignment): stencils on a chunk's window, the chunk solve
// with its two carry exchanges, the accumulator and the flushes of y/z
// chunks.  The solve itself is described at the top of linesolve_chunk.cu.
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "linesolve_chunk.h"
#include "ptx.cuh"
#include "x3d_internal.h"

namespace x3d {

// Two x-adjacent y/z lines' values in one 64-bit register pair, computed with
// the packed FP32 instructions of sm_100: per lane the same IEEE operations
// (round-to-nearest add, multiply, fused multiply-add) as the scalar code,
// for half the instructions.
struct F2 {
    float2 v;
    F2() = default;
    __device__ __forceinline__ explicit F2(float s) : v(make_float2(s, s)) {}
    __device__ __forceinline__ explicit F2(float2 x) : v(x) {}
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
// a - b as b * (-1) + a: one rounding of the exact difference, as a subtraction
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 &operator+=(F2 &a, F2 b) { return a = a + b; }
// fma for the scalar types too, so that the unqualified calls below resolve
// to the exact overload inside this namespace
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ float fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma(double a, double b, double c) { return ::fma(a, b, c); }

// Value type of a stage kernel that carries PR lines per thread.
template <typename T, int PR>
struct PairOf {
    using type = T;
};
template <>
struct PairOf<float, 2> {
    using type = F2;
};

// PR consecutive values of U (one per line of a pair), as one load or store.
template <typename U, int PR>
struct Lanes {
    using type = U;
};
template <>
struct Lanes<float, 2> {
    using type = float2;
};
template <>
struct Lanes<double, 2> {
    using type = double2;
};

// Launch bounds of the stage kernels: up to 512 threads with the registers
// of one such CTA per SM (128 per thread), so that no configuration spills
// its chunk; a paired kernel with long chunks keeps twice the values per
// thread and is limited to 256 threads.
template <typename T, int L, int PR>
constexpr int kStageThreads = PR == 2 && L == kChunkLong<T> ? 256 : 512;

// RHS scalars of a stencil (the operator's, times 1 + rho^2).
template <typename T>
struct Coef {
    T a, b, c, d;
};

template <int KIND, typename T>
__device__ __forceinline__ T stencil_at(const T *v, const Coef<T> &k)
{
    // v[m] = u_{i-4+m}.  The terms are added from the smallest up, so that only
    // the last fused multiply-add rounds at the size of the result (FP32
    // interpolation at 512 points: 0.85e-6 of the result against 1.1e-6 with
    // the largest term first).
    if constexpr (KIND == DER) return fma(k.a, v[5] - v[3], k.b * (v[6] - v[2]));
    if constexpr (KIND == DER2)
        return fma(k.a, (v[5] - v[4]) - (v[4] - v[3]), k.b * ((v[6] - v[4]) - (v[4] - v[2])));
    if constexpr (KIND == DERVP) return fma(k.a, v[5] - v[4], k.b * (v[6] - v[3]));
    if constexpr (KIND == DERPV) return fma(k.a, v[4] - v[3], k.b * (v[5] - v[2]));
    if constexpr (KIND == INTVP)
        return fma(k.a, v[5] + v[4], fma(k.b, v[6] + v[3], fma(k.c, v[7] + v[2], k.d * (v[8] + v[1]))));
    if constexpr (KIND == INTPV)
        return fma(k.a, v[4] + v[3], fma(k.b, v[5] + v[2], fma(k.c, v[6] + v[1], k.d * (v[7] + v[0]))));
    return v[4];
}

// r[OFF + j] for j < N from a window w of N + 8 values (w[m] = u_{OFF+j-4+m}).
template <int KIND, typename T, int N, int L, int OFF>
__device__ __forceinline__ void chunk_stencil(const T (&w)[N + 8], T (&r)[L], const Coef<T> &k)
{
#pragma unroll
    for (int j = 0; j < N; ++j) r[OFF + j] = stencil_at<KIND>(w + j, k);
}

template <typename T, int N, int L, int OFF, typename S>
__device__ __forceinline__ void chunk_stencil_kind(int kind, const T (&w)[N + 8], T (&r)[L],
                                                   const LineOp<S> &op)
{
    const Coef<T> k{T(op.ca), T(op.cb), T(op.cc), T(op.cd)};
    switch (kind) {
    case DER: chunk_stencil<DER, T, N, L, OFF>(w, r, k); break;
    case DER2: chunk_stencil<DER2, T, N, L, OFF>(w, r, k); break;
    case DERVP: chunk_stencil<DERVP, T, N, L, OFF>(w, r, k); break;
    case DERPV: chunk_stencil<DERPV, T, N, L, OFF>(w, r, k); break;
    case INTVP: chunk_stencil<INTVP, T, N, L, OFF>(w, r, k); break;
    case INTPV: chunk_stencil<INTPV, T, N, L, OFF>(w, r, k); break;
    default: chunk_stencil<IDENT, T, N, L, OFF>(w, r, k); break;
    }
}

// The explicit right-hand side of a whole chunk, in P parts of L/P points,
// each from its own window of L/P + 8 staged values, so that only one part's
// window is live next to r.  load(w, J0) fills w[m] = u_{cs+J0-4+m}.
template <typename T, int L, int P, int I = 0, typename Load, typename S>
__device__ __forceinline__ void chunk_rhs(int kind, const Load &load, T (&r)[L], const LineOp<S> &op)
{
    if constexpr (I < P) {
        constexpr int N = L / P;
        {
            T w[N + 8];
            load(w, std::integral_constant<int, I * N>{});
            chunk_stencil_kind<T, N, L, I * N>(kind, w, r, op);
        }
        chunk_rhs<T, L, P, I + 1>(kind, load, r, op);
    }
}

// Staged lines carry periodic halos, so a chunk's window never wraps:
// shared-memory row (y/z tiles) or element (x rows) kHalo + i holds point i
// of the line for -4 <= i < n + 4, and the rows past that up to the end of
// the last chunk's window exist but hold values that are never used.
constexpr int kHalo = 4;

constexpr uint64_t kChunkWaitNs = 2000000000ull;  // bounded waits on a tile's copies: 2 s

// Fills the halos of ntiles staged y/z tiles of W columns whose point i sits
// in row h0 + i: rows h0-4 .. h0-1 from points n-4 .. n-1, rows h0+n ..
// h0+n+3 from points 0 .. 3.
template <typename T>
__device__ __forceinline__ void fill_halos_yz(unsigned char *base, size_t tile_bytes, int ntiles, int n, int W,
                                              int h0)
{
    const int per = 8 * W;
    for (int i = threadIdx.x; i < per * ntiles; i += blockDim.x) {
        const int ti = i / per, r = i - ti * per;
        const int h = r / W, x = r - h * W;
        T *tp = reinterpret_cast<T *>(base + ti * tile_bytes);
        const int dst = h < 4 ? h0 - 4 + h : h0 + n + h - 4;
        const int src = h < 4 ? h0 + n - 4 + h : h0 + h - 4;
        tp[dst * W + x] = tp[src * W + x];
    }
}

// 16-byte vector of T.
template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
    static constexpr int N = 4;
    using type = float4;
};
template <>
struct Vec4<double> {
    static constexpr int N = 2;
    using type = double2;
};
template <>
struct Vec4<F2> {
    static constexpr int N = 2;
    using type = float4;
};

// Fills the halos of ntiles staged x tiles of `rows` padded rows whose
// point i sits at element kHalo + i: elements 0 .. 3 from points n-4 .. n-1,
// elements n+4 .. n+7 from points 0 .. 3, moved as 16-byte vectors.
template <typename T>
__device__ __forceinline__ void fill_halos_x(unsigned char *base, size_t tile_bytes, int ntiles, int rows,
                                             int pitch, int n)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    constexpr int per_row = 8 / V;
    const int per = rows * per_row;
    for (int i = threadIdx.x; i < per * ntiles; i += blockDim.x) {
        const int ti = i / per, r = i - ti * per;
        const int rr = r / per_row, h = (r - rr * per_row) * V;
        T *row = reinterpret_cast<T *>(base + ti * tile_bytes) + (size_t)rr * pitch;
        const int dst = h < 4 ? h : n + h;
        const int src = h < 4 ? n + h : h;
        *reinterpret_cast<VT *>(row + dst) = *reinterpret_cast<const VT *>(row + src);
    }
}

// Scratch in shared memory after the input tiles: per (chunk, line) the
// forward end value and the backward start value of the local sweeps.
template <typename T>
struct ChunkScratch {
    T *fz, *bz;
};

// Carry into chunk c: the end values e of the chunks before it (STEP = 1,
// forward sweep) or the start values of the chunks after it (STEP = -1,
// backward), folded from the farthest in over depth chunks, or over the
// whole line once and scaled by 1 / (1 - rho^n).  A chunk propagates an
// incoming carry by rho^L (rho^nv for the last, possibly short, chunk); the
// first chunk folded multiplies zero, so only a later visit to chunk C-1
// needs its own multiplier.  The visits run as at most two unwrapped
// segments of e.
template <typename T, int STEP>
__device__ __forceinline__ T chunk_carry(const T *e, int K, T mf, T ml, T wrap, int W, int l, int c, int C)
{
    const bool full = K >= C;
    T carry = T(0);
    if (STEP == 1) {
        int s = full ? c : c - K;
        s = s < 0 ? s + C : s;
        const int n1 = min(K, C - s);  // chunks s .. s+n1-1, then 0 .. K-n1-1
        const T *p = e + s * W + l;
#pragma unroll 4
        for (int k = 1; k < n1; ++k, p += W) carry = fma(mf, carry, *p);
        carry = fma(s + n1 == C ? ml : mf, carry, *p);
        p = e + l;
#pragma unroll 4
        for (int k = n1; k < K; ++k, p += W) carry = fma(mf, carry, *p);
    } else {
        int s = full ? c : c + K;
        s = s >= C ? s - C : s;
        const int n1 = min(K, s + 1);  // chunks s .. s-n1+1, then C-1 .. C-K+n1
        const T *p = e + s * W + l;
#pragma unroll 4
        for (int k = 0; k < n1; ++k, p -= W) carry = fma(mf, carry, *p);
        if (K > n1) {
            p = e + (C - 1) * W + l;
            carry = fma(ml, carry, *p);
            p -= W;
#pragma unroll 4
            for (int k = n1 + 1; k < K; ++k, p -= W) carry = fma(mf, carry, *p);
        }
    }
    return full ? carry * wrap : carry;
}

// Shared-memory copy of the carry responses of a stage's operators, laid
// out [operator][4][L] (see StageOp::resp), made once per CTA.
template <typename V, int L, typename S>
__device__ __forceinline__ void load_resp(const StageProgram<S> &prog, V *dst)
{
    const int total = prog.nops * 4 * L;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int k = i / (4 * L), rem = i - k * 4 * L, a = rem / L, j = rem - a * L;
        dst[i] = V(prog.ops[k].resp[a][j]);
    }
}

// Solves one operator for one chunk; the solved values end in r[] (chunk
// local).  load(w, J0) fills a window u[cs+J0-4 ...] of the size of w from the
// staged line and its periodic halos; nv = points of the chunk inside the
// line (L except for the last chunk of a ragged line).  The carry fixes are
// folded into two precomputed responses: both local sweeps run before the
// first barrier (the backward one on the local forward values), and since
// the solve is linear,
//   y_j = y_j(local) + F h_j + B g_j,
//   h_j = sum_{m=j}^{len-1} rho^(2m-j+1),   g_j = rho^(len-j),
// with F the true v just before the chunk and B the true y just after it.
// The chunk's start value for the backward scan is y_0(local) + F h_0, so
// each thread publishes it after finding its own F.  h and g (resp[0..1],
// or resp[2..3] for a short last chunk) come from this operator's block of
// the shared-memory copy as 16-byte vectors, so each fix is one fused
// multiply-add per carry and half a load per point.
//
// keep = nh | ng << 8 (full chunks): the fixes by h_j for j >= nh and by
// g_j for j < L - ng are dropped, their responses being below 2^-32 (FP32)
// or 2^-62 (FP64) of the largest, far under the sweep's rounding (for the
// first derivative, rho = -0.38, that is all h past the 24th point and all g
// before the 8th; operators with |rho| < 0.2 keep half of each).  They go in
// blocks of 8 points, chosen by tests uniform across the CTA.
// Only kernels whose registers allow it (TRIM) compile the trimmed form.
template <typename T, int L, bool TRIM = false, typename Load, typename S>
__device__ __forceinline__ void chunk_solve_resp(const LineOp<S> &op, int kind, const T *resp, const Load &load,
                                                 T (&r)[L], const ChunkScratch<T> &sc, int W, int l, int c,
                                                 int C, int nv, int q, int keep = 0)
{
    constexpr int ti = L == kChunkLong<S> ? 0 : 1;
    // operator fields into registers once (the parameters are read through
    // a generic pointer, and would be read again after every barrier)
    const T rho = T(op.rho), mf = T(op.mfull[ti]), ml = T(op.mlast[ti]), wrap = T(op.wrap);
    const int K = op.depth[ti];
    chunk_rhs<T, L, 2>(kind, load, r, op);
    // local forward sweep; the chunk's end value goes straight to shared
    // memory (for a short last chunk, the value at point nv - 1, captured in
    // the sweep: selecting it from r afterwards would index r at run time
    // and move the whole array to local memory)
    T v = T(0);
    if (nv == L) {
#pragma unroll
        for (int j = 0; j < L; ++j) {
            v = fma(rho, v, r[j]);
            r[j] = v;
        }
        sc.fz[q] = v;
    } else {
#pragma unroll
        for (int j = 0; j < L; ++j) {
            v = fma(rho, v, r[j]);
            if (j + 1 == nv) sc.fz[q] = v;
            r[j] = j < nv ? v : T(0);
        }
    }
    T y = T(0);
#pragma unroll
    for (int j = L - 1; j >= 0; --j) {
        y = fma(rho, y, r[j]);
        r[j] = y;
    }
    __syncthreads();
    const T F = chunk_carry<T, 1>(sc.fz, K, mf, ml, wrap, W, l, c, C);
    const T *h = resp + (nv == L ? 0 : 2 * L);
    const T *g = h + L;
    sc.bz[q] = fma(F, h[0], y);
    __syncthreads();
    const T B = chunk_carry<T, -1>(sc.bz, K, mf, ml, wrap, W, l, c, C);
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    const int nh = keep & 0xff, ng = keep >> 8;
    if (TRIM && nv == L && keep && (nh < L || ng < L)) {
        constexpr int B8 = L < 8 ? L : 8;
#pragma unroll
        for (int j0 = 0; j0 < L; j0 += B8) {
            const bool dh = j0 < nh, dg = j0 + B8 > L - ng;
            if (dh && dg) {
#pragma unroll
                for (int j = j0; j < j0 + B8; j += V) {
                    const VT hv = *reinterpret_cast<const VT *>(h + j);
                    const VT gv = *reinterpret_cast<const VT *>(g + j);
                    const T *he = reinterpret_cast<const T *>(&hv);
                    const T *ge = reinterpret_cast<const T *>(&gv);
#pragma unroll
                    for (int v = 0; v < V; ++v) r[j + v] = fma(F, he[v], fma(B, ge[v], r[j + v]));
                }
            } else if (dh) {
#pragma unroll
                for (int j = j0; j < j0 + B8; j += V) {
                    const VT hv = *reinterpret_cast<const VT *>(h + j);
                    const T *he = reinterpret_cast<const T *>(&hv);
#pragma unroll
                    for (int v = 0; v < V; ++v) r[j + v] = fma(F, he[v], r[j + v]);
                }
            } else if (dg) {
#pragma unroll
                for (int j = j0; j < j0 + B8; j += V) {
                    const VT gv = *reinterpret_cast<const VT *>(g + j);
                    const T *ge = reinterpret_cast<const T *>(&gv);
#pragma unroll
                    for (int v = 0; v < V; ++v) r[j + v] = fma(B, ge[v], r[j + v]);
                }
            }
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < L; j += V) {
        const VT hv = *reinterpret_cast<const VT *>(h + j);
        const VT gv = *reinterpret_cast<const VT *>(g + j);
        const T *he = reinterpret_cast<const T *>(&hv);
        const T *ge = reinterpret_cast<const T *>(&gv);
#pragma unroll
        for (int v = 0; v < V; ++v) r[j + v] = fma(F, he[v], fma(B, ge[v], r[j + v]));
    }
}

template <typename T>
__device__ __forceinline__ ChunkScratch<T> carve_scratch(unsigned char *base, int C, int W)
{
    ChunkScratch<T> sc;
    T *t = reinterpret_cast<T *>(base);
    sc.fz = t;
    sc.bz = t + C * W;
    return sc;
}

// acc (+)= m * r, with m = 1 or the staged tile value at the point;
// tile_at(ti, j) returns TV consecutive tile values from point j (a 16-byte
// vector along an x row, one value per point down a y/z column).
template <typename T, int L, int TV, typename S, typename TileAt>
__device__ __forceinline__ void accumulate(const StageOp<S> &so, T (&acc)[L], const T (&r)[L],
                                           int nv, const TileAt &tile_at)
{
    if (so.mul_tile < 0) {
        if (so.accumulate) {
#pragma unroll
            for (int j = 0; j < L; ++j) acc[j] += r[j];
        } else {
#pragma unroll
            for (int j = 0; j < L; ++j) acc[j] = r[j];
        }
    } else if (so.accumulate) {
        // points past a short chunk's end read staged halo/padding rows and
        // are never stored
#pragma unroll
        for (int j = 0; j < L; j += TV) {
            const auto tv = tile_at(so.mul_tile, j);
            const T *te = reinterpret_cast<const T *>(&tv);
#pragma unroll
            for (int v = 0; v < TV; ++v) acc[j + v] = fma(te[v], r[j + v], acc[j + v]);
        }
    } else {
#pragma unroll
        for (int j = 0; j < L; j += TV) {
            const auto tv = tile_at(so.mul_tile, j);
            const T *te = reinterpret_cast<const T *>(&tv);
#pragma unroll
            for (int v = 0; v < TV; ++v) acc[j + v] = te[v] * r[j + v];
        }
    }
}

// Flush fields of a stage operator, read from the parameters once per
// flush rather than at every store.
template <typename T>
struct FlushArgs {
    void *out;
    const void *base;
    void *out2;
    const void *base2;
    double sign, scale2;
    bool f64, plain;
    const T *b2s;  // base2 from a staged tile: this thread's point cs there, or null
    int b2step;    // elements between consecutive points of the line in that tile
    __device__ FlushArgs(const StageOp<T> &so, const T *b2s_ = nullptr, int b2step_ = 1)
        : out(so.out), base(so.base), out2(so.out2), base2(so.base2), sign(so.sign), scale2(so.scale2),
          f64(so.out_f64 != 0), b2s(b2s_), b2step(b2step_)
    {
        plain = !base && !out2 && !f64 && sign == 1.0;
    }
};

// General flush of a y/z chunk in blocks of up to 8 points: every load of a
// block (base, base2) is issued before its stores.  base and base2 are often
// the output arrays themselves (du += ..., u = u + dt du in place), so a load
// placed after a store could not be moved ahead of it, and each point would
// wait for memory in turn.  V holds PR x-adjacent lines (PR = 1 or 2), moved
// as one PR-wide load or store of U.
template <typename T, typename V, typename U, int L>
__device__ __forceinline__ void flush_yz_blocked(const FlushArgs<T> &fa, const V (&res)[L], size_t obase,
                                                 size_t ostride, int nv)
{
    constexpr int PR = sizeof(V) / sizeof(T);
    using UP = typename Lanes<U, PR>::type;
    constexpr int B = L < 8 ? L : 8;
    const U *base = static_cast<const U *>(fa.base);
    const U *base2 = static_cast<const U *>(fa.base2);
    U *out = static_cast<U *>(fa.out);
    U *out2 = static_cast<U *>(fa.out2);
    const U sign = (U)fa.sign, scale2 = (U)fa.scale2;
#pragma unroll
    for (int j0 = 0; j0 < L; j0 += B) {
        UP bv[B], b2v[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const size_t p = obase + (size_t)(j0 + i) * ostride;
            const bool in = j0 + i < nv;
            bv[i] = base && in ? *reinterpret_cast<const UP *>(base + p) : UP{};
            if constexpr (std::is_same<T, U>::value) {
                if (fa.b2s) b2v[i] = *reinterpret_cast<const UP *>(fa.b2s + (j0 + i) * fa.b2step);
                else b2v[i] = base2 && in ? *reinterpret_cast<const UP *>(base2 + p) : UP{};
            } else {
                b2v[i] = base2 && in ? *reinterpret_cast<const UP *>(base2 + p) : UP{};
            }
        }
#pragma unroll
        for (int i = 0; i < B; ++i) {
            if (j0 + i < nv) {
                const size_t p = obase + (size_t)(j0 + i) * ostride;
                const T *rv = reinterpret_cast<const T *>(&res[j0 + i]);
                const U *bl = reinterpret_cast<const U *>(&bv[i]);
                const U *b2l = reinterpret_cast<const U *>(&b2v[i]);
                UP o;
                U *ol = reinterpret_cast<U *>(&o);
#pragma unroll
                for (int e = 0; e < PR; ++e) ol[e] = bl[e] + sign * (U)rv[e];
                *reinterpret_cast<UP *>(out + p) = o;
                if (out2) {
                    UP o2;
                    U *o2l = reinterpret_cast<U *>(&o2);
#pragma unroll
                    for (int e = 0; e < PR; ++e) o2l[e] = b2l[e] + scale2 * ol[e];
                    *reinterpret_cast<UP *>(out2 + p) = o2;
                }
            }
        }
    }
}

// The general flush of a whole chunk (nv == L) in the forms the Euler-step
// stages use, with every test hoisted out of the point loop and the
// addresses stepped by pointer increments:
//   HB:  out = base + sign * res (else out = sign * res)
//   B2T: out2 = base2 + scale2 * out, base2 read from the staged tile b2s
// U = double writes FP64 outputs.
template <typename T, typename V, typename U, int L, bool HB, bool B2T>
__device__ __forceinline__ void flush_yz_whole(const FlushArgs<T> &fa, const V (&res)[L], size_t obase,
                                               size_t ostride)
{
    constexpr int PR = sizeof(V) / sizeof(T);
    using UP = typename Lanes<U, PR>::type;
    constexpr int B = L < 8 ? L : 8;
    const U *bp = static_cast<const U *>(fa.base) + obase;
    U *op = static_cast<U *>(fa.out) + obase;
    U *op2 = static_cast<U *>(fa.out2) + obase;
    const T *b2p = fa.b2s;
    const int b2step = fa.b2step;
    const U sign = (U)fa.sign, scale2 = (U)fa.scale2;
#pragma unroll
    for (int j0 = 0; j0 < L; j0 += B) {
        UP bv[B];
        if constexpr (HB) {
#pragma unroll
            for (int i = 0; i < B; ++i) bv[i] = *reinterpret_cast<const UP *>(bp + (size_t)i * ostride);
            bp += (size_t)B * ostride;
        }
#pragma unroll
        for (int i = 0; i < B; ++i) {
            const T *rv = reinterpret_cast<const T *>(&res[j0 + i]);
            UP o;
            U *ol = reinterpret_cast<U *>(&o);
            if constexpr (HB) {
                const U *bl = reinterpret_cast<const U *>(&bv[i]);
#pragma unroll
                for (int e = 0; e < PR; ++e) ol[e] = bl[e] + sign * (U)rv[e];
            } else {
#pragma unroll
                for (int e = 0; e < PR; ++e) ol[e] = sign * (U)rv[e];
            }
            *reinterpret_cast<UP *>(op + (size_t)i * ostride) = o;
            if constexpr (B2T) {
                const V b2 = *reinterpret_cast<const V *>(b2p + (j0 + i) * b2step);
                const T *b2l = reinterpret_cast<const T *>(&b2);
                UP o2;
                U *o2l = reinterpret_cast<U *>(&o2);
#pragma unroll
                for (int e = 0; e < PR; ++e) o2l[e] = (U)b2l[e] + scale2 * ol[e];
                *reinterpret_cast<UP *>(op2 + (size_t)i * ostride) = o2;
            }
        }
        op += (size_t)B * ostride;
        if constexpr (B2T) op2 += (size_t)B * ostride;
    }
}

// Writes one thread's solved chunk of a y/z line, or of PR x-adjacent lines
// (points j < nv), each point ostride elements after the previous one.
// GENERAL = false: the program's flushes are all plain (out = res), and the
// other forms are not compiled into the kernel.
template <typename T, typename V, int L, bool GENERAL>
__device__ __forceinline__ void flush_yz(const FlushArgs<T> &fa, const V (&res)[L], size_t obase,
                                         size_t ostride, int nv)
{
    if (GENERAL && nv == L && !fa.plain) {
        // du += ...; du += ... with u = u + dt du; pp3 = ... in FP64
        const bool hb = fa.base != nullptr, o2 = fa.out2 != nullptr;
        if (!fa.f64 && hb && !o2) return flush_yz_whole<T, V, T, L, true, false>(fa, res, obase, ostride);
        if (!fa.f64 && hb && o2 && fa.b2s)
            return flush_yz_whole<T, V, T, L, true, true>(fa, res, obase, ostride);
        if (fa.f64 && !hb && !o2) return flush_yz_whole<T, V, double, L, false, false>(fa, res, obase, ostride);
    }
    if (!GENERAL || fa.plain) {
        T *dst = static_cast<T *>(fa.out) + obase;
        if (nv == L) {  // every chunk but a short last one: no per-point test
#pragma unroll
            for (int j = 0; j < L; ++j) {
                *reinterpret_cast<V *>(dst) = res[j];
                dst += ostride;
            }
        } else {
#pragma unroll
            for (int j = 0; j < L; ++j) {
                if (j < nv) *reinterpret_cast<V *>(dst) = res[j];
                dst += ostride;
            }
        }
    } else if constexpr (GENERAL) {
        if (fa.f64) flush_yz_blocked<T, V, double, L>(fa, res, obase, ostride, nv);
        else flush_yz_blocked<T, V, T, L>(fa, res, obase, ostride, nv);
    }
}

// Writes a solved y/z chunk one point further along its periodic line
// (StageOp::shift_out): obase is point cs, and the line's last point, which
// the thread of the last chunk holds, goes to its first.
template <typename T, typename V, int L>
__device__ __forceinline__ void flush_yz_shifted(void *shift_out, const V (&res)[L], size_t obase, int cs,
                                                 size_t ostride, int nv, bool last)
{
    T *const out = static_cast<T *>(shift_out);
    T *dst = out + obase + ostride;
    if (!last) {
#pragma unroll
        for (int j = 0; j < L; ++j, dst += ostride) *reinterpret_cast<V *>(dst) = res[j];
        return;
    }
#pragma unroll
    for (int j = 0; j < L; ++j, dst += ostride) {
        if (j + 1 < nv) *reinterpret_cast<V *>(dst) = res[j];
        else if (j + 1 == nv) *reinterpret_cast<V *>(out + obase - (size_t)cs * ostride) = res[j];
    }
}

// The same for a tile of x lines from its staging rows: element i of a row is
// read from i - 1.  Vectors of 16 bytes (VEC: n and the output are whole ones)
// take their first element from the lane before.
template <typename T, bool VEC>
__device__ __forceinline__ void flush_rows_shifted(void *shift_out, const T *out_s, long l0, int rows, int pitch,
                                                   int n)
{
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int rr = threadIdx.x >> 5; rr < rows; rr += nw) {
        const T *row = out_s + (size_t)rr * pitch;
        T *dst = static_cast<T *>(shift_out) + (size_t)(l0 + rr) * n;
        if constexpr (VEC) {
            using VT = typename Vec4<T>::type;
            constexpr int N = Vec4<T>::N;
            const int nvec = n / N;
            for (int q0 = 0; q0 < nvec; q0 += 32) {
                const int q = q0 + lane;
                VT v = *reinterpret_cast<const VT *>(row + (q < nvec ? q : 0) * N);
                T *e = reinterpret_cast<T *>(&v);
                T prev = __shfl_up_sync(0xffffffffu, e[N - 1], 1);
                if (lane == 0) prev = row[q ? q * N - 1 : n - 1];
#pragma unroll
                for (int i = N - 1; i > 0; --i) e[i] = e[i - 1];
                e[0] = prev;
                if (q < nvec) *reinterpret_cast<VT *>(dst + q * N) = v;
            }
        } else {
            for (int i = lane; i < n; i += 32) dst[i] = row[i ? i - 1 : n - 1];
        }
    }
}

// ---------------------------------------------------------------------------
// Host side.

// Carry responses of chunk_solve_resp for chunk length L on lines of n
// points: h_j = rho^(j+1) sum_{i < len-j} rho^(2i) and g_j = rho^(len-j),
// len = L (resp[0..1]) and len = the last chunk's length (resp[2..3]).
// Returns chunk_solve_resp's keep for full chunks: nh | ng << 8, the counts
// of leading h and trailing g entries above 2^-32 (FP32) or 2^-62 (FP64) of
// the largest, rounded up to whole blocks of 8.
template <typename T>
inline int fill_op_resp(T (&resp)[4][kChunkLong<T>], double al, int L, int n)
{
    const int C = (n + L - 1) / L, last = n - (C - 1) * L;
    const double rho = al == 0.0 ? 0.0 : -2.0 * al / (1.0 + std::sqrt(1.0 - 4.0 * al * al));
    double pw[kChunkLong<T>];
    double q = 1.0;
    for (int j = 0; j < kChunkLong<T>; ++j) pw[j] = (q *= rho);  // rho^(j+1)
    auto fill = [&](T *h, T *g, int len) {
        double S = 0.0, G = 1.0;
        for (int j = kChunkLong<T> - 1; j >= 0; --j) {
            if (j >= len) {
                h[j] = g[j] = T(0);
                continue;
            }
            S = 1.0 + rho * rho * S;
            G *= rho;
            h[j] = (T)(pw[j] * S);
            g[j] = (T)G;
        }
    };
    fill(resp[0], resp[1], L);
    fill(resp[2], resp[3], last);
    const double thr = sizeof(T) == 4 ? std::ldexp(1.0, -32) : std::ldexp(1.0, -62);
    double hmax = 0.0, gmax = 0.0;
    for (int j = 0; j < L; ++j) {
        hmax = std::max(hmax, std::fabs((double)resp[0][j]));
        gmax = std::max(gmax, std::fabs((double)resp[1][j]));
    }
    int nh = 0, ng = 0;
    for (int j = 0; j < L; ++j)
        if (std::fabs((double)resp[0][j]) > thr * hmax) nh = j + 1;
    for (int j = L - 1; j >= 0; --j)
        if (std::fabs((double)resp[1][j]) > thr * gmax) ng = L - j;
    const int b = L < 8 ? L : 8;
    nh = std::min(L, (nh + b - 1) / b * b);
    ng = std::min(L, (ng + b - 1) / b * b);
    return nh | ng << 8;
}

}  // namespace x3d
