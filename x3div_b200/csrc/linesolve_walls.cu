// Non-periodic operators (der?_ij and the nclx = .false. staggered branches)
// as chunked line solves.
//
// Their factors vary along the line near the walls, so the circulant form of
// linesolve_chunk.cu does not apply, but the two sweeps of ?thomas_12
// (src/thomas.f90:61-84) are still affine in the value that enters a chunk:
//   z_i = r_i - s_i z_{i-1},   y_i = w_i z_i - fw_i y_{i+1}.
// A thread sweeps its chunk of kChunkLong points from zero both ways and the
// solution is y_i = y_i(local) + F H_i + B G_i, with F the true z before the
// chunk, B the true y after it, and H, G the responses of the chunk's values
// to them.  s, w, fw, H, G and each chunk's two multipliers are tables made
// once per operator in FP64 (build_wall_tables) and read through L1, where
// every lane of a chunk reads the same entries.
//
// Before, a line ran on one thread: 32-thread CTAs with a line each in shared
// memory (der), or straight from global memory, a warp's x lines in 32 rows at
// once (staggered).  The figures are at launch_wall.
#include <algorithm>

#include "chunk_solve.cuh"
#include "der_closure.cuh"
#include "launch_pdl.h"
#include "linesolve_chunk.h"
#include "ptx.cuh"
#include "tile_copy.cuh"
#include "x3d_internal.h"

namespace x3d {

// An operator's tables for chunks of L points, P = C L entries a row: s, w,
// fw, H, G, then the chunks' forward and backward multipliers.  depth: chunks
// a carry scan visits before the product of multipliers is below 1e-20
// (FP64) or 1e-12 (FP32).
template <typename T>
struct WallTables {
    const T *s, *w, *fw, *h, *g, *mf, *mb;
    int depth;
};

// Point k of a line of n_in points, where the staggered stencils reach past
// its ends: refl 0 mirrors (vp: about the end points, else half a cell out),
// 1 takes 2 u(end) - mirrored (vp only), as ls_np_stag; the derivative's
// closures never read past the ends, so any value does there.
__device__ __forceinline__ int reflected(int k, int n_in, bool vp)
{
    if (k < 0) return vp ? -k : -1 - k;
    if (k >= n_in) return vp ? 2 * (n_in - 1) - k : 2 * n_in - 1 - k;
    return k;
}

// One point of a tile from global memory (src: the line's first point).
template <typename T>
__device__ __forceinline__ void stage_point(T *dst, const T *src, size_t stride, int k, int n_in, bool vp, int refl)
{
    const int q = reflected(k, n_in, vp);
    if (refl == 0 || q == k) {
        cp_async<sizeof(T)>(dst, src + (size_t)q * stride);
    } else {
        const T e = src[(size_t)(k < 0 ? 0 : n_in - 1) * stride];
        *dst = (e + e) - src[(size_t)q * stride];
    }
}

// Solves one chunk: r holds the right-hand side on entry and y on return.
// Points past a short last chunk's end are zeroed and have zero factors in the
// tables, so the sweeps need no test per point; no chunk takes the last one's
// forward end value.
template <typename T, int L>
__device__ __forceinline__ void wall_solve(const WallTables<T> &tb, T (&r)[L], const ChunkScratch<T> &sc, int W, int l,
                                           int c, int C, int nv, int q)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    const int cs = c * L;
    if (nv < L) {
#pragma unroll
        for (int j = 0; j < L; ++j) r[j] = j < nv ? r[j] : T(0);
    }
    T z = T(0), y = T(0);
#pragma unroll
    for (int j = 0; j < L; j += V) {
        const VT sv = __ldg(reinterpret_cast<const VT *>(tb.s + cs + j));
        const T *se = reinterpret_cast<const T *>(&sv);
#pragma unroll
        for (int v = 0; v < V; ++v) r[j + v] = z = fma(-se[v], z, r[j + v]);
    }
    sc.fz[q] = z;
    // the smaller product (|fw| < w) is the one rounded by itself: FP32 derxvp
    // of 256 points has a 2-norm error of 4.99e-8 so, 5.54e-8 with w z rounded
    // first, which would be off the chain from y to y (free-slip box 337 us
    // against 345; channel 92.8 against 92.0)
#pragma unroll
    for (int j = L - V; j >= 0; j -= V) {
        const VT wv = __ldg(reinterpret_cast<const VT *>(tb.w + cs + j));
        const VT fv = __ldg(reinterpret_cast<const VT *>(tb.fw + cs + j));
        const T *we = reinterpret_cast<const T *>(&wv), *fe = reinterpret_cast<const T *>(&fv);
#pragma unroll
        for (int v = V - 1; v >= 0; --v) r[j + v] = y = fma(r[j + v], we[v], -fe[v] * y);
    }
    __syncthreads();
    T F = T(0);
    for (int k = max(0, c - tb.depth); k < c; ++k) F = fma(__ldg(tb.mf + k), F, sc.fz[k * W + l]);
    sc.bz[q] = fma(F, __ldg(tb.h + cs), y);
    __syncthreads();
    T B = T(0);
    for (int k = min(C - 1, c + tb.depth); k > c; --k) B = fma(__ldg(tb.mb + k), B, sc.bz[k * W + l]);
#pragma unroll
    for (int j = 0; j < L; j += V) {
        const VT hv = __ldg(reinterpret_cast<const VT *>(tb.h + cs + j));
        const VT gv = __ldg(reinterpret_cast<const VT *>(tb.g + cs + j));
        const T *he = reinterpret_cast<const T *>(&hv), *ge = reinterpret_cast<const T *>(&gv);
#pragma unroll
        for (int v = 0; v < V; ++v) r[j + v] = fma(F, he[v], fma(B, ge[v], r[j + v]));
    }
}

// The right-hand side of a chunk from its window (at(k) = staged point k of
// the line), with the derivative's closures at the first and last two points.
template <typename T, int L, typename Load, typename At>
__device__ __forceinline__ void wall_rhs(const LineOp<T> &op, int kind, const Load &load, const At &at, T (&r)[L],
                                         int cs)
{
    chunk_rhs<T, L, 2>(kind, load, r, op);
    if (kind != DER) return;
    const int n = op.n;
    auto closed = [&](int i, T inner) {
        T v[9] = {};
#pragma unroll
        for (int k = 2; k < 7; ++k) v[k] = at(i - 4 + k);  // rows past the ends exist; their values are unused
        return der_closure(i, n, v, op, inner);
    };
    if (cs == 0) {
        r[0] = closed(0, r[0]);
        r[1] = closed(1, r[1]);
    }
    if (cs + L > n - 2) {
        const T a = closed(n - 2, T(0)), b = closed(n - 1, T(0));
#pragma unroll
        for (int j = 0; j < L; ++j) {
            if (cs + j == n - 2) r[j] = a;
            if (cs + j == n - 1) r[j] = b;
        }
    }
}

// y- and z-lines: W x-adjacent lines, n_in points in and op.n out (o1 the x
// extent, ny_in the input's and output's y extents along z).
template <typename T, int W, int L>
__global__ void __launch_bounds__(256, 3)
    ls_wall_yz(const T *__restrict__ in, T *__restrict__ out, const __grid_constant__ LineOp<T> op,
               const __grid_constant__ WallTables<T> tb, int kind, int n_in, int nx, int ny, int dir, int refl, int C,
               bool vec)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *const tile = reinterpret_cast<T *>(smem_raw);
    const int m = op.n;
    const bool vp = kind == DERVP || kind == INTVP;
    const int t = threadIdx.x, nt = blockDim.x;
    const int tiles_x = (nx + W - 1) / W;
    const int x0 = (int)(blockIdx.x % tiles_x) * W;
    const int o = (int)(blockIdx.x / tiles_x);
    const size_t stride = dir == DY ? (size_t)nx : (size_t)nx * ny;
    const size_t bi = (size_t)x0 + (dir == DY ? (size_t)nx * n_in * o : (size_t)nx * o);
    const size_t bo = (size_t)x0 + (dir == DY ? (size_t)nx * m * o : (size_t)nx * o);
    const int cols = min(W, nx - x0);
    pdl_trigger();
    pdl_wait();
    in = pdl_after(in);
    copy_columns<W>(tile + kHalo * W, in + bi, stride, n_in, cols, vec);
    if (kind != DER)  // the reflected rows: points -4 .. -1 and n_in .. m + 3
        for (int i = t; i < (m - n_in + 2 * kHalo) * W; i += nt) {
            const int h = i / W, x = i % W, k = h < kHalo ? h - kHalo : n_in + h - kHalo;
            if (x < cols) stage_point(tile + (kHalo + k) * W + x, in + bi + x, stride, k, n_in, vp, refl);
        }
    const ChunkScratch<T> sc = carve_scratch<T>(smem_raw + (size_t)(C * L + 2 * kHalo) * W * sizeof(T), nt, 1);
    cp_async_wait_all();
    __syncthreads();
    const bool active = t < W * C;
    const int l = active ? t % W : 0, c = active ? t / W : 0;
    const int cs = c * L;
    const int nv = min(L, m - cs);
    const T *col = tile + cs * W + l;  // points cs - 4 ...
    auto load = [&](auto &w, auto j0) {
        constexpr int J0 = decltype(j0)::value;
        constexpr int NW = sizeof(w) / sizeof(T);
#pragma unroll
        for (int j = 0; j < NW; ++j) w[j] = col[(J0 + j) * W];
    };
    auto at = [&](int i) { return tile[(kHalo + i) * W + l]; };
    T r[L];
    wall_rhs<T, L>(op, kind, load, at, r, cs);
    wall_solve<T, L>(tb, r, sc, W, l, c, C, nv, t);
    if (!active || l >= cols) return;
    T *dst = out + bo + l + (size_t)cs * stride;
    if (nv == L) {
#pragma unroll
        for (int j = 0; j < L; ++j, dst += stride) *dst = r[j];
    } else {
#pragma unroll
        for (int j = 0; j < L; ++j, dst += stride)
            if (j < nv) *dst = r[j];
    }
}

// x-lines: W rows, results through the tile's own rows (each thread writes
// its chunk over the points it alone still needs after the solve's barriers)
// so that the stores are consecutive.
template <typename T, int W, int L>
__global__ void __launch_bounds__(256, 3)
    ls_wall_x(const T *__restrict__ in, T *__restrict__ out, const __grid_constant__ LineOp<T> op,
              const __grid_constant__ WallTables<T> tb, int kind, int n_in, long nlines, int pitch, int refl, int C,
              bool vec)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *const tile = reinterpret_cast<T *>(smem_raw);
    const int m = op.n;
    const bool vp = kind == DERVP || kind == INTVP;
    const int t = threadIdx.x, nt = blockDim.x;
    const long l0 = (long)blockIdx.x * W;
    const int rows = (int)min((long)W, nlines - l0);
    pdl_trigger();
    pdl_wait();
    in = pdl_after(in);
    copy_rows(tile + kHalo, pitch, in + (size_t)l0 * n_in, n_in, n_in, rows, vec);
    if (kind != DER) {
        const int nh = m - n_in + 2 * kHalo;
        for (int i = t; i < nh * rows; i += nt) {
            const int rr = i / nh, h = i % nh, k = h < kHalo ? h - kHalo : n_in + h - kHalo;
            stage_point(tile + (size_t)rr * pitch + kHalo + k, in + (size_t)(l0 + rr) * n_in, 1, k, n_in, vp, refl);
        }
    }
    const ChunkScratch<T> sc = carve_scratch<T>(smem_raw + (((size_t)W * pitch * sizeof(T) + 127) & ~(size_t)127), nt, 1);
    cp_async_wait_all();
    __syncthreads();
    const bool active = t < W * C;
    const int l = active ? t % W : 0, c = active ? t / W : 0;
    const int cs = c * L;
    const int nv = min(L, m - cs);
    const int lr = l < rows ? l : 0;
    T *const row = tile + (size_t)lr * pitch;
    auto load = [&](auto &w, auto j0) {
        constexpr int J0 = decltype(j0)::value;
        constexpr int NW = sizeof(w) / sizeof(T);
#pragma unroll
        for (int j = 0; j < NW; j += V) {
            const VT q = *reinterpret_cast<const VT *>(row + cs + J0 + j);
            const T *e = reinterpret_cast<const T *>(&q);
#pragma unroll
            for (int v = 0; v < V; ++v) w[j + v] = e[v];
        }
    };
    auto at = [&](int i) { return row[kHalo + i]; };
    T r[L];
    wall_rhs<T, L>(op, kind, load, at, r, cs);
    wall_solve<T, L>(tb, r, sc, W, l, c, C, nv, t);  // every read of the rows is before its barriers
    if (active && l < rows) {
#pragma unroll
        for (int j = 0; j < L; j += V) {
            VT q;
            T *e = reinterpret_cast<T *>(&q);
#pragma unroll
            for (int v = 0; v < V; ++v) e[v] = r[j + v];
            *reinterpret_cast<VT *>(row + cs + j) = q;
        }
    }
    __syncthreads();
    for (int rr = t >> 5; rr < rows; rr += nt >> 5) {
        T *dst = out + (size_t)(l0 + rr) * m;
#pragma unroll 4
        for (int i = t & 31; i < m; i += 32) dst[i] = tile[(size_t)rr * pitch + i];
    }
}

template <typename T>
static int launch_wall_t(x3d_ctx_s *ctx, const x3d_op_s *op, int kind, int dir, const T *in, T *out, int n_in, int o1,
                         int o2, int refl)
{
    constexpr int L = kChunkLong<T>;
    constexpr int V = Vec4<T>::N;
    const T *tab;
    LineOp<T> lo;
    WallTables<T> tb;
    constexpr int p = sizeof(T) == 4 ? 0 : 1;
    if constexpr (p == 0) tab = op->wallf, lo = op->opf;
    else tab = op->walld, lo = op->opd;
    tb.depth = op->wall_depth[p];
    if (!tab) return X3D_EUNSUPPORTED;
    // the chunk stencils take the scalars that the circulant form scales
    lo.ca = lo.a, lo.cb = lo.b, lo.cc = lo.c, lo.cd = lo.d;
    const int m = lo.n, C = (m + L - 1) / L;
    const size_t P = (size_t)C * L;
    tb.s = tab, tb.w = tab + P, tb.fw = tab + 2 * P, tb.h = tab + 3 * P, tb.g = tab + 4 * P;
    tb.mf = tab + 5 * P, tb.mb = tb.mf + C;
    auto run = [&](auto w) {
        constexpr int W = decltype(w)::value;
        const int threads = (C * W + 31) / 32 * 32;
        const size_t scratch = (size_t)2 * threads * sizeof(T);
        int pitch = C * L + 2 * kHalo;
        while (((size_t)pitch * sizeof(T) / 16) % 2 == 0) pitch += V;
        const size_t tile = dir == DX ? ((size_t)W * pitch * sizeof(T) + 127) & ~(size_t)127
                                      : (size_t)(C * L + 2 * kHalo) * W * sizeof(T);
        const size_t smem = tile + scratch;
        const long lines = (long)o1 * o2;
        const long grid = dir == DX ? (lines + W - 1) / W : (long)((o1 + W - 1) / W) * o2;
        if (threads > 256 || smem + 1024 > ctx->smem_optin || grid > 0x7fffffffL) return (int)X3D_EUNSUPPORTED;
        // rows of whole, aligned 16-byte units (along x a row is a line)
        const bool vec = ((size_t)(dir == DX ? n_in : o1) * sizeof(T)) % 16 == 0 &&
                         (reinterpret_cast<uintptr_t>(in) & 15) == 0;
        ++ctx->launches;
        if (dir == DX) {
            auto kern = ls_wall_x<T, W, L>;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            return cuda_check(ctx, launch_pdl(kern, grid, (unsigned)grid, threads, smem, ctx->stream, in, out, lo, tb, kind,
                                              n_in, lines, pitch, refl, C, vec),
                              "ls_wall_x launch");
        }
        auto kern = ls_wall_yz<T, W, L>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return cuda_check(ctx, launch_pdl(kern, grid, (unsigned)grid, threads, smem, ctx->stream, in, out, lo, tb, kind, n_in,
                                          o1, o2, dir, refl, C, vec),
                          "ls_wall_yz launch");
    };
    const int lines = dir == DX ? x_tile_lines(32, C, (long)o1 * o2, ctx->num_sms, sizeof(T)) : 32;
    int rc = lines == 32 ? run(std::integral_constant<int, 32>{}) : X3D_EUNSUPPORTED;
    if (rc == X3D_EUNSUPPORTED && lines >= 16) rc = run(std::integral_constant<int, 16>{});
    if (rc == X3D_EUNSUPPORTED) rc = run(std::integral_constant<int, 8>{});
    return rc;
}

// A non-periodic operator along dir: n_in points a line in, the operator's
// length out, o1 x o2 lines (the extents of the other two directions).
// Four operators along y at 256 x 129 x 128 FP64 took 264 us on one thread per
// line and take 92 us (2.9 TB/s of one read and one write each); fourteen at
// 193^3 FP32 1634 and 345 us (2.3 TB/s).  What bounds them is latency at three
// CTAs of 5 to 7 warps an SM (30 % of its warps) with L1 at 55 %: the five table
// rows, 16 bytes a load, beside the tile.  32 lines a CTA, where every lane of a
// warp reads the same table entries, came to 361 us against 377 for 16, both
// before dependent launches.
int launch_wall(x3d_ctx_s *ctx, const x3d_op_s *op, int kind, int dir, const void *in, void *out, int n_in, int o1,
                int o2, int refl, bool fp32)
{
    return fp32 ? launch_wall_t<float>(ctx, op, kind, dir, static_cast<const float *>(in), static_cast<float *>(out),
                                       n_in, o1, o2, refl)
                : launch_wall_t<double>(ctx, op, kind, dir, static_cast<const double *>(in),
                                        static_cast<double *>(out), n_in, o1, o2, refl);
}

}  // namespace x3d
