// Stage programs on grids whose rows are not whole 16-byte units (odd x
// extents, FP32 x extents not a multiple of 4) or whose fields start at an
// unaligned address: the chunked solve of linesolve_chunk.cu on tiles that
// every thread of the CTA copies element by element (cp.async), since TMA
// boxes and bulk copies move whole 16-byte units only.
//
// What bounds these launches is still HBM: an element copy costs one
// instruction per 32 elements and input, against some twenty per point and
// operator for the solve (short x lines excepted, see x_tile_lines).  Before, such grids went one thread per line through
// global memory (ls_generic), where a warp's 32 x lines touch 32 rows at
// once; the figures are at launch_stage_any.
//
// One CTA per tile and one staging slot: several CTAs share an SM (three of
// 256 threads for plain programs, 80 registers a thread), and their copies,
// solves and stores overlap.
#include "chunk_solve.cuh"
#include "launch_pdl.h"
#include "linesolve_chunk.h"
#include "ptx.cuh"
#include "tile_copy.cuh"
#include "x3d_internal.h"

namespace x3d {

// y- and z-lines: W x-adjacent lines of n points, with the periodic halo rows
// taken straight from global memory.  Threads past the tile's W C chunks run
// chunk 0 of line 0 into scratch slots of their own and store nothing.
template <typename T, int W, int L, bool ACC, int OCC, typename TI = T>
__global__ void __launch_bounds__(OCC > 1 ? 256 : 512, OCC)
    ls_any_yz(const __grid_constant__ StageProgram<T> prog, int nx, int ny, int dir, int C, size_t tile_bytes)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int n = prog.ops[0].op.n;
    const int t = threadIdx.x, nt = blockDim.x;
    const int tiles_x = (nx + W - 1) / W;
    const int x0 = (int)(blockIdx.x % tiles_x) * W;
    const int o = (int)(blockIdx.x / tiles_x);
    const size_t stride = dir == DY ? (size_t)nx : (size_t)nx * ny;
    const size_t plane = (size_t)x0 + (dir == DY ? (size_t)nx * ny * o : (size_t)nx * o);
    const int cols = min(W, nx - x0);
    pdl_trigger();
    T *resp_s = reinterpret_cast<T *>(smem_raw + prog.ntiles * tile_bytes +
                                      (((size_t)2 * nt * sizeof(T) + 15) & ~(size_t)15));
    load_resp<T, L>(prog, resp_s);
    pdl_wait();
    for (int ti = 0; ti < prog.ntiles; ++ti) {
        const TI *src = reinterpret_cast<const TI *>(prog.in[ti]) + plane;
        TI *tp = reinterpret_cast<TI *>(smem_raw + ti * tile_bytes);
        copy_columns<W>(tp + kHalo * W, src, stride, n, cols, false);
        for (int i = t; i < 2 * kHalo * W; i += nt) {  // the periodic halo rows
            const int h = i / W, x = i % W;
            if (x < cols)
                cp_async<sizeof(TI)>(tp + (h < kHalo ? h : n + h) * W + x,
                                     src + (size_t)(h < kHalo ? n - kHalo + h : h - kHalo) * stride + x);
        }
    }
    const ChunkScratch<T> sc = carve_scratch<T>(smem_raw + prog.ntiles * tile_bytes, nt, 1);
    cp_async_wait_all();
    __syncthreads();

    const bool active = t < W * C;
    const int l = active ? t % W : 0, c = active ? t / W : 0;
    const int cs = c * L;
    const int nv = min(L, n - cs);
    auto col = [&](int ti) {
        return reinterpret_cast<const TI *>(smem_raw + ti * tile_bytes) + (kHalo + cs - 4) * W + l;
    };
    auto tile_at = [&](int ti, int j) { return T(col(ti)[(4 + j) * W]); };
    auto flush_args = [&](const StageOp<T> &so) {
        if constexpr (std::is_same<TI, T>::value)
            return FlushArgs<T>(so, so.base2_tile >= 0 ? col(so.base2_tile) + 4 * W : nullptr, W);
        else return FlushArgs<T>(so);
    };
    const bool live = active && l < cols;
    const size_t obase = plane + l + (size_t)cs * stride;
    T r[L];
    T acc[ACC ? L : 1];
    for (int k = 0; k < prog.nops; ++k) {
        const StageOp<T> &so = prog.ops[k];
        const TI *ca = col(so.src_a);
        const TI *cb = so.src_b >= 0 ? col(so.src_b) : nullptr;
        auto load = [&](auto &w, auto j0) {
            constexpr int J0 = decltype(j0)::value;
            constexpr int NW = sizeof(w) / sizeof(T);
            if (cb) {
#pragma unroll
                for (int j = 0; j < NW; ++j) w[j] = T(ca[(J0 + j) * W]) * T(cb[(J0 + j) * W]);
            } else {
#pragma unroll
                for (int j = 0; j < NW; ++j) w[j] = T(ca[(J0 + j) * W]);
            }
        };
        constexpr bool trim = !ACC && (OCC == 1 || sizeof(T) == 4);  // FP64 at 80 registers would spill
        chunk_solve_resp<T, L, trim>(so.op, so.kind, resp_s + k * 4 * L, load, r, sc, W, l, c, C, nv, t, so.keep);
        if constexpr (ACC) {
            accumulate<T, L, 1>(so, acc, r, nv, tile_at);
            if (so.flush && live) flush_yz<T, T, L, true>(flush_args(so), acc, obase, stride, nv);
        } else {
            if (so.flush && live) flush_yz<T, T, L, false>(flush_args(so), r, obase, stride, nv);
            if (so.shift_out && live) flush_yz_shifted<T, T, L>(so.shift_out, r, obase, cs, stride, nv, c == C - 1);
        }
    }
}

// The flush of a tile of x lines from its staging rows, element by element:
// each warp takes whole rows, so its loads and stores are consecutive.  A
// lane's elements go in blocks of 4 whose loads precede their stores (base
// and base2 are often the outputs themselves).  U = double: FP64 outputs.
template <typename T, typename U, bool GENERAL>
__device__ __forceinline__ void flush_rows_any(const StageOp<T> &so, const T *out_s, size_t g0, int rows, int pitch,
                                               int n)
{
    constexpr int NB = 4;
    const U *base = GENERAL ? static_cast<const U *>(so.base) : nullptr;
    const U *base2 = GENERAL ? static_cast<const U *>(so.base2) : nullptr;
    U *out = static_cast<U *>(so.out);
    U *out2 = GENERAL ? static_cast<U *>(so.out2) : nullptr;
    const U sign = (U)so.sign, scale2 = (U)so.scale2;
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int rr = threadIdx.x >> 5; rr < rows; rr += nw) {
        const T *row = out_s + (size_t)rr * pitch;
        const size_t g = g0 + (size_t)rr * n;
        for (int i0 = lane; i0 < n; i0 += 32 * NB) {
            U b[NB], b2[NB];
            if constexpr (GENERAL) {
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    const int i = i0 + 32 * q;
                    b[q] = base && i < n ? base[g + i] : U(0);
                    b2[q] = base2 && i < n ? base2[g + i] : U(0);
                }
            }
#pragma unroll
            for (int q = 0; q < NB; ++q) {
                const int i = i0 + 32 * q;
                if (i < n) {
                    if constexpr (GENERAL) {
                        const U v = b[q] + sign * (U)row[i];
                        out[g + i] = v;
                        if (out2) out2[g + i] = b2[q] + scale2 * v;
                    } else {
                        out[g + i] = (U)row[i];
                    }
                }
            }
        }
    }
}

// x-lines: W rows of n points in padded rows (odd 16-byte granules, so the
// vector reads of the windows do not conflict), outputs staged in rows of the
// same pitch.
template <typename T, int W, int L, bool ACC, int OCC>
__global__ void __launch_bounds__(OCC > 1 ? 256 : 512, OCC)
    ls_any_x(const __grid_constant__ StageProgram<T> prog, long nlines, int pitch, int C, size_t tile_bytes)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int n = prog.ops[0].op.n;
    const int t = threadIdx.x, nt = blockDim.x;
    const long l0 = (long)blockIdx.x * W;
    const int rows = (int)min((long)W, nlines - l0);
    pdl_trigger();
    T *resp_s = reinterpret_cast<T *>(smem_raw + prog.ntiles * tile_bytes +
                                      (((size_t)2 * nt * sizeof(T) + 15) & ~(size_t)15));
    load_resp<T, L>(prog, resp_s);
    pdl_wait();
    for (int ti = 0; ti < prog.ntiles; ++ti) {
        T *tp = reinterpret_cast<T *>(smem_raw + ti * tile_bytes);
        const T *src = prog.in[ti] + (size_t)l0 * n;
        copy_rows(tp + kHalo, pitch, src, n, n, rows, false);
        for (int i = t; i < 2 * kHalo * rows; i += nt) {  // the periodic halos
            const int rr = i / (2 * kHalo), h = i % (2 * kHalo);
            cp_async<sizeof(T)>(tp + (size_t)rr * pitch + (h < kHalo ? h : n + h),
                                src + (size_t)rr * n + (h < kHalo ? n - kHalo + h : h - kHalo));
        }
    }
    const ChunkScratch<T> sc = carve_scratch<T>(smem_raw + prog.ntiles * tile_bytes, nt, 1);
    T *out_s = resp_s + prog.nops * 4 * L;
    cp_async_wait_all();
    __syncthreads();

    const bool active = t < W * C;
    const int l = active ? t % W : 0, c = active ? t / W : 0;
    const int cs = c * L;
    const int nv = min(L, n - cs);
    const int lr = l < rows ? l : 0;  // rows past the end compute on row 0 and store nothing
    auto row = [&](int ti) {
        return reinterpret_cast<const T *>(smem_raw + ti * tile_bytes) + (size_t)lr * pitch + cs;
    };
    auto tile_at = [&](int ti, int j) { return *reinterpret_cast<const VT *>(row(ti) + kHalo + j); };
    T r[L];
    T acc[ACC ? L : 1];
    for (int k = 0; k < prog.nops; ++k) {
        const StageOp<T> &so = prog.ops[k];
        const T *ra = row(so.src_a);
        const T *rb = so.src_b >= 0 ? row(so.src_b) : nullptr;
        auto load = [&](auto &w, auto j0) {
            constexpr int J0 = decltype(j0)::value;
            constexpr int NW = sizeof(w) / sizeof(T);
#pragma unroll
            for (int j = 0; j < NW; j += V) {
                const VT qa = *reinterpret_cast<const VT *>(ra + J0 + j);
                const T *ea = reinterpret_cast<const T *>(&qa);
                if (rb) {
                    const VT qb = *reinterpret_cast<const VT *>(rb + J0 + j);
                    const T *eb = reinterpret_cast<const T *>(&qb);
#pragma unroll
                    for (int v = 0; v < V; ++v) w[j + v] = ea[v] * eb[v];
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) w[j + v] = ea[v];
                }
            }
        };
        constexpr bool trim = !ACC && (OCC == 1 || sizeof(T) == 4);
        // its barriers also end every thread's reads of the staging rows by
        // the previous operator's flush
        chunk_solve_resp<T, L, trim>(so.op, so.kind, resp_s + k * 4 * L, load, r, sc, W, l, c, C, nv, t, so.keep);
        if constexpr (ACC) accumulate<T, L, V>(so, acc, r, nv, tile_at);
        if (!so.flush) continue;
        if (active && l < rows) {
            T *dst = out_s + (size_t)l * pitch + cs;  // room for the last window past n
#pragma unroll
            for (int j = 0; j < L; j += V) {
                VT q;
                T *e = reinterpret_cast<T *>(&q);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if constexpr (ACC) e[v] = acc[j + v];
                    else e[v] = r[j + v];
                }
                *reinterpret_cast<VT *>(dst + j) = q;
            }
        }
        __syncthreads();
        const size_t g0 = (size_t)l0 * n;
        if constexpr (ACC) {
            if (so.out_f64) flush_rows_any<T, double, true>(so, out_s, g0, rows, pitch, n);
            else flush_rows_any<T, T, true>(so, out_s, g0, rows, pitch, n);
        } else {
            flush_rows_any<T, T, false>(so, out_s, g0, rows, pitch, n);
            if (so.shift_out) flush_rows_shifted<T, false>(so.shift_out, out_s, l0, rows, pitch, n);
        }
    }
}

// The derivative sweep (18 operators of one field, three launches) took 1547 us
// at 171 x 129 x 150 FP64 on ls_generic and takes 170 us here (3.3 TB/s of one
// read per direction and the outputs); 1575 and 157 us at 250 x 171 x 129 FP32.
// The periodic correction, an FP64 sum there, is the carry scan in the program's
// type here; the errors against 64 bits are no larger (FP32, 2-norm, rms over 21
// lines of 17 to 255 points a kind: der 1.13e-7 there, 0.97e-7 here, der2 6.9e-8
// and 6.8e-8, dervp 7.0e-8 and 5.9e-8, interpvp 9.9e-7 and 8.7e-7; FP64 der
// 1.30e-15 both, dervp 1.42e-15 and 1.44e-15, interpvp 2.2e-15 and 1.9e-15).
// prog: its responses filled for chunks of kChunkLong<T> points (launch_stage
// did), acc: it needs the accumulator or a general flush.
template <typename T, int W>
int launch_stage_any(x3d_ctx_s *ctx, const StageProgram<T> &prog, bool acc, int dir, int nx, int ny, int nz)
{
    constexpr int L = kChunkLong<T>;
    constexpr int V = Vec4<T>::N;
    const int n = prog.ops[0].op.n;
    const int C = (n + L - 1) / L;
    const int threads = (C * W + 31) / 32 * 32;
    if (threads > 512) return X3D_EUNSUPPORTED;
    const size_t es = sizeof(T);
    const size_t scratch = ((size_t)2 * threads * es + 15) & ~(size_t)15;
    const size_t resp = (size_t)prog.nops * 4 * L * es;
    const bool small = threads <= 256;
    auto launch = [&](auto kern, size_t smem, long grid, auto... args) {
        if (smem + 1024 > ctx->smem_optin || grid > 0x7fffffffL) return (int)X3D_EUNSUPPORTED;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ++ctx->launches;
        return cuda_check(ctx, launch_pdl(kern, grid, (unsigned)grid, threads, smem, ctx->stream, prog, args...),
                          "ls_any launch");
    };
    if (dir == DX) {
        int pitch = C * L + 2 * kHalo;
        while (((size_t)pitch * es / 16) % 2 == 0) pitch += V;
        const size_t tile = ((size_t)W * pitch * es + 127) & ~(size_t)127;
        const size_t smem = prog.ntiles * tile + scratch + resp + (size_t)W * pitch * es;
        const long nlines = (long)ny * nz, grid = (nlines + W - 1) / W;
        if (acc) return launch(ls_any_x<T, W, L, true, 1>, smem, grid, nlines, pitch, C, tile);
        if (small) return launch(ls_any_x<T, W, L, false, 3>, smem, grid, nlines, pitch, C, tile);
        return launch(ls_any_x<T, W, L, false, 1>, smem, grid, nlines, pitch, C, tile);
    }
    const size_t tile = ((size_t)(C * L + 2 * kHalo) * W * (prog.in_f64 ? sizeof(double) : es) + 127) & ~(size_t)127;
    const size_t smem = prog.ntiles * tile + scratch + resp;
    const long grid = (long)((nx + W - 1) / W) * (dir == DY ? nz : ny);
    if constexpr (sizeof(T) == 4)
        if (prog.in_f64) {
            if (small) return launch(ls_any_yz<T, W, L, false, 3, double>, smem, grid, nx, ny, dir, C, tile);
            return launch(ls_any_yz<T, W, L, false, 1, double>, smem, grid, nx, ny, dir, C, tile);
        }
    if (acc) return launch(ls_any_yz<T, W, L, true, 1>, smem, grid, nx, ny, dir, C, tile);
    if (small) return launch(ls_any_yz<T, W, L, false, 3>, smem, grid, nx, ny, dir, C, tile);
    return launch(ls_any_yz<T, W, L, false, 1>, smem, grid, nx, ny, dir, C, tile);
}

template int launch_stage_any<float, 32>(x3d_ctx_s *, const StageProgram<float> &, bool, int, int, int, int);
template int launch_stage_any<float, 16>(x3d_ctx_s *, const StageProgram<float> &, bool, int, int, int, int);
template int launch_stage_any<float, 8>(x3d_ctx_s *, const StageProgram<float> &, bool, int, int, int, int);
template int launch_stage_any<double, 16>(x3d_ctx_s *, const StageProgram<double> &, bool, int, int, int, int);
template int launch_stage_any<double, 8>(x3d_ctx_s *, const StageProgram<double> &, bool, int, int, int, int);

}  // namespace x3d
