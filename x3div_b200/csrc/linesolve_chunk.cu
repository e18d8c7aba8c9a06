// Chunked periodic line solves: the fast path for whole-field operator
// applications, and the stage kernels that fuse several operators, their
// pointwise products and their sums into one pass over the staged inputs.
//
// The reference sweeps each line serially (?thomas_12, src/thomas.f90:61-84)
// with the LU factors of its periodic matrix, then corrects for periodicity
// with the precomputed vector p (xthomas_0 :49-55).  The matrix that pair
// inverts is exactly the circulant (alfa, 1, alfa), which factors as
//   M = (1 + rho^2)^-1 (1 - rho E^-1)(1 - rho E),  alfa rho^2 + rho + alfa = 0,
// |rho| < 1.  So y = M^-1 r is two first-order periodic recurrences with one
// constant coefficient:
//   forward  v_i = (1 + rho^2) r_i + rho v_{i-1}     backward  y_i = v_i + rho y_{i+1}
// (the factor 1 + rho^2 is folded into the RHS scalars).
//
// A line of n points is cut into C chunks of L points; thread (l, c) owns
// chunk c of line l and keeps it in registers.  Each recurrence is affine in
// its incoming value, so a chunk is swept locally from zero and later
// shifted by rho^k * carry:
//   1. stencil r_i for the chunk from an L+8 window of the staged input;
//   2. local forward sweep, chunk end value to shared memory;
//   -- barrier -- each thread folds the end values of the chunks before it
//      (depth chunks, or the whole line divided by 1 - rho^n) into its
//      carry, fixes its values and sweeps backward locally;
//   -- barrier -- the same for the backward carry from the chunks after it.
// Every chunk does the same work: no tables, no per-line scalar, two
// barriers per operator and one HBM read and write per application.
//
// A stage (StageProgram) runs up to six such operators over up to three
// staged inputs, combining the results in a register accumulator and
// writing only what the program flushes, so e.g. one x-pencil pass of
// momentum_rhs_eq (src/transeq.f90:99-116, six derx calls and their
// products and sums for three velocity components) is one kernel.
//
// Staging: y/z tiles of W x-adjacent lines arrive by TMA tensor loads and
// results go straight to global memory, coalesced across the W lines; x
// tiles arrive as W padded rows by 1-D bulk copies and results leave as
// 16-byte vector stores of each thread's contiguous chunk.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "chunk_solve.cuh"
#include "launch_pdl.h"
#include "linesolve_chunk.h"
#include "ptx.cuh"
#include "x3d_internal.h"

namespace x3d {

// ---------------------------------------------------------------------------
// y- and z-lines.
struct StageMaps {
    CUtensorMap m[kMaxStageTiles];   // inputs
    CUtensorMap hm[kMaxStageTiles];  // the same inputs in boxes of kHalo rows: the periodic halos
    CUtensorMap pm[kMaxStageOps];    // base (else base2) arrays prefetched into L2 (ops with prefetch_base)
};

// PERSIST: a CTA loops over tiles with two staging slots, issuing the loads
// of tile k+1 before computing tile k; otherwise one CTA per tile.  PR = 2
// (FP32 only): each thread carries the same chunk of two x-adjacent lines in
// packed registers, so every arithmetic instruction, shared-memory load and
// global store serves two lines (x extents must then be even).
//
// A persistent CTA claims its tiles one at a time from a counter (the next
// one claimed as soon as the current one's copies are issued) rather than
// taking every gridDim-th tile.  CTAs that take tiles at a fixed stride
// drift apart over a launch, and then x-adjacent tiles of a plane, whose
// 64-byte row segments make up whole rows only together, are written at
// different times.  Claimed in order, the tiles in flight stay a window of
// consecutive tiles: one read and six writes of 16-column y tiles run at
// 6.4 TB/s that way against 4.6 TB/s at a fixed stride (x3d_roofline_probe
// patterns 5 and 1).  The launcher zeroes the counter before each launch.
//
// TI: the element type of the staged inputs.  TI = double with T = float
// (plain programs, PR = 1, OCC = 1) stages FP64 fields and solves them in FP32: the
// pressure gradient reads the FP64 pressure this way, with no FP32 copy.
//
// OCC > 1: the kernel is compiled for OCC CTAs of at most 256 threads per SM
// (at most 65536 / (256 OCC) registers a thread).  With OCC = 3 the plain
// FP32 16-line, 32-point-chunk kernel fits 80 registers without spilling, so
// an SM holds 24 warps instead of 16 -- the sweep kernels are latency- and
// issue-bound at 16 (issue active about half the cycles).
//
// SHIFT: the plain kernel for programs with shifted second outputs (StageOp::
// shift_out).  Programs without run the kernel without that code: compiled in and
// unused it cost 512^3 launches of one operator 4 to 8 % (FP32 y, configuration
// 17, 167 -> 180 us; FP64 x, configuration 9, 381 -> 400).
template <typename T, int W, int L, bool ACC, bool PERSIST, int PR = 1, int OCC = 1, typename TI = T,
          bool SHIFT = false>
__global__ void __launch_bounds__(OCC > 1 ? 256 : kStageThreads<T, L, PR>, OCC)
    ls_stage_yz(const __grid_constant__ StageMaps maps, const __grid_constant__ StageProgram<T> prog, int nx,
                int ny, int dir, int box_n, int nbox, int tma_halo, size_t tile_bytes, long ntiles,
                unsigned long long *claim, int *err)
{
    using V = typename PairOf<T, PR>::type;
    static_assert(std::is_same<TI, T>::value || (PR == 1 && !ACC), "wider staged inputs: plain, unpaired");
    constexpr int WP = W / PR;  // threads across the tile's lines
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t bars[2];
    __shared__ long s_tile[2];  // by iteration parity: rewritten only after every thread has read it
    const int n = prog.ops[0].op.n;
    const int C = blockDim.x / WP;
    const int t = threadIdx.x;
    const int l = t % WP, c = t / WP;
    const int tiles_x = (nx + W - 1) / W;
    const size_t slot_bytes = (size_t)prog.ntiles * tile_bytes;
    V *resp_s = reinterpret_cast<V *>(smem_raw + (PERSIST ? 2 : 1) * slot_bytes +
                                      (((size_t)2 * C * W * sizeof(T) + 15) & ~(size_t)15));
    pdl_trigger();
    load_resp<V, L>(prog, resp_s);
    if (t == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](long tile, int slot) {
        const int x0 = (int)(tile % tiles_x) * W;
        const int o = (int)(tile / tiles_x);
        uint64_t *bar = &bars[slot];
        mbar_arrive_expect_tx(bar, (uint32_t)((size_t)prog.ntiles * (nbox * box_n + (tma_halo ? 2 * kHalo : 0)) *
                                              W * sizeof(TI)));
        for (int ti = 0; ti < prog.ntiles; ++ti) {
            TI *tp = reinterpret_cast<TI *>(smem_raw + slot * slot_bytes + ti * tile_bytes) + kHalo * W;
            for (int b = 0; b < nbox; ++b) {
                if (dir == DY)
                    tma_load_3d(tp + (size_t)b * box_n * W, &maps.m[ti], bar, x0, b * box_n, o);
                else
                    tma_load_3d(tp + (size_t)b * box_n * W, &maps.m[ti], bar, x0, o, b * box_n);
            }
            if (tma_halo) {  // points n-4 .. n-1 before the line, 0 .. 3 after it
                TI *hb = tp - kHalo * W, *ha = tp + (size_t)n * W;
                if (dir == DY) {
                    tma_load_3d(hb, &maps.hm[ti], bar, x0, n - kHalo, o);
                    tma_load_3d(ha, &maps.hm[ti], bar, x0, 0, o);
                } else {
                    tma_load_3d(hb, &maps.hm[ti], bar, x0, o, n - kHalo);
                    tma_load_3d(ha, &maps.hm[ti], bar, x0, o, 0);
                }
            }
        }
        // the tile's base arrays (read back by the flushes) into L2
        for (int mask = prog.prefetch_mask, k = 0; mask; mask >>= 1, ++k) {
            if (!(mask & 1)) continue;
            for (int b = 0; b < nbox; ++b) {
                if (dir == DY) tma_prefetch_3d(&maps.pm[k], x0, b * box_n, o);
                else tma_prefetch_3d(&maps.pm[k], x0, o, b * box_n);
            }
        }
    };
    const ChunkScratch<V> sc = carve_scratch<V>(smem_raw + (PERSIST ? 2 : 1) * slot_bytes, C, WP);
    const int cs = c * L;
    const int nv = min(L, n - cs);
    const size_t ostride = dir == DY ? (size_t)nx : (size_t)nx * ny;
    pdl_wait();
    long tile = blockIdx.x;
    if (t == 0) {
        if (PERSIST) s_tile[0] = tile = (long)atomicAdd(claim, 1ull);
        if (tile < ntiles) issue(tile, 0);
    }
    __syncthreads();
    if (PERSIST) tile = s_tile[0];
    for (int it = 0; tile < ntiles; ++it) {
        const int slot = PERSIST ? (it & 1) : 0;
        const uint32_t parity = PERSIST ? ((it >> 1) & 1) : 0;
        const bool ok = mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
        // this barrier also ends every thread's reads of the other slot (the
        // previous tile), so the next tile's copies may go there now
        if (!__syncthreads_and(ok)) {
            if (t == 0) {
                atomicExch(err, 1);
                mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
            }
            return;
        }
        if (PERSIST && t == 0) {
            const long next = (long)atomicAdd(claim, 1ull);
            s_tile[(it + 1) & 1] = next;  // read after this tile's operator barriers
            if (next < ntiles) issue(next, slot ^ 1);
        }
        const int x0 = (int)(tile % tiles_x) * W;
        const int o = (int)(tile / tiles_x);
        unsigned char *base = smem_raw + slot * slot_bytes;
        if (!tma_halo) {
            fill_halos_yz<TI>(base, tile_bytes, prog.ntiles, n, W, kHalo);
            fence_proxy_async_smem();  // the halo rows are refilled by TMA two tiles later
            __syncthreads();
        }
        // window of this chunk: rows kHalo + cs - 4 ...
        auto col = [&](int ti) {
            return reinterpret_cast<const TI *>(base + ti * tile_bytes) + (kHalo + cs - 4) * W + PR * l;
        };
        auto at = [](const TI *p) {
            if constexpr (std::is_same<TI, T>::value) return *reinterpret_cast<const V *>(p);
            else return V(*p);
        };
        auto tile_at = [&](int ti, int j) { return at(col(ti) + (4 + j) * W); };
        auto flush_args = [&](const StageOp<T> &so) {
            if constexpr (std::is_same<TI, T>::value)
                return FlushArgs<T>(so, so.base2_tile >= 0 ? col(so.base2_tile) + 4 * W : nullptr, W);
            else return FlushArgs<T>(so);
        };
        const bool live = x0 + PR * l < nx;
        const size_t obase = (size_t)(x0 + PR * l) + (dir == DY ? (size_t)nx * ny * o : (size_t)nx * o) +
                             (size_t)cs * ostride;
        V r[L];
        V acc[ACC ? L : 1];
        for (int k = 0; k < prog.nops; ++k) {
            const StageOp<T> &so = prog.ops[k];
            const TI *ca = col(so.src_a);
            const TI *cb = so.src_b >= 0 ? col(so.src_b) : nullptr;
            auto load = [&](auto &w, auto j0) {
                constexpr int J0 = decltype(j0)::value;
                constexpr int NW = sizeof(w) / sizeof(V);
                if (cb) {
#pragma unroll
                    for (int j = 0; j < NW; ++j) w[j] = at(ca + (J0 + j) * W) * at(cb + (J0 + j) * W);
                } else {
#pragma unroll
                    for (int j = 0; j < NW; ++j) w[j] = at(ca + (J0 + j) * W);
                }
            };
            constexpr bool trim = !ACC && (OCC == 1 || sizeof(T) == 4);  // FP64 at 80 registers would spill
            chunk_solve_resp<V, L, trim>(so.op, so.kind, resp_s + k * 4 * L, load, r, sc, WP, l, c, C, nv,
                                         c * WP + l, so.keep);
            if constexpr (ACC) {
                accumulate<V, L, 1>(so, acc, r, nv, tile_at);
                if (so.flush && live) flush_yz<T, V, L, true>(flush_args(so), acc, obase, ostride, nv);
            } else {
                if (so.flush && live) flush_yz<T, V, L, false>(flush_args(so), r, obase, ostride, nv);
                if constexpr (SHIFT)
                    if (so.shift_out && live)
                        flush_yz_shifted<T, V, L>(so.shift_out, r, obase, cs, ostride, nv, c == C - 1);
            }
        }
        if (!PERSIST) break;
        // written by thread 0 before the operator barriers above; rewritten two
        // tiles later, after the next wait barrier, which every thread reaches
        // after reading it here
        tile = s_tile[(it + 1) & 1];
    }
}

// ---------------------------------------------------------------------------
// x-lines.

// General flush of an x chunk (contiguous from element p0) as 16-byte
// vectors of the output type U, in blocks of up to 8 points whose loads
// (base, base2, often the output arrays themselves) all precede their stores.
template <typename T, typename U, int L>
__device__ __forceinline__ void flush_x_blocked(const FlushArgs<T> &fa, const T (&res)[L], size_t p0, int nv)
{
    using UV = typename Vec4<U>::type;
    constexpr int VU = Vec4<U>::N;
    constexpr int B = L < 8 ? L : 8;
    constexpr int NQ = B / VU;
    const U *base = static_cast<const U *>(fa.base);
    const U *base2 = static_cast<const U *>(fa.base2);
    U *out = static_cast<U *>(fa.out);
    U *out2 = static_cast<U *>(fa.out2);
    const U sign = (U)fa.sign, scale2 = (U)fa.scale2;
#pragma unroll
    for (int j0 = 0; j0 < L; j0 += B) {
        UV bq[NQ], b2q[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int j = j0 + q * VU;
            const bool in = j < nv;
            bq[q] = base && in ? *reinterpret_cast<const UV *>(base + p0 + j) : UV{};
            if constexpr (std::is_same<T, U>::value) {
                if (fa.b2s) b2q[q] = *reinterpret_cast<const UV *>(fa.b2s + j);
                else b2q[q] = base2 && in ? *reinterpret_cast<const UV *>(base2 + p0 + j) : UV{};
            } else {
                b2q[q] = base2 && in ? *reinterpret_cast<const UV *>(base2 + p0 + j) : UV{};
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int j = j0 + q * VU;
            if (j < nv) {
                UV o, o2;
                U *ov = reinterpret_cast<U *>(&o);
                U *o2v = reinterpret_cast<U *>(&o2);
                const U *bv = reinterpret_cast<const U *>(&bq[q]);
                const U *b2v = reinterpret_cast<const U *>(&b2q[q]);
#pragma unroll
                for (int e = 0; e < VU; ++e) {
                    ov[e] = bv[e] + sign * (U)res[j + e];
                    o2v[e] = b2v[e] + scale2 * ov[e];
                }
                *reinterpret_cast<UV *>(out + p0 + j) = o;
                if (out2) *reinterpret_cast<UV *>(out2 + p0 + j) = o2;
            }
        }
    }
}

// Writes one thread's solved chunk of an x line (points j < nv) as 16-byte
// vectors starting at element p0.
template <typename T, int L>
__device__ __forceinline__ void flush_x(const FlushArgs<T> &fa, const T (&res)[L], size_t p0, int nv)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    if (fa.plain) {
        T *dst = static_cast<T *>(fa.out) + p0;
#pragma unroll
        for (int j = 0; j < L; j += V) {
            if (j < nv) {
                VT q;
                T *e = reinterpret_cast<T *>(&q);
#pragma unroll
                for (int v = 0; v < V; ++v) e[v] = res[j + v];
                *reinterpret_cast<VT *>(dst + j) = q;
            }
        }
        return;
    }
    if (fa.f64) flush_x_blocked<T, double, L>(fa, res, p0, nv);
    else flush_x_blocked<T, T, L>(fa, res, p0, nv);
}

// The general flush of a tile of x lines from its staging rows: the CTA's
// threads sweep the rows as 16-byte vectors, consecutive threads on
// consecutive vectors of a row, so the loads of base and base2 and the
// stores of out and out2 are coalesced across each warp (each thread's own
// chunk would touch a different line per vector).  A thread's vectors go in
// blocks of NB (2: the accumulator stays live across the flush, so more
// would spill) whose loads all precede their stores: base2 is often out2
// itself (u = u - p in place), so a load after a store could not move ahead
// of it and each vector would wait for memory in turn.  U = double writes
// FP64 outputs.
template <typename T, typename U>
__device__ __forceinline__ void flush_x_rows(const FlushArgs<T> &fa, const T *out_s, long l0, int rows,
                                             int pitch, int n)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    using UV = typename Vec4<U>::type;
    constexpr int NU = V / Vec4<U>::N;  // U vectors per T vector
    constexpr int NB = 2;
    const U *base = static_cast<const U *>(fa.base);
    const U *base2 = static_cast<const U *>(fa.base2);
    U *out = static_cast<U *>(fa.out);
    U *out2 = static_cast<U *>(fa.out2);
    const U sign = (U)fa.sign, scale2 = (U)fa.scale2;
    // this thread's vectors: (row r0 + i * G, vector q) for i = 0, 1, ...
    const int per_row = n / V, nt = blockDim.x, t = threadIdx.x;
    int G, r0, q, qs;  // rows step, first row, vector, vector step
    if (nt >= per_row) {
        G = nt / per_row;
        r0 = t / per_row;
        q = t - r0 * per_row;
        qs = per_row;  // one vector per row
        if (r0 >= G) return;
    } else {
        G = 1;
        r0 = 0;
        q = t;
        qs = nt;
    }
    for (int rr0 = r0; rr0 < rows; rr0 += NB * G) {
        for (int q0 = q; q0 < per_row; q0 += qs) {
            UV b[NB][NU], b2[NB][NU];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const int rr = rr0 + i * G;
                const size_t g = (size_t)(l0 + rr) * n + (size_t)q0 * V;
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    b[i][u] = base && rr < rows ? *reinterpret_cast<const UV *>(base + g + u * (V / NU)) : UV{};
                    b2[i][u] = base2 && rr < rows ? *reinterpret_cast<const UV *>(base2 + g + u * (V / NU)) : UV{};
                }
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const int rr = rr0 + i * G;
                if (rr >= rows) break;
                const size_t g = (size_t)(l0 + rr) * n + (size_t)q0 * V;
                const VT v = *reinterpret_cast<const VT *>(out_s + (size_t)rr * pitch + (size_t)q0 * V);
                const T *vl = reinterpret_cast<const T *>(&v);
                const U *bl = reinterpret_cast<const U *>(b[i]);
                const U *b2l = reinterpret_cast<const U *>(b2[i]);
                UV o[NU], o2[NU];
                U *ol = reinterpret_cast<U *>(o);
                U *o2l = reinterpret_cast<U *>(o2);
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    ol[e] = bl[e] + sign * (U)vl[e];
                    o2l[e] = b2l[e] + scale2 * ol[e];
                }
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    *reinterpret_cast<UV *>(out + g + u * (V / NU)) = o[u];
                    if (out2) *reinterpret_cast<UV *>(out2 + g + u * (V / NU)) = o2[u];
                }
            }
        }
    }
}

// Flush of one operator for a tile of x lines.  Every thread first writes
// its chunk into the tile's staging rows (odd 16-byte granules per row, so
// the vector stores do not conflict).  A plain output then leaves as one
// bulk copy per row; any other (base, base2, FP64) is written by the whole
// CTA row by row (flush_x_rows).  A base2 that is a staged input (read from
// the tile, per thread) keeps the direct per-chunk flush.  The caller waits
// for the copies' reads before the staging rows are reused.  fa.plain and
// fa.b2s are the same for the whole CTA, so the barrier is uniform.
// GENERAL = false: the program's flushes are all plain, and the other forms
// are not compiled into the kernel.
template <typename T, int L, bool GENERAL>
__device__ __forceinline__ void flush_x_staged(const FlushArgs<T> &fa, const T (&res)[L], T *out_s, int l,
                                               long l0, int rows, int pitch, int n, int cs, int nv)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    if constexpr (GENERAL) {
        if (fa.b2s) {
            if (l < rows) flush_x<T, L>(fa, res, (size_t)(l0 + l) * n + cs, nv);
            return;
        }
    }
    if (l < rows) {
        // the staging row is the tile's own: a short last chunk may write
        // past the line's end there (room for the last window), and the
        // row pass sends only the line's n points
        T *dst = out_s + (size_t)l * pitch + cs;
#pragma unroll
        for (int j = 0; j < L; j += V) {
            VT q;
            T *e = reinterpret_cast<T *>(&q);
#pragma unroll
            for (int v = 0; v < V; ++v) e[v] = res[j + v];
            *reinterpret_cast<VT *>(dst + j) = q;
        }
    }
    fence_proxy_async_smem();
    __syncthreads();
    if constexpr (GENERAL) {
        if (!fa.plain) {
            if (fa.f64) flush_x_rows<T, double>(fa, out_s, l0, rows, pitch, n);
            else flush_x_rows<T, T>(fa, out_s, l0, rows, pitch, n);
            return;
        }
    }
    const int t = threadIdx.x;
    if (t < rows) {
        bulk_store(static_cast<T *>(fa.out) + (size_t)(l0 + t) * n, out_s + (size_t)t * pitch,
                   (uint32_t)(n * sizeof(T)));
        bulk_commit();
    }
}

// SHIFT as for ls_stage_yz.
template <typename T, int W, int L, bool ACC, bool PERSIST, int OCC = 1, bool SHIFT = false>
__global__ void __launch_bounds__(OCC > 1 ? 256 : 512, OCC)
    ls_stage_x(const __grid_constant__ StageProgram<T> prog, long nlines, int pitch, size_t tile_bytes,
               long ntiles, unsigned long long *claim, int *err)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t bars[2];
    __shared__ long s_tile[2];  // persistent: tiles claimed in order, as ls_stage_yz does
    const int n = prog.ops[0].op.n;
    const int C = blockDim.x / W;
    const int t = threadIdx.x;
    const int l = t % W, c = t / W;
    const uint32_t row_bytes = (uint32_t)(n * sizeof(T));
    const size_t slot_bytes = (size_t)prog.ntiles * tile_bytes;
    T *resp_s = reinterpret_cast<T *>(smem_raw + (PERSIST ? 2 : 1) * slot_bytes +
                                      (((size_t)2 * C * W * sizeof(T) + 15) & ~(size_t)15));
    pdl_trigger();
    load_resp<T, L>(prog, resp_s);
    if (t == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](long tile, int slot) {
        const long l0 = tile * W;
        const int rows = (int)min((long)W, nlines - l0);
        uint64_t *bar = &bars[slot];
        mbar_arrive_expect_tx(bar, row_bytes * (uint32_t)rows * (uint32_t)prog.ntiles);
        for (int ti = 0; ti < prog.ntiles; ++ti) {
            T *tp = reinterpret_cast<T *>(smem_raw + slot * slot_bytes + ti * tile_bytes) + kHalo;
            for (int rr = 0; rr < rows; ++rr)
                bulk_load(tp + (size_t)rr * pitch, prog.in[ti] + (size_t)(l0 + rr) * n, row_bytes, bar);
        }
        // the tile's base rows (read back by the flushes) into L2
        for (int mask = prog.prefetch_mask, k = 0; mask; mask >>= 1, ++k)
            if (mask & 1)
                bulk_prefetch(static_cast<const T *>(prog.ops[k].base ? prog.ops[k].base : prog.ops[k].base2) +
                                  (size_t)l0 * n,
                              row_bytes * (uint32_t)rows);
    };
    const ChunkScratch<T> sc = carve_scratch<T>(smem_raw + (PERSIST ? 2 : 1) * slot_bytes, C, W);
    // staging rows for plain outputs, after the responses (128-byte aligned)
    T *out_s = reinterpret_cast<T *>(
        smem_raw + ((reinterpret_cast<unsigned char *>(resp_s + prog.nops * 4 * L) - smem_raw + 127) & ~(size_t)127));
    const int cs = c * L;
    const int nv = min(L, n - cs);
    pdl_wait();
    long tile = blockIdx.x;
    if (t == 0) {
        if (PERSIST) s_tile[0] = tile = (long)atomicAdd(claim, 1ull);
        if (tile < ntiles) issue(tile, 0);
    }
    __syncthreads();
    if (PERSIST) tile = s_tile[0];
    for (int it = 0; tile < ntiles; ++it) {
        const int slot = PERSIST ? (it & 1) : 0;
        const uint32_t parity = PERSIST ? ((it >> 1) & 1) : 0;
        const bool ok = mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
        // this barrier also ends every thread's reads of the other slot (the
        // previous tile), so the next tile's copies may go there now
        if (!__syncthreads_and(ok)) {
            if (t == 0) {
                atomicExch(err, 1);
                mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
            }
            if (t < W) bulk_wait_all();
            return;
        }
        if (PERSIST && t == 0) {
            const long next = (long)atomicAdd(claim, 1ull);
            s_tile[(it + 1) & 1] = next;  // read after this tile's barriers
            if (next < ntiles) issue(next, slot ^ 1);
        }
        const long l0 = tile * W;
        const int rows = (int)min((long)W, nlines - l0);
        const int lr = l < rows ? l : 0;  // rows past the end compute on row 0 and store nothing
        unsigned char *base = smem_raw + slot * slot_bytes;
        fill_halos_x<T>(base, tile_bytes, prog.ntiles, rows, pitch, n);
        fence_proxy_async_smem();  // halo elements are refilled by bulk copies two tiles later
        __syncthreads();
        // window of this chunk: elements cs .. cs+L+7 (points cs-4 .. cs+L+3)
        auto row = [&](int ti) {
            return reinterpret_cast<const T *>(base + ti * tile_bytes) + (size_t)lr * pitch + cs;
        };
        auto tile_at = [&](int ti, int j) { return *reinterpret_cast<const VT *>(row(ti) + kHalo + j); };
        auto flush_args = [&](const StageOp<T> &so) {
            return FlushArgs<T>(so, so.base2_tile >= 0 ? row(so.base2_tile) + kHalo : nullptr, 1);
        };
        T r[L];
        T acc[ACC ? L : 1];
        for (int k = 0; k < prog.nops; ++k) {
            const StageOp<T> &so = prog.ops[k];
            const T *ra = row(so.src_a);
            const T *rb = so.src_b >= 0 ? row(so.src_b) : nullptr;
            auto load = [&](auto &w, auto j0) {
                constexpr int J0 = decltype(j0)::value;
                constexpr int NW = sizeof(w) / sizeof(T);
                if (rb) {
#pragma unroll
                    for (int j = 0; j < NW; j += V) {
                        const VT qa = *reinterpret_cast<const VT *>(ra + J0 + j);
                        const VT qb = *reinterpret_cast<const VT *>(rb + J0 + j);
                        const T *ea = reinterpret_cast<const T *>(&qa);
                        const T *eb = reinterpret_cast<const T *>(&qb);
#pragma unroll
                        for (int v = 0; v < V; ++v) w[j + v] = ea[v] * eb[v];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NW; j += V) {
                        const VT qa = *reinterpret_cast<const VT *>(ra + J0 + j);
                        const T *ea = reinterpret_cast<const T *>(&qa);
#pragma unroll
                        for (int v = 0; v < V; ++v) w[j + v] = ea[v];
                    }
                }
            };
            // the previous operator's row copies must have read the staging
            // rows before anyone writes them again (after this solve's barriers)
            if (t < W) bulk_wait_read_all();
            chunk_solve_resp<T, L, !ACC>(so.op, so.kind, resp_s + k * 4 * L, load, r, sc, W, l, c, C, nv, c * W + l,
                                         so.keep);
            if constexpr (ACC) {
                accumulate<T, L, V>(so, acc, r, nv, tile_at);
                if (so.flush) flush_x_staged<T, L, true>(flush_args(so), acc, out_s, l, l0, rows, pitch, n, cs, nv);
            } else {
                if (so.flush) flush_x_staged<T, L, false>(flush_args(so), r, out_s, l, l0, rows, pitch, n, cs, nv);
                // from the staging rows, which the next operator writes only
                // after its solve's barriers
                if constexpr (SHIFT)
                    if (so.shift_out) flush_rows_shifted<T, true>(so.shift_out, out_s, l0, rows, pitch, n);
            }
        }
        if (!PERSIST) break;
        tile = s_tile[(it + 1) & 1];  // as in ls_stage_yz
    }
    if (t < W) bulk_wait_all();
}

// ---------------------------------------------------------------------------
// Host side.

PFN_cuTensorMapEncodeTiled_v12000 encode_tiled()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

static size_t scratch_bytes(int C, int W, size_t es) { return ((size_t)2 * C * W * es + 15) & ~(size_t)15; }

static bool al8(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; }

template <typename Kern>
static unsigned persistent_grid(x3d_ctx_s *ctx, Kern kern, int threads, size_t smem, long ntiles)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    const long g = (long)ctx->num_sms * (per_sm < 1 ? 1 : per_sm);
    return (unsigned)(g < ntiles ? g : ntiles);
}

// Whether the tiled and bulk copies can move a program's fields: rows of
// whole 16-byte units, 16-byte aligned inputs and, along x, outputs.
template <typename T>
static bool whole_vectors(const StageProgram<T> &p, int dir, int nx)
{
    if (((size_t)nx * (p.in_f64 ? sizeof(double) : sizeof(T))) % 16) return false;
    for (int ti = 0; ti < p.ntiles; ++ti)
        if (!al16(p.in[ti])) return false;
    for (int k = 0; k < p.nops && dir == DX; ++k) {
        const StageOp<T> &so = p.ops[k];
        if (so.flush && (!al16(so.out) || !al16(so.base) || !al16(so.out2) || !al16(so.base2) || !al16(so.shift_out)))
            return false;
    }
    return true;
}

template <typename T>
static void fill_resp(StageProgram<T> &p, int L, int n)
{
    for (int k = 0; k < p.nops; ++k) p.ops[k].keep = fill_op_resp(p.ops[k].resp, p.ops[k].op.alfa, L, n);
}

// PR = 2: the paired y/z kernel (FP32 only).  OCC > 1: the y/z kernel built
// for OCC CTAs per SM (plain programs, at most 256 threads).  Persistent
// kernels claim their tiles from the context's counter, zeroed here before
// each launch.
template <typename T, int W, int L, bool PERSIST, int PR = 1, int OCC = 1>
static int launch_stage_cfg(x3d_ctx_s *ctx, const StageProgram<T> &prog_in, int dir, int nx, int ny,
                            int nz)
{
    if constexpr (PR == 2 && !std::is_same<T, float>::value) {
        return X3D_EUNSUPPORTED;
    } else {
        StageProgram<T> prog = prog_in;
        // base2 that is a staged input comes from shared memory; T-typed bases
        // are prefetched into L2 with the tile's inputs
        for (int k = 0; k < prog.nops; ++k) {
            StageOp<T> &so = prog.ops[k];
            so.base2_tile = -1;
            for (int ti = 0; ti < prog.ntiles; ++ti)
                if (!so.out_f64 && so.base2 && so.base2 == prog.in[ti]) so.base2_tile = (short)ti;
            so.prefetch_base = (so.flush && !so.out_f64 && (so.base || (so.base2 && so.base2_tile < 0))) ? 1 : 0;
        }
        prog.prefetch_mask = 0;
        for (int k = 0; k < prog.nops; ++k)
            if (prog.ops[k].prefetch_base) prog.prefetch_mask |= 1 << k;
        // the ACC kernels carry the accumulator and every flush form; the
        // others only plain operators (out = the solve)
        const bool acc = program_acc(prog);
        bool shift = false;  // plain programs only (plain_program)
        for (int k = 0; k < prog.nops; ++k) shift = shift || prog.ops[k].shift_out;
        const int n = prog.ops[0].op.n;
        for (int k = 0; k < prog.nops; ++k)
            if (!prog.ops[k].op.circ || prog.ops[k].op.n != n) return X3D_EUNSUPPORTED;
        const size_t es = sizeof(T);
        const int C = (n + L - 1) / L;
        const int threads = C * W / PR;
        // FP64 inputs of an FP32 program: staged as FP64 by the plain,
        // unpaired y/z kernels only
        const bool in64 = prog.in_f64 != 0;
        if (in64 && (!std::is_same<T, float>::value || PR != 1 || OCC != 1 || acc || dir == DX))
            return X3D_EUNSUPPORTED;
        const size_t resp_bytes = (size_t)prog.nops * 4 * L * es * PR;
        if (!whole_vectors(prog, dir, nx)) {
            if constexpr (PR == 1 && OCC == 1 && !PERSIST && L == kChunkLong<T> && W <= 16)
                if (!prog.aligned_only) {
                    fill_resp(prog, L, n);
                    // FP32: 32 lines a tile where plain programs still fit 256
                    // threads.  A warp then holds one chunk of 32 lines, so a
                    // short last chunk does not run beside a full one in the
                    // same warp (250 x 171 x 129 sweep 189 -> 155 us; six y
                    // operators 10.9 us against 15.4 with 16 lines at 65^3, 18.9
                    // and 26.0 at 97^3, 173 and 229 at 255^3; behind only where
                    // a last tile of a column or so adds a fourth, 29.0 and 24.3
                    // at 129^3; FP64 lines of that length do not fit)
                    const bool wide = W == 16 && sizeof(T) == 4 && !acc && C * 32 <= 256;
                    int lines = wide ? 32 : W;
                    if (W == 16 && dir == DX) lines = x_tile_lines(lines, C, (long)ny * nz, ctx->num_sms, es);
                    if constexpr (W == 16)
                        if (lines == 8) return launch_stage_any<T, 8>(ctx, prog, acc, dir, nx, ny, nz);
                    if constexpr (W == 16 && sizeof(T) == 4)
                        if (lines == 32) {
                            const int rc = launch_stage_any<T, 32>(ctx, prog, acc, dir, nx, ny, nz);
                            if (rc != X3D_EUNSUPPORTED) return rc;
                        }
                    return launch_stage_any<T, W>(ctx, prog, acc, dir, nx, ny, nz);
                }
            return X3D_EUNSUPPORTED;
        }
        if (threads > kStageThreads<T, L, PR> || threads % 32) return X3D_EUNSUPPORTED;
        if (OCC > 1 && (acc || threads > 256)) return X3D_EUNSUPPORTED;
        cudaStream_t st = ctx->stream;
        if constexpr (PR == 2) {
            // paired y/z lines: even x extent; pairs are loaded and stored whole,
            // 8 bytes of FP32 or 16 of FP64
            if (dir == DX || nx % 2) return X3D_EUNSUPPORTED;
            for (int k = 0; k < prog.nops; ++k) {
                const StageOp<T> &so = prog.ops[k];
                auto pairs = [&](const void *p) { return so.out_f64 ? al16(p) : al8(p); };
                if (so.flush && (!pairs(so.out) || !pairs(so.base) || !pairs(so.out2) || !pairs(so.base2) ||
                                 !al8(so.shift_out)))
                    return X3D_EUNSUPPORTED;
            }
        } else if (dir == DX) {
            constexpr int V = Vec4<T>::N;
            // row: kHalo halo elements, the line, and room for the last chunk's window
            int pitch = C * L + 2 * kHalo;
            while (((size_t)pitch * es / 16) % 2 == 0) pitch += V;
            const size_t tile = ((size_t)W * pitch * es + 127) & ~(size_t)127;
            // + staging rows for plain outputs (W rows of the same pitch, 128-byte aligned)
            const size_t smem = (((PERSIST ? 2 : 1) * prog.ntiles * tile + scratch_bytes(C, W, es) + resp_bytes + 127) &
                                 ~(size_t)127) +
                                (size_t)W * pitch * es;
            if (smem + 1024 > ctx->smem_optin) return X3D_EUNSUPPORTED;
            fill_resp(prog, L, n);
            auto kern = shift ? ls_stage_x<T, W, L, false, PERSIST, OCC, true> : ls_stage_x<T, W, L, false, PERSIST, OCC>;
            if constexpr (OCC == 1)  // the OCC > 1 kernels take plain programs only
                if (acc) kern = ls_stage_x<T, W, L, true, PERSIST>;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            const long nlines = (long)ny * nz;
            const long ntiles = (nlines + W - 1) / W;
            const unsigned grid = PERSIST ? persistent_grid(ctx, kern, threads, smem, ntiles) : (unsigned)ntiles;
            if (PERSIST) {
                const int rc = cuda_check(ctx, cudaMemsetAsync(ctx->d_claim, 0, sizeof(*ctx->d_claim), st),
                                          "tile counter reset");
                if (rc) return rc;
            }
            ++ctx->launches;
            return cuda_check(ctx, launch_pdl(kern, ntiles, grid, threads, smem, st, prog, nlines, pitch, tile, ntiles,
                                              ctx->d_claim, ctx->d_err),
                              "ls_stage_x launch");
        }
        auto enc = encode_tiled();
        const size_t esi = in64 ? sizeof(double) : es;  // staged element bytes
        if (!enc) return X3D_EUNSUPPORTED;
        const int nb = (n + 255) / 256;
        int box_n = (n + nb - 1) / nb;
        const int align_rows = (int)(128 / (W * esi) > 0 ? 128 / (W * esi) : 1);
        box_n = (box_n + align_rows - 1) / align_rows * align_rows;
        if (box_n > 256) return X3D_EUNSUPPORTED;
        // rows: kHalo halo rows (kHalo * W * esi is a multiple of 128 bytes, so the
        // boxes land 128-byte aligned), the boxes, and room for the last window
        const int rows = kHalo + std::max(nb * box_n, C * L + kHalo);
        const size_t tile = ((size_t)rows * W * esi + 127) & ~(size_t)127;
        const size_t smem = (PERSIST ? 2 : 1) * prog.ntiles * tile + scratch_bytes(C, W, es) + resp_bytes;
        if (smem + 1024 > ctx->smem_optin) return X3D_EUNSUPPORTED;
        fill_resp(prog, L, n);
        StageMaps maps;
        std::memset(&maps, 0, sizeof(maps));
        auto encode = [&](CUtensorMap *m, const void *ptr, int rows_in_box, size_t eb) {
            cuuint64_t gdim[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
            cuuint64_t gstride[2] = {(cuuint64_t)nx * eb, (cuuint64_t)nx * ny * eb};
            cuuint32_t box[3] = {(cuuint32_t)W, 1, 1};
            box[dir == DY ? 1 : 2] = (cuuint32_t)rows_in_box;
            cuuint32_t estr[3] = {1, 1, 1};
            return enc(m, eb == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
                       const_cast<void *>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
        };
        for (int ti = 0; ti < prog.ntiles; ++ti)
            if (!encode(&maps.m[ti], prog.in[ti], box_n, esi)) return X3D_EUNSUPPORTED;
        // the periodic halos come by TMA too where the boxes end exactly at the
        // line's end (a box running past it would fill the rows after the line
        // with zeros); otherwise the kernel copies them in shared memory
        int tma_halo = nb * box_n == n ? 1 : 0;
        for (int ti = 0; ti < prog.ntiles && tma_halo; ++ti)
            if (!encode(&maps.hm[ti], prog.in[ti], kHalo, esi)) tma_halo = 0;
        for (int k = 0; k < prog.nops; ++k)
            if (prog.ops[k].prefetch_base &&
                !encode(&maps.pm[k], prog.ops[k].base ? prog.ops[k].base : prog.ops[k].base2, box_n, es))
                prog.ops[k].prefetch_base = 0;
        prog.prefetch_mask = 0;
        for (int k = 0; k < prog.nops; ++k)
            if (prog.ops[k].prefetch_base) prog.prefetch_mask |= 1 << k;
        auto kern = shift ? ls_stage_yz<T, W, L, false, PERSIST, PR, OCC, T, true>
                          : ls_stage_yz<T, W, L, false, PERSIST, PR, OCC>;
        if constexpr (OCC == 1)  // the OCC > 1 kernels take plain programs only
            if (acc) kern = ls_stage_yz<T, W, L, true, PERSIST, PR, OCC>;
        if constexpr (std::is_same<T, float>::value && PR == 1 && OCC == 1)
            if (in64) kern = ls_stage_yz<T, W, L, false, PERSIST, PR, OCC, double>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        const long tiles_x = (nx + W - 1) / W;
        const long ntiles = tiles_x * (dir == DY ? nz : ny);
        const unsigned grid = PERSIST ? persistent_grid(ctx, kern, threads, smem, ntiles) : (unsigned)ntiles;
        if (PERSIST) {
            const int rc = cuda_check(ctx, cudaMemsetAsync(ctx->d_claim, 0, sizeof(*ctx->d_claim), st),
                                      "tile counter reset");
            if (rc) return rc;
        }
        ++ctx->launches;
        return cuda_check(ctx, launch_pdl(kern, ntiles, grid, threads, smem, st, maps, prog, nx, ny, dir, box_n, nb, tma_halo,
                                          tile, ntiles, ctx->d_claim, ctx->d_err),
                          "ls_stage_yz launch");

    }
}

template <typename T>
static int launch_stage_sel(x3d_ctx_s *ctx, const StageProgram<T> &prog, int dir, int nx, int ny, int nz, int cfg);

template <typename T>
int launch_stage(x3d_ctx_s *ctx, const StageProgram<T> &prog, int dir, int nx, int ny, int nz, int cfg)
{
    const int rc = launch_stage_sel<T>(ctx, prog, dir, nx, ny, nz, cfg);
    if (rc == X3D_OK) ctx->last_cfg = cfg;
    return rc;
}

template <typename T>
static int launch_stage_sel(x3d_ctx_s *ctx, const StageProgram<T> &prog, int dir, int nx, int ny, int nz, int cfg)
{
    if (prog.nops < 1 || prog.nops > kMaxStageOps || prog.ntiles < 1 || prog.ntiles > kMaxStageTiles)
        return X3D_EINVAL;
    // cfg selects (lines per CTA, chunk length).
    constexpr int Lbig = sizeof(T) == 4 ? 32 : 16;
    constexpr int Lsmall = sizeof(T) == 4 ? 16 : 8;
    // 0-5: one CTA per tile; 6-11: the same shapes, persistent with two slots
    switch (cfg) {
    case 0: return launch_stage_cfg<T, 16, Lbig, false>(ctx, prog, dir, nx, ny, nz);
    case 1: return launch_stage_cfg<T, 32, Lbig, false>(ctx, prog, dir, nx, ny, nz);
    case 2: return launch_stage_cfg<T, 16, Lsmall, false>(ctx, prog, dir, nx, ny, nz);
    case 3: return launch_stage_cfg<T, 8, Lbig, false>(ctx, prog, dir, nx, ny, nz);
    case 4: return launch_stage_cfg<T, 32, Lsmall, false>(ctx, prog, dir, nx, ny, nz);
    case 5: return launch_stage_cfg<T, 8, Lsmall, false>(ctx, prog, dir, nx, ny, nz);
    case 6: return launch_stage_cfg<T, 16, Lbig, true>(ctx, prog, dir, nx, ny, nz);
    case 7: return launch_stage_cfg<T, 32, Lbig, true>(ctx, prog, dir, nx, ny, nz);
    case 8: return launch_stage_cfg<T, 16, Lsmall, true>(ctx, prog, dir, nx, ny, nz);
    case 9: return launch_stage_cfg<T, 8, Lbig, true>(ctx, prog, dir, nx, ny, nz);
    case 10: return launch_stage_cfg<T, 32, Lsmall, true>(ctx, prog, dir, nx, ny, nz);
    case 11: return launch_stage_cfg<T, 8, Lsmall, true>(ctx, prog, dir, nx, ny, nz);
    // 12-15: y/z lines in packed pairs (FP32, even nx)
    case 12: return launch_stage_cfg<T, 32, Lsmall, true, 2>(ctx, prog, dir, nx, ny, nz);
    case 13: return launch_stage_cfg<T, 16, Lsmall, true, 2>(ctx, prog, dir, nx, ny, nz);
    case 14: return launch_stage_cfg<T, 32, Lsmall, false, 2>(ctx, prog, dir, nx, ny, nz);
    case 15: return launch_stage_cfg<T, 32, Lbig, true, 2>(ctx, prog, dir, nx, ny, nz);
    // 17: configuration 6 (y/z) compiled for three CTAs per SM (plain programs)
    case 17: return launch_stage_cfg<T, 16, Lbig, true, 1, 3>(ctx, prog, dir, nx, ny, nz);
    // 18: configuration 9 (8 lines, long chunks, y/z) built for three CTAs per SM
    case 18: return launch_stage_cfg<T, 8, Lbig, true, 1, 3>(ctx, prog, dir, nx, ny, nz);
    // 19: configuration 3 (8 lines, long chunks, one CTA per tile) built for
    // three CTAs per SM: with one staging slot the FP64 x tiles fit three
    case 19: return launch_stage_cfg<T, 8, Lbig, false, 1, 3>(ctx, prog, dir, nx, ny, nz);
    // 20: configuration 0 (16 lines, long chunks, one CTA per tile) built for
    // three CTAs per SM
    case 20: return launch_stage_cfg<T, 16, Lbig, false, 1, 3>(ctx, prog, dir, nx, ny, nz);
    default: return X3D_EUNSUPPORTED;
    }
}

// Which configuration an untuned program takes was measured on 41 boxes of 16
// to 384 points a side, cubes and flat ones, both precisions: every
// configuration on one and six operators and on the nine fused stages of a step.
//
// Fields above 24 MiB fill the SMs many times over, and the order is the same
// for all of them: the kernels built for three CTAs per SM for plain programs
// (384^3 FP64, six y operators: 541 us on 19, 889 on 0; 256^3 FP32 y 92 on
// 20, 106 on 0), pairs of lines a thread for FP32 y/z momentum (256^3 z 198 on
// 14, 236 on 0), 8-line tiles for FP64 x programs that accumulate, whose three
// staged fields then fit more CTAs (256^3 momentum x 313 on 3, 460 on 0).
//
// Below that what matters is how the tiles of a configuration divide into
// waves, and no line through the sizes holds: stage_cost estimates each
// configuration's time from its waves, and one that comes out at least a tenth
// below the long-chunk default replaces it.  It was fitted before derpv and
// interpv became second outputs of their twins' solves; over 270 launches since
// (22 boxes up to 24 MiB, one and six operators) the pick is on average 4 and 5 %
// behind the fastest configuration and 9 and 18 % ahead of 0 (64^3 FP32, six y
// operators: 7.6 us on 2, 7.3 on 4, 10.7 on 0), at worst 40 % behind (112^3
// FP32 along y: 19.9 us on the picked, 14.2 on 0).  nops counts every operator
// of the list, whether or not it gets a solve of its own; counting solves
// instead picks the same.  Rows that are not whole 16-byte units are the business
// of linesolve_any.cu, reached through configuration 0 or 3, whichever of the
// pick or the order after it comes first.
//
// The persistent configurations are left to the autotuner, although 17 is up
// to 8 % ahead of 20: they claim tiles from the context's one counter, and an
// untuned context may be moved between streams with launches in flight.
struct StageShape {
    int W, L, PR, regs, threads, ctas, per_sm;  // threads: 0 where it does not fit
};

// Tile width, chunk, resident CTAs of configuration cfg for a program.
static StageShape stage_shape(int cfg, size_t es, int dir, int nx, int ny, int nz, int ntiles, int nops, bool acc,
                              bool in64)
{
    const int n = dir == DX ? nx : (dir == DY ? ny : nz);
    const int Llong = es == 4 ? 32 : 16;
    StageShape s{};
    s.PR = cfg == 14 ? 2 : 1;
    s.regs = cfg >= 19 ? 80 : 128;
    s.W = cfg == 3 || cfg == 5 || cfg == 19 ? 8 : (cfg == 1 || cfg == 4 || cfg == 14 ? 32 : 16);
    s.L = cfg == 2 || cfg == 4 || cfg == 5 || cfg == 14 ? Llong / 2 : Llong;
    const int C = (n + s.L - 1) / s.L, threads = C * s.W / s.PR;
    if (threads % 32 || threads > (cfg >= 19 ? 256 : 512) || (cfg >= 19 && (acc || in64))) return s;
    if (cfg == 14 && (es != 4 || dir == DX || nx % 2 || in64)) return s;
    const size_t line = (size_t)s.W * (C * s.L + 2 * kHalo);
    const size_t smem = line * (dir == DX ? (ntiles + 1) * es : ntiles * (in64 ? 8 : es)) + (size_t)2 * C * s.W * es +
                        (size_t)nops * 4 * s.L * es * s.PR + 1024;
    if (smem > (size_t)228 * 1024) return s;
    s.threads = threads;
    const long lines = dir == DX ? (long)ny * nz : nx;
    const long tiles = (lines + s.W - 1) / s.W * (dir == DX ? 1 : (dir == DY ? nz : ny));
    s.ctas = (int)std::min<long>(tiles, 1 << 30);
    s.per_sm = std::max(1, std::min({65536 / (s.regs * threads), (int)(228 * 1024 / smem), 32, 2048 / threads}));
    return s;
}

// Estimated microseconds of a launch of at most a few waves: a wave costs a
// start, its operators one after another at a warp's own pace (a constant and
// a slope in the chunk length) or, with r CTAs on an SM, at the SM's, and the
// movement of its tiles.  The constants are a least-squares fit of the
// logarithm to the measured launches up to 24 MiB (16 % rms).
static double stage_cost(const StageShape &s, size_t es, int dir, int ntiles, int nops, bool acc, int num_sms)
{
    const bool f = es == 4, x = dir == DX;
    const double op0 = f ? 0.2595 : 1.03, opL = f ? 0.06694 : 0.04398, issue = f ? 0.007064 : 0.01147;
    const double start = f ? 0.2606 : 0.6114, move = f ? 1.011 : 0.007316;
    const double kx = x ? 1.113 : 1.0, ka = acc ? 1.254 : 1.0, pair = s.PR == 2 ? 1.104 : 1.0;
    const double alone = (op0 + opL * s.L * (s.PR == 2 ? 1.15 : 1.0)) * nops * kx * ka;
    const double a4 = alone * alone * alone * alone;
    auto wave = [&](int r) {
        const double shared = r * (s.threads / 32) * s.L * nops * issue * kx * ka * pair * (s.W == 8 ? 1.125 : 1.0);
        return start * kx + (x ? 0.0475 * s.W * ntiles : 0.0) +
               std::sqrt(std::sqrt(a4 + shared * shared * shared * shared)) * (s.PR == 2 && acc ? 1.217 : 1.0) +
               move * 1e-5 * r * s.threads * s.L * s.PR * (double)es;
    };
    const int slots = num_sms * s.per_sm, full = s.ctas / slots, rest = s.ctas - full * slots;
    return 2.0 + full * wave(s.per_sm) + (rest ? wave((rest + num_sms - 1) / num_sms) : 0.0);
}

static DefaultCfgs weigh_cfgs(size_t es, int dir, int nx, int ny, int nz, int ntiles, int nops, bool acc, bool in64,
                              int num_sms)
{
    const bool f32 = es == 4;
    if ((size_t)nx * ny * nz * es > (size_t)24 << 20) {
        if (dir == DX) {
            if (acc) return f32 ? DefaultCfgs{2, {0, 3}} : DefaultCfgs{2, {3, 0}};
            if (f32 && ntiles > 1) return {3, {5, 19, 0}};
            return {3, {19, 20, 0}};
        }
        if (acc) return f32 && nops == 6 ? DefaultCfgs{2, {14, 0}} : DefaultCfgs{2, {0, 3}};
        if (in64) return {1, {0}};
        return {3, {20, 19, 0}};
    }
    static const int cand[] = {0, 1, 2, 3, 4, 5, 14, 19, 20};
    int base = -1, best = -1;
    double tbase = 0.0, tbest = 0.0;
    for (const int cfg : cand) {
        const StageShape s = stage_shape(cfg, es, dir, nx, ny, nz, ntiles, nops, acc, in64);
        if (!s.threads) continue;
        // 32 row copies issued by one thread: only where nothing else fits
        if (cfg == 4 && dir == DX && base >= 0) continue;
        const double t = stage_cost(s, es, dir, ntiles, nops, acc, num_sms);
        if (base < 0) base = cfg, tbase = t;
        if (best < 0 || t < tbest) best = cfg, tbest = t;
    }
    if (base < 0) return {1, {0}};
    if (tbest < 0.9 * tbase) return {2, {best, base}};
    return {1, {base}};
}

DefaultCfgs default_cfgs(size_t es, int dir, int nx, int ny, int nz, int ntiles, int nops, bool acc, bool in64,
                         int num_sms)
{
    thread_local CfgPicks<64> picks;
    return picks.get({{(int)es, dir, nx, ny, nz, ntiles, nops, acc, in64, num_sms}},
                     [&] { return weigh_cfgs(es, dir, nx, ny, nz, ntiles, nops, acc, in64, num_sms); });
}

template <typename T>
StageProgram<T> plain_program(const T *in, const LineOp<T> *const *ops, const int *kinds,
                              void *const *outs, int nops)
{
    StageProgram<T> p{};
    p.ntiles = 1;
    p.in[0] = in;
    // twin[k] = j: operator k is j's shifted twin, written by j's solve (one
    // twin a solve; not where the list names an output twice, whose order of
    // writes it would change)
    int twin[kMaxStageOps];
    bool taken[kMaxStageOps] = {};
    for (int k = 0; k < nops; ++k) {
        twin[k] = -1;
        bool twice = false;
        for (int j = 0; j < nops; ++j) twice = twice || (j != k && outs[j] == outs[k]);
        for (int j = 0; j < nops && twin[k] < 0 && !twice; ++j)
            if (j != k && !taken[j] && shifted_twin<T>(*ops[j], kinds[j], *ops[k], kinds[k])) {
                twin[k] = j;
                taken[j] = true;
            }
    }
    for (int k = 0; k < nops; ++k) {
        if (twin[k] >= 0) continue;
        StageOp<T> &so = p.ops[p.nops++];
        so.op = *ops[k];
        so.kind = kinds[k];
        so.src_a = 0;
        so.src_b = -1;
        so.mul_tile = -1;
        so.accumulate = 0;
        so.flush = 1;
        so.out = outs[k];
        so.base = nullptr;
        so.out2 = nullptr;
        so.base2 = nullptr;
        so.sign = 1.0;
        so.scale2 = 0.0;
        so.out_f64 = 0;
        for (int j = 0; j < nops; ++j)
            if (twin[j] == k) so.shift_out = outs[j];
    }
    return p;
}

template int launch_stage<float>(x3d_ctx_s *, const StageProgram<float> &, int, int, int, int, int);
template int launch_stage<double>(x3d_ctx_s *, const StageProgram<double> &, int, int, int, int, int);
template StageProgram<float> plain_program<float>(const float *, const LineOp<float> *const *,
                                                  const int *, void *const *, int);
template StageProgram<double> plain_program<double>(const double *, const LineOp<double> *const *,
                                                    const int *, void *const *, int);

}  // namespace x3d
