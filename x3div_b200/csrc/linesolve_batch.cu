// Batches of uneven boxes: one persistent launch applies the operator groups
// of every (box, field, direction) job.  CTAs pull tiles from a global
// counter, so boxes of different sizes balance across the SMs; each tile
// uses its job's lines per tile (W), chunk count (C), tensor map or padded
// rows.  Threads beyond W*C of a job idle through its barriers.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstddef>

#include "chunk_solve.cuh"
#include "linesolve_chunk.h"
#include "ptx.cuh"
#include "x3d_internal.h"

namespace x3d {

// Carry scratch, then the carry responses of the item's operators.
template <typename T>
constexpr size_t batch_scratch_bytes_c()
{
    return (((size_t)2 * kBatchThreads * sizeof(T) + 15) & ~(size_t)15) +
           (size_t)kMaxStageOps * 4 * kChunkLong<T> * sizeof(T);
}

// Byte offset of the x staging rows: after the two slots, the scratch and
// the responses, 128-byte aligned.
template <typename T>
__host__ __device__ constexpr size_t batch_out_offset(size_t tile_cap)
{
    return (2 * tile_cap + batch_scratch_bytes_c<T>() + 127) & ~(size_t)127;
}

// One work item of the batch kernel with chunk length L (the job's): the
// operators of the job solved over the staged tile and written out.  y/z
// outputs go straight to global memory, coalesced across the tile's lines;
// x outputs either go straight out as each thread's 16-byte vectors or, for
// jobs with xstage set, are staged in shared-memory rows (out_s, the tile's
// pitch) and leave as one bulk copy per row, as in ls_stage_x.
template <typename T, int L, bool XS, bool SHIFT>
__device__ __forceinline__ void batch_item(const BatchJob<T> &J, const T *tile, T *out_s, const T *resp_s,
                                           const ChunkScratch<T> &scf, int t, long l0, int rows, int x0, int o)
{
    using VT = typename Vec4<T>::type;
    constexpr int V = Vec4<T>::N;
    const int W = J.W, C = J.C, n = J.n;
    const int dir = J.dir;
    const bool active = t < W * C;
    const int l = active ? t % W : 0, c = active ? t / W : 0;
    const int q = t;  // scratch slot: active threads use c*W + l == t
    ChunkScratch<T> sc = scf;
    const int cs = c * L;
    const int nv = min(L, n - cs);
    T r[L];
    if (dir == DX) {
        const int lr = l < rows ? l : 0;
        const T *row = tile + (size_t)lr * J.pitch + cs;  // points cs-4 .. cs+L+3
        auto load = [&](auto &w, auto j0) {
            constexpr int J0 = decltype(j0)::value;
            constexpr int NW = sizeof(w) / sizeof(T);
#pragma unroll
            for (int j = 0; j < NW; j += V) {
                const VT qa = *reinterpret_cast<const VT *>(row + J0 + j);
                const T *ea = reinterpret_cast<const T *>(&qa);
#pragma unroll
                for (int v = 0; v < V; ++v) w[j + v] = ea[v];
            }
        };
        for (int k = 0; k < J.nops; ++k) {
            // the previous operator's row copies have read the staging
            // rows before anyone writes them again (after this solve's barriers)
            if (XS) bulk_wait_read_all();
            chunk_solve_resp<T, L, true>(J.op[k], J.kind[k], resp_s + k * 4 * L, load, r, sc, W, l, c, C, nv,
                                         q, J.keep[k]);
            if (!XS || !J.xstage) {  // each thread's chunk straight out, 16 bytes at a time
                if (active && l < rows) {
                    T *dst = J.out[k] + (size_t)(l0 + l) * n + cs;
#pragma unroll
                    for (int j = 0; j < L; j += V) {
                        if (j < nv) {
                            VT qv;
                            T *e = reinterpret_cast<T *>(&qv);
#pragma unroll
                            for (int v = 0; v < V; ++v) e[v] = r[j + v];
                            *reinterpret_cast<VT *>(dst + j) = qv;
                        }
                    }
                }
                if (SHIFT && J.shift_out[k]) {
                    // one point on: the chunk's first point is the end of the
                    // chunk before, passed through the scratch that held the
                    // forward ends (read before the solve's second barrier)
                    T end = T(0);
#pragma unroll
                    for (int j = 0; j < L; ++j)
                        if (j + 1 == nv) end = r[j];
                    sc.fz[q] = end;
                    __syncthreads();
                    T prev = sc.fz[(c ? c - 1 : C - 1) * W + l];
                    if (active && l < rows) {
                        T *dst = J.shift_out[k] + (size_t)(l0 + l) * n + cs;
#pragma unroll
                        for (int j = 0; j < L; j += V) {
                            if (j < nv) {
                                VT qv;
                                T *e = reinterpret_cast<T *>(&qv);
                                e[0] = prev;
#pragma unroll
                                for (int v = 1; v < V; ++v) e[v] = r[j + v - 1];
                                prev = r[j + V - 1];
                                *reinterpret_cast<VT *>(dst + j) = qv;
                            }
                        }
                    }
                    __syncthreads();  // before the next operator writes the scratch
                }
                continue;
            }
            if (active && l < rows) {
                T *dst = out_s + (size_t)l * J.pitch + cs;  // room for the last window past n
#pragma unroll
                for (int j = 0; j < L; j += V) {
                    VT qv;
                    T *e = reinterpret_cast<T *>(&qv);
#pragma unroll
                    for (int v = 0; v < V; ++v) e[v] = r[j + v];
                    *reinterpret_cast<VT *>(dst + j) = qv;
                }
            }
            fence_proxy_async_smem();
            __syncthreads();
            if (t < rows) {
                bulk_store(J.out[k] + (size_t)(l0 + t) * n, out_s + (size_t)t * J.pitch,
                           (uint32_t)(n * sizeof(T)));
                bulk_commit();
            }
            if (SHIFT && J.shift_out[k])
                flush_rows_shifted<T, true>(J.shift_out[k], out_s, l0, rows, J.pitch, n);
        }
    } else {
        const T *col = tile + (size_t)(J.halo + cs - 4) * W + l;  // points cs-4 .. cs+L+3
        auto load = [&](auto &w, auto j0) {
            constexpr int J0 = decltype(j0)::value;
            constexpr int NW = sizeof(w) / sizeof(T);
#pragma unroll
            for (int j = 0; j < NW; ++j) w[j] = col[(J0 + j) * W];
        };
        const bool live = active && x0 + l < J.nx;
        const size_t ostride = dir == DY ? (size_t)J.nx : (size_t)J.nx * J.ny;
        const size_t obase = (size_t)(x0 + l) +
                             (dir == DY ? (size_t)J.nx * J.ny * o : (size_t)J.nx * o) +
                             (size_t)cs * ostride;
        for (int k = 0; k < J.nops; ++k) {
            chunk_solve_resp<T, L, true>(J.op[k], J.kind[k], resp_s + k * 4 * L, load, r, sc, W, l, c, C, nv,
                                         q, J.keep[k]);
            if (live) {
                T *dst = J.out[k] + obase;
                if (nv == L) {  // every chunk but a short last one: no per-point test
#pragma unroll
                    for (int j = 0; j < L; ++j) {
                        *dst = r[j];
                        dst += ostride;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < L; ++j) {
                        if (j < nv) *dst = r[j];
                        dst += ostride;
                    }
                }
                if (SHIFT && J.shift_out[k])
                    flush_yz_shifted<T, T, L>(J.shift_out[k], r, obase, cs, ostride, nv, c == C - 1);
            }
        }
    }
}

// VAR (BatchVariant): kBatchLong runs every job with the long chunk and
// its x outputs straight out; kBatchMixed takes each job's chunk length;
// kBatchStaged also stages the x outputs of jobs with xstage set.  The
// narrower variants carry less code and no staging rows.
// Bytes of a job's header (every field before its responses), in 16-byte units.
template <typename T>
constexpr int kBatchHdrVecs = (int)((offsetof(BatchJob<T>, resp) + 15) / 16);

template <typename T, int VAR, bool SHIFT>
__global__ void __launch_bounds__(kBatchThreads, 2)
    ls_batch(const BatchJob<T> *__restrict__ jobs, int njobs, long total,
             unsigned long long *counter, size_t tile_cap, int *err)
{
    static_assert(kBatchHdrVecs<T> <= kBatchThreads, "one 16-byte copy per thread");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t bars[2];
    __shared__ long s_item;
    __shared__ int s_job;  // the job of s_item
    // the headers of the current and the next item's jobs, by iteration parity
    __shared__ __align__(64) uint4 s_hdr[2][kBatchHdrVecs<T>];
    const int t = threadIdx.x;
    // two staging slots of tile_cap bytes, then the carry scratch and the
    // carry responses of the item's operators
    const ChunkScratch<T> scf = carve_scratch<T>(smem_raw + 2 * tile_cap, kBatchThreads / 1, 1);
    T *resp_s = reinterpret_cast<T *>(smem_raw + 2 * tile_cap +
                                      (((size_t)2 * kBatchThreads * sizeof(T) + 15) & ~(size_t)15));
    // staging rows of x outputs (one tile's worth), after the responses
    T *out_s = reinterpret_cast<T *>(smem_raw + batch_out_offset<T>(tile_cap));
    auto job_of = [&](long item) {
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].tile0 <= item) lo = mid;
            else hi = mid - 1;
        }
        return lo;
    };
    // The copies of one work item of job jb into staging slot `slot` (one thread).
    auto issue = [&](long item, int jb, int slot) {
        const BatchJob<T> &J = jobs[jb];
        const long tl = item - J.tile0;
        T *tile = reinterpret_cast<T *>(smem_raw + slot * tile_cap);
        uint64_t *bar = &bars[slot];
        if (J.dir == DX) {
            const long l0 = tl * J.W;
            const int rows = (int)min((long)J.W, J.span - l0);
            const uint32_t row_bytes = (uint32_t)(J.n * sizeof(T));
            mbar_arrive_expect_tx(bar, row_bytes * (uint32_t)rows);
            for (int rr = 0; rr < rows; ++rr)
                bulk_load(tile + (size_t)rr * J.pitch + kHalo, J.in + (size_t)(l0 + rr) * J.n, row_bytes, bar);
        } else {
            const int x0 = (int)(tl % J.span) * J.W, o = (int)(tl / J.span);
            fence_tensormap_acquire(&J.tmap);
            mbar_arrive_expect_tx(bar, (uint32_t)((size_t)J.nbox * J.box_n * J.W * sizeof(T)));
            T *dst = tile + (size_t)J.halo * J.W;
            for (int b = 0; b < J.nbox; ++b) {
                if (J.dir == DY)
                    tma_load_3d(dst + (size_t)b * J.box_n * J.W, &J.tmap, bar, x0, b * J.box_n, o);
                else
                    tma_load_3d(dst + (size_t)b * J.box_n * J.W, &J.tmap, bar, x0, o, b * J.box_n);
            }
        }
    };
    // every thread copies at most one 16-byte piece of job jb's header
    auto copy_header = [&](int jb, int hs) {
        if (t < kBatchHdrVecs<T>) s_hdr[hs][t] = reinterpret_cast<const uint4 *>(jobs + jb)[t];
    };
    if (t == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
        s_item = (long)atomicAdd(counter, 1ull);
        if (s_item < total) {
            s_job = job_of(s_item);
            issue(s_item, s_job, 0);
        }
    }
    __syncthreads();
    if (s_item < total) copy_header(s_job, 0);
    uint32_t phases = 0;  // bit s: parity of slot s's next completion
    int resp_have = -1;   // the response class in resp_s (the same in every thread)
    for (int it = 0;; ++it) {
        const int slot = it & 1;
        const long item = s_item;  // claimed during the previous item (or above)
        if (item >= total) break;
        const int jb = s_job;
        unsigned char *tbase = smem_raw + slot * tile_cap;
        const T *tile = reinterpret_cast<const T *>(tbase);
        const uint32_t parity = (phases >> slot) & 1u;
        const bool ok = mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
        if (!__syncthreads_and(ok)) {
            if (t == 0) atomicExch(err, 1);
            mbar_wait_bounded(&bars[slot], parity, kChunkWaitNs);
            if (VAR == kBatchStaged) bulk_wait_all();
            return;
        }
        phases ^= 1u << slot;
        // The job's header, copied during the previous item (or above) and
        // ordered by the barrier just passed.  Every thread is done with the
        // previous item (its responses are read after its last barrier, its
        // tile and header before): this item's responses go in place, and the
        // next item, claimed now, is copied into the other slot while this
        // one is solved.
        const BatchJob<T> &J = *reinterpret_cast<const BatchJob<T> *>(s_hdr[slot]);
        const long tl = item - J.tile0;
        const int W = J.W, n = J.n;
        const int dir = J.dir;
        long l0 = 0;
        int rows = W, x0 = 0, o = 0;
        if (dir == DX) {
            l0 = tl * W;
            rows = (int)min((long)W, J.span - l0);
        } else {
            x0 = (int)(tl % J.span) * W;
            o = (int)(tl / J.span);
        }
        const int L = VAR == kBatchLong ? kChunkLong<T> : J.L;
        if (J.rclass != resp_have) {  // consecutive items mostly share a job, so this is rare
            const T *resp_g = &jobs[jb].resp[0][0][0];
            for (int i = t; i < J.nops * 4 * L; i += kBatchThreads) {
                const int k = i / (4 * L), rem = i - k * 4 * L, a = rem / L, j = rem - a * L;
                resp_s[i] = resp_g[(k * 4 + a) * kChunkLong<T> + j];
            }
            resp_have = J.rclass;
        }
        if (t == 0) {
            const long next = (long)atomicAdd(counter, 1ull);
            s_item = next;
            if (next < total) {
                const int nj = job_of(next);
                s_job = nj;
                issue(next, nj, slot ^ 1);
            }
        }
        if (dir == DX) fill_halos_x<T>(tbase, 0, 1, rows, J.pitch, n);
        else fill_halos_yz<T>(tbase, 0, 1, n, W, J.halo);
        fence_proxy_async_smem();  // copies into this slot two items later overwrite the halos
        __syncthreads();
        // the next item's header into the other slot, read after the next wait barrier
        if (s_item < total) copy_header(s_job, slot ^ 1);
        constexpr bool XS = VAR == kBatchStaged;
        if (VAR == kBatchLong || J.L == kChunkLong<T>)
            batch_item<T, kChunkLong<T>, XS, SHIFT>(J, tile, out_s, resp_s, scf, t, l0, rows, x0, o);
        else
            batch_item<T, kChunkShort<T>, XS, SHIFT>(J, tile, out_s, resp_s, scf, t, l0, rows, x0, o);
    }
    if (VAR == kBatchStaged) bulk_wait_all();  // x rows in flight (issued by this thread)
}


static int gcd_int(int a, int b) { return b ? gcd_int(b, a % b) : a; }

// Fills the geometry, tiling and staging fields of a job; false when the
// job's box cannot take the chunked batch kernel.
template <typename T>
bool plan_batch_job(BatchJob<T> &J, int L, int w_req, int xstage, size_t *tile_bytes)
{
    const size_t es = sizeof(T);
    const int n = J.n;
    constexpr int V = Vec4<T>::N;
    if (L != kChunkLong<T> && L != kChunkShort<T>) return false;
    for (int k = 0; k < J.nops; ++k)
        if (!J.op[k].circ || J.op[k].n != n) return false;
    for (int k = 0; k < J.nops; ++k) J.keep[k] = fill_op_resp(J.resp[k], J.op[k].alfa, L, n);
    J.L = L;
    J.C = (n + L - 1) / L;
    if (J.C > kBatchThreads) return false;
    int W = kBatchThreads / J.C;
    if (w_req > 0) W = std::min(W, w_req);
    const int wq = (int)(16 / es);  // TMA inner extent: multiple of 16 bytes
    W = std::max(wq, W / wq * wq);
    if (W * J.C > kBatchThreads || W > 256) return false;
    J.W = W;
    if (J.dir == DX) {
        // rows move as 16-byte vectors or bulk copies, in and out
        if (n % V || !al16(J.in)) return false;
        for (int k = 0; k < J.nops; ++k)
            if (!al16(J.out[k]) || !al16(J.shift_out[k])) return false;
        J.xstage = xstage ? 1 : 0;
        int pitch = J.C * L + 2 * kHalo;
        while (((size_t)pitch * es / 16) % 2 == 0) pitch += V;
        J.pitch = pitch;
        J.span = (long)J.ny * J.nz;
        J.ntiles = (J.span + W - 1) / W;
        *tile_bytes = ((size_t)W * pitch * es + 127) & ~(size_t)127;
        return true;
    }
    if (((size_t)J.nx * es) % 16) return false;
    const int nb = (n + 255) / 256;
    int box_n = (n + nb - 1) / nb;
    const int align_rows = 128 / gcd_int(128, (int)(W * es));
    box_n = (box_n + align_rows - 1) / align_rows * align_rows;
    if (box_n > 256) return false;
    J.box_n = box_n;
    J.nbox = nb;
    J.span = (J.nx + W - 1) / W;
    J.ntiles = J.span * (J.dir == DY ? J.nz : J.ny);
    // halo rows in front of the boxes: at least kHalo, keeping the boxes
    // 128-byte aligned
    J.halo = kHalo;
    while (((size_t)J.halo * W * es) % 128) ++J.halo;
    const int rows = J.halo + std::max(nb * box_n, J.C * L + kHalo);
    *tile_bytes = ((size_t)rows * W * es + 127) & ~(size_t)127;
    auto enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t gdim[3] = {(cuuint64_t)J.nx, (cuuint64_t)J.ny, (cuuint64_t)J.nz};
    cuuint64_t gstride[2] = {(cuuint64_t)J.nx * es, (cuuint64_t)J.nx * J.ny * es};
    cuuint32_t box[3] = {(cuuint32_t)W, 1, 1};
    box[J.dir == DY ? 1 : 2] = (cuuint32_t)box_n;
    cuuint32_t estr[3] = {1, 1, 1};
    return enc(&J.tmap, sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
               const_cast<T *>(J.in), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Two slots, scratch and responses, then (kBatchStaged) the x staging rows;
// without them more CTAs may fit an SM.
template <typename T>
size_t batch_smem_bytes(size_t tile_cap, int variant)
{
    return (variant & 3) == kBatchStaged ? batch_out_offset<T>(tile_cap) + tile_cap
                                         : 2 * tile_cap + batch_scratch_bytes_c<T>();
}

template <typename T>
static void (*batch_kernel(int variant))(const BatchJob<T> *, int, long, unsigned long long *, size_t, int *)
{
    const bool shift = variant & kBatchShift;
    switch (variant & 3) {
    case kBatchStaged: return shift ? ls_batch<T, kBatchStaged, true> : ls_batch<T, kBatchStaged, false>;
    case kBatchMixed: return shift ? ls_batch<T, kBatchMixed, true> : ls_batch<T, kBatchMixed, false>;
    default: return shift ? ls_batch<T, kBatchLong, true> : ls_batch<T, kBatchLong, false>;
    }
}

template <typename T>
int batch_variant(const BatchJob<T> *jobs, int njobs)
{
    int v = kBatchLong, shift = 0;
    for (int i = 0; i < njobs; ++i) {
        if (jobs[i].dir == DX && jobs[i].xstage) v = kBatchStaged;
        else if (jobs[i].L != kChunkLong<T>) v = std::max(v, (int)kBatchMixed);
        for (int k = 0; k < jobs[i].nops; ++k)
            if (jobs[i].shift_out[k]) shift = kBatchShift;
    }
    return v | shift;
}

template <typename T>
int prepare_batch(size_t tile_cap, int variant, size_t smem_optin, int num_sms, int *grid)
{
    const size_t smem = batch_smem_bytes<T>(tile_cap, variant);
    if (smem + 1024 > smem_optin) return X3D_EUNSUPPORTED;
    auto kern = batch_kernel<T>(variant);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return X3D_ECUDA;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBatchThreads, smem);
    *grid = num_sms * (per_sm < 1 ? 1 : per_sm);
    return X3D_OK;
}

template <typename T>
int launch_batch(cudaStream_t st, int grid, const BatchJob<T> *d_jobs, int njobs, long total,
                 unsigned long long *d_counter, size_t tile_cap, int variant, int *d_err)
{
    const size_t smem = batch_smem_bytes<T>(tile_cap, variant);
    if (cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st) != cudaSuccess) return X3D_ECUDA;
    batch_kernel<T>(variant)<<<(unsigned)grid, kBatchThreads, smem, st>>>(d_jobs, njobs, total, d_counter,
                                                                           tile_cap, d_err);
    return cudaGetLastError() == cudaSuccess ? X3D_OK : X3D_ECUDA;
}

template bool plan_batch_job<float>(BatchJob<float> &, int, int, int, size_t *);
template bool plan_batch_job<double>(BatchJob<double> &, int, int, int, size_t *);
template int batch_variant<float>(const BatchJob<float> *, int);
template int batch_variant<double>(const BatchJob<double> *, int);
template int prepare_batch<float>(size_t, int, size_t, int, int *);
template int prepare_batch<double>(size_t, int, size_t, int, int *);
template int launch_batch<float>(cudaStream_t, int, const BatchJob<float> *, int, long, unsigned long long *,
                                 size_t, int, int *);
template int launch_batch<double>(cudaStream_t, int, const BatchJob<double> *, int, long, unsigned long long *,
                                  size_t, int, int *);

}  // namespace x3d
