// Chunked line-solve stage kernels (linesolve_chunk.cu).
#pragma once

#include <cuda.h>

#include "x3d_internal.h"

namespace x3d {

constexpr int kMaxStageOps = 6;
constexpr int kMaxStageTiles = 3;

// One operator application inside a stage.  Its input is staged tile src_a,
// or the pointwise product of tiles src_a and src_b.  The solved values x
// update a register accumulator: acc = m x (accumulate = 0) or acc += m x,
// with m = 1 or m = tile[mul_tile] at the same point.  With flush set the
// accumulator is written out:  out = base + sign * acc  (base may be null,
// and may alias out), then optionally  out2 = base2 + scale2 * out.
template <typename T>
struct StageOp {
    LineOp<T> op;
    void *out;
    const void *base;
    void *out2;
    const void *base2;
    double sign, scale2;
    int kind;
    short src_a, src_b;
    short mul_tile;
    short accumulate;
    short flush;
    short out_f64;  // out, base, out2, base2 hold double rather than T
    // Set by launch_stage: base2 is staged input tile base2_tile (-1: read
    // from global memory); prefetch_base: base (or, without one, a base2
    // read from global memory) is prefetched into L2 when
    // the tile's inputs are requested.
    short base2_tile;
    short prefetch_base;
    // Plain programs: a second output, the solve one point further along the
    // line (shift_out[i + 1] = x[i], periodic), or null; see shifted_twin.
    void *shift_out;
    // Set by launch_stage: the response entries the fixes of a full chunk
    // use (see chunk_solve_resp).
    int keep;
    // Responses of a chunk's solved values to its carries, for the launch's
    // chunk length L (set by launch_stage): y_j = y_j(local) + F resp[0][j]
    // + B resp[1][j] for a full chunk, resp[2], resp[3] for a short last
    // chunk, F and B the forward and backward carries (see chunk_solve_resp).
    T resp[4][kChunkLong<T>];
};

// Up to six operators along one direction over up to three staged inputs of
// one (nx, ny, nz) grid: one read of each input, the writes the flushes ask for.
template <typename T>
struct StageProgram {
    StageOp<T> ops[kMaxStageOps];
    const T *in[kMaxStageTiles];
    int nops, ntiles;
    int prefetch_mask;  // bit k: operator k's base is prefetched (set by launch_stage)
    int in_f64;         // T = float: in[] hold FP64 fields (y/z plain programs only)
    int aligned_only;   // refuse extents and addresses that need linesolve_any.cu
};

inline bool al16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Number of (lines per CTA, chunk length, persistence, lines per thread)
// configurations launch_stage knows in 0 .. 15; 16 is the one-thread-per-line
// kernel (not a launch_stage configuration); 17, 18, 19 and 20 are
// configurations 6, 9, 3 and 0 compiled for three CTAs per SM (plain
// programs).
// kAllConfigs counts every configuration the
// dispatch tries.
constexpr int kChunkConfigs = 16;
constexpr int kAllConfigs = 21;
inline bool is_stage_cfg(int cfg) { return cfg >= 0 && cfg < kAllConfigs && cfg != kChunkConfigs; }

// Launches the chunked stage kernel with configuration cfg (is_stage_cfg).  Returns X3D_EUNSUPPORTED, launching nothing, when the
// shape, alignment or shared-memory budget rules that configuration out.
template <typename T>
int launch_stage(x3d_ctx_s *ctx, const StageProgram<T> &prog, int dir, int nx, int ny, int nz,
                 int cfg);

// Configurations for a program that the autotuner has not timed, best first, by
// the rule at default_cfgs (linesolve_chunk.cu).
struct DefaultCfgs {
    int count, cfg[3];
};
// es: element bytes of the context; ntiles, nops: staged inputs and operators;
// acc: the program accumulates or flushes other than plainly; in64: FP64 inputs
// of an FP32 program.
DefaultCfgs default_cfgs(size_t es, int dir, int nx, int ny, int nz, int ntiles, int nops, bool acc, bool in64,
                         int num_sms);

// The rule's last picks, by its arguments: weighing the configurations takes
// 0.2 to 0.6 us of a call's host time, a small operator's whole launch 7 (at 48 x
// 64 x 80 FP32 the rule had made it 0.3 to 0.5 us slower).  One entry a slot, the
// newest; a thread keeps its own.
struct CfgKey {
    int arg[10];
    bool operator==(const CfgKey &o) const
    {
        for (int i = 0; i < 10; ++i)
            if (arg[i] != o.arg[i]) return false;
        return true;
    }
};
template <int N>
struct CfgPicks {
    struct Slot {
        CfgKey key;
        DefaultCfgs pick;
    } slot[N] = {};  // a key of zeros is none the rule is asked for
    template <typename Rule>
    DefaultCfgs get(const CfgKey &k, const Rule &rule)
    {
        unsigned h = 0;
        for (const int a : k.arg) h = h * 31u + (unsigned)a;
        Slot &s = slot[h % N];
        if (!(s.key == k)) s = {k, rule()};
        return s.pick;
    }
};

// The pressure-to-velocity operators (derpv, interpv) take the stencil of their
// velocity-to-pressure twins one point back, r_pv[i] = r_vp[i - 1], and a
// periodic operator's matrix is circulant, so on one input the solve of pv is
// that of vp one point on: where a group applies both, one solve is written
// twice.  Whether pv is vp's shifted twin in that sense.
template <typename T>
inline bool shifted_twin(const LineOp<T> &vp, int vp_kind, const LineOp<T> &pv, int pv_kind)
{
    if (!(vp_kind == DERVP && pv_kind == DERPV) && !(vp_kind == INTVP && pv_kind == INTPV)) return false;
    return vp.circ && pv.circ && vp.n == pv.n && vp.alfa == pv.alfa && vp.a == pv.a && vp.b == pv.b && vp.c == pv.c &&
           vp.d == pv.d;
}

// Whether a program needs the kernels with the accumulator and every flush form.
template <typename T>
inline bool program_acc(const StageProgram<T> &p)
{
    for (int k = 0; k < p.nops; ++k) {
        const StageOp<T> &so = p.ops[k];
        if (!so.flush || so.accumulate || so.mul_tile >= 0 || so.base || so.out2 || so.out_f64 || so.sign != 1.0)
            return true;
    }
    return false;
}

// Lines per CTA for x lines of C chunks whose rows every warp copies in turn
// (linesolve_any.cu, linesolve_walls.cu), at most `widest`.  A tile of one or
// two chunks is one or two warps, which take 32 or 16 rows each: where few such
// warps share an SM that is the launch's time, and 8 lines a CTA (8 rows a warp,
// most of its lanes idle in the solve) are faster, up to the number of warps at
// which the idle lanes cost as much.  FP32, 17 points, one operator: 600 lines
// 10.8 us on 32 lines, 5.0 on 8; 16384 lines 11.5 and 9.2; 40000 lines (8 warps
// an SM) walls 15.3 on 32, 10.9 on 16, 13.4 on 8; 90000 lines 16.5 on 32, 18.7
// on 16.  Two chunks: FP64 17 points, 16384 lines (7 warps an SM) 9.1 and 7.6,
// 40000 lines 10.0 and 12.8; FP32 33 points, 4096 lines 7.1 and 5.6, 8000 lines
// (3.4 warps) 7.5 and 7.8.
inline int x_tile_lines(int widest, int C, long lines, int num_sms, size_t es)
{
    const int warps = (C * widest + 31) / 32, rows = widest / warps;
    const double per_sm = (double)((lines + widest - 1) / widest * warps) / num_sms;
    if (rows >= 32) return per_sm < 4.0 ? 8 : (per_sm < 16.0 ? 16 : widest);
    if (rows >= 16 && per_sm < (es == 8 ? 8.0 : 2.5)) return 8;
    return widest;
}

// The same program on a grid whose rows or addresses are not whole 16-byte
// units, W lines per CTA in chunks of kChunkLong<T> points (linesolve_any.cu);
// launch_stage's configurations 0 (W = 16) and 3 (W = 8) fall through to it.
template <typename T, int W>
int launch_stage_any(x3d_ctx_s *ctx, const StageProgram<T> &prog, bool acc, int dir, int nx, int ny, int nz);

// One job of a box batch: up to six operators applied along one direction to
// one field of one box.  Filled on the host, read by the persistent batch
// kernel from device memory (the tensor map first, for its 64-byte alignment).
constexpr int kBatchThreads = 256;

template <typename T>
struct BatchJob {
    CUtensorMap tmap;  // y/z input map
    const T *in;
    T *out[kMaxStageOps];
    T *shift_out[kMaxStageOps];  // as StageOp::shift_out
    LineOp<T> op[kMaxStageOps];
    int kind[kMaxStageOps];
    int nops, dir, n, nx, ny, nz;
    int L;       // chunk length (kChunkLong or kChunkShort of T)
    int rclass;  // jobs with equal rclass have equal responses (same operators, line length and L)
    int xstage;  // x jobs: outputs staged in shared-memory rows, bulk row copies
    int W, C, box_n, nbox, pitch;
    int halo;    // y/z: staged rows in front of the line (periodic halo + alignment)
    long span;   // x: number of lines; y/z: tiles across x
    long tile0;  // first work item of the job
    long ntiles;
    // the entries of each operator's responses the fixes use (as
    // StageOp::keep; set by plan_batch_job)
    int keep[kMaxStageOps];
    // carry responses of each operator for the job's chunk length (as
    // StageOp::resp).  Everything before them is the job's header, which the
    // kernel copies to shared memory once per work item.
    T resp[kMaxStageOps][4][kChunkLong<T>];
};

// Chooses tiling for the job (chunk length L, kChunkLong or kChunkShort of
// T; at most w_req lines per tile when w_req > 0, else as many as the
// threads allow; x outputs staged in shared memory when xstage) and encodes
// its tensor map; false when the batch kernel cannot take the job.
template <typename T>
bool plan_batch_job(BatchJob<T> &J, int L, int w_req, int xstage, size_t *tile_bytes);

// Variants of the batch kernel: every job on the long chunk with x outputs
// straight out; each job's own chunk length; and x outputs staged in shared
// memory where a job sets xstage; each with and without (kBatchShift) shifted
// second outputs, whose code costs lists that never run it 2 % (five boxes, FP32,
// three operators: 390 us, 380 without).  batch_variant picks the narrowest one
// a host job list needs.
enum BatchVariant { kBatchLong = 0, kBatchMixed = 1, kBatchStaged = 2, kBatchShift = 4 };
template <typename T>
int batch_variant(const BatchJob<T> *jobs, int njobs);

// Sets the shared-memory attribute of the batch kernel's variant for tiles
// up to tile_cap bytes and returns the persistent grid (SMs x resident CTAs
// per SM).
template <typename T>
int prepare_batch(size_t tile_cap, int variant, size_t smem_optin, int num_sms, int *grid);

// One persistent launch over every tile of every job (jobs and counter in
// device memory; the counter is reset by the launch itself, so the pair of
// operations can be captured in a CUDA graph and replayed).
template <typename T>
int launch_batch(cudaStream_t st, int grid, const BatchJob<T> *d_jobs, int njobs, long total,
                 unsigned long long *d_counter, size_t tile_cap, int variant, int *d_err);

// A plain program: operator k reads input 0 and writes out[k].
template <typename T>
StageProgram<T> plain_program(const T *in, const LineOp<T> *const *ops, const int *kinds,
                              void *const *outs, int nops);

}  // namespace x3d
