// Host-side launchers of the pipeline kernels (one launch per stage over all
// jobs of a batch).  `prefix` is the device copy of the per-job block prefix
// of that stage and `blocks` its last entry.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "qm_internal.cuh"

namespace qm
{

// throws CudaError (engine.h) on failure
void check(cudaError_t e, const char *what);

// Launches a kernel that starts with after_previous().  early: its blocks may be
// set up while the kernel before it in the stream still runs, which hides the
// launch's own latency.  For one stream's work or one keyframe's: with several
// streams on the GPU the waiting blocks only take the others' place.  Measured,
// late -> early: BP of one 640x480 x 48 keyframe (20 launches then) 160 -> 128 us, a
// fitting step at 160x128 848 -> 765, a 160x128 stream (in its graph) 194 -> 190;
// 32 x 752x480 (submit + wait) 3.19 -> 3.47 ms, so not there.  Several handles of one
// stream each on threads are not told apart from one: a frame at 160x128 with 2 / 4 /
// 8 of them 107 / 77 / 66 us late and 103 / 73 / 66 early, at 752x480 415 / 309 / 362
// and 406 / 298 / 388 (runs of one kind differ by up to 15 %).
template <class... P, class... A>
void launch_kernel(void (*k)(P...), int blocks, int threads, size_t smem, cudaStream_t s,
                   int early, A &&...args)
{
  cudaLaunchConfig_t c = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.gridDim = dim3(blocks);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = early ? 1 : 0;
  check(cudaLaunchKernelEx(&c, k, std::forward<A>(args)...), "kernel launch");
}

// threads per block of the flat per-element kernels
constexpr int kFlatThreads = 256;
// warps per block of the warp-per-cell kernels (BP sweep, extraction): the
// default and the largest the kernels are compiled for (the autotuner picks
// among 4, 8 and 16)
constexpr int kCellWarps = 8;
constexpr int kMaxCellWarps = 16;
// line solvers: one warp per line; rows per block of the row pass and
// columns per block (stripe width) of the column pass: defaults and maxima
constexpr int kRowWarps = 2;
constexpr int kColLines = 4;
constexpr int kMaxRowWarps = 4;
constexpr int kMaxColLines = 8;
// cost kernel: resident blocks of 256 threads per SM it is compiled for
constexpr int kCostBlocks = 4;
// longest lines the solvers' shared memory holds
constexpr int kMaxRowLen = 4096;
constexpr int kMaxColLen = 2048;
size_t row_solve_smem(int max_w, int rows = kRowWarps);
size_t col_solve_smem(int max_h, int lines = kColLines);

// shared memory one block may take
constexpr int kMaxBlockSmem = 227 * 1024;

// Launch shapes of one active job set (chosen by the engine's autotuner).
struct Tune
{
  int sweep_warps = kCellWarps;   // warps per block of the BP half-sweeps
  int extract_warps = kCellWarps; // warps per block of the extraction
  int row_warps = kRowWarps;      // rows per block of the row solve
  int col_lines = kColLines;      // columns per block of the column solve
  int cost_blocks = kCostBlocks;  // resident cost-kernel blocks per SM (3, 4 or 5)
};
void prepare_upsample_kernels();

// blocks of the quadtree launch for one W x H image
int quadtree_blocks(int W, int H, int qt_max);

// Every launcher takes the batch by value (the kernels receive it as a
// __grid_constant__ parameter); B.prefix must point at the stage's prefix.
void launch_quadtree(const Batch &B, int blocks, KParams kp, cudaStream_t s);
// cells per block of the cost kernel (one tile of a cell row)
constexpr int kCostCells = 32;
constexpr int kMaxHyp = 128;
int cost_tiles(int cw, int ch);
// blocks per tile when the launch's jobs have `tiles` tiles in all
int cost_split(long tiles);
// max_d: largest hypothesis count of the batch (sizes the shared tile); split:
// blocks per tile (1, 2 or 4); blocks_per_sm: 3, 4 or 5, the instance's
// register budget
// view: the blocks first find the hypotheses at which a slot cannot be in view
void launch_cost(const Batch &B, int blocks, int arith, int max_d, int split, bool view,
                 cudaStream_t s, int blocks_per_sm = kCostBlocks);
// Hypotheses x slots of a block from which that pays: it takes a block about a
// microsecond, and of few slots, whose frames are near, little is out of view.
// Measured, without -> with: 1920x1080 x 128 hypotheses, 20 slots 794 -> 733 us,
// eight of them 4.33 -> 3.83 ms; 2560x1440 x 128, 10 slots 628 -> 615, 1280x720
// x 128, 10 slots 263 -> 260; 752x480 x 64, 10 slots 92 -> 94, 5 slots 62.8 ->
// 65.5.
constexpr int kViewWork = 1024;
// Data terms of the levels `level` .. level + n - 1 (n <= kPyramidLevels) from
// level - 1; pyramid_blocks of level `level`'s size
constexpr int kPyramidLevels = 3;
int pyramid_blocks(int w, int h);
void launch_pyramid(const Batch &B, int blocks, int level, int n, cudaStream_t s);
// writes the inherited messages of level `level` that its sweeps will read
// (cells the quadtree test skips; all unswept cells when iters < 2)
void launch_msg_inherit(const Batch &B, int blocks, int level, int iters, int qt_max,
                        cudaStream_t s);
// half-sweep `it` (0-based) of level `level`; `warps` per block.  inherit:
// half-sweeps 0 and 1 also write the inherited messages of their colour's
// cells the quadtree test skips (instead of launch_msg_inherit; the level
// must have at least two half-sweeps)
void launch_bp_sweep(const Batch &B, int blocks, int d, int level, int it, KParams kp, int arith,
                     cudaStream_t s, int warps = kCellWarps, int inherit = 0);
// Message states a level keeps for the adjoint of the soft BP.  Half-sweeps
// it = iters - 1 and iters - 2 write the level's own message images (together
// every cell), the two before them the first kept state, and so on: half-sweep
// it + 1 and its adjoint only read the colour that half-sweep it wrote.
struct HistLevel
{
  float *base;      // kept states, 4 images each (null: none)
  size_t dir, slot; // floats between the images of a state and between states
  // image `m` of the state half-sweep `it` writes; own: the level's image
  __host__ __device__ float *at(int it, int iters, int m, float *own) const
  {
    const int k = (iters - 1 - it) >> 1;
    return k <= 0 ? own : base + (size_t)(k - 1) * slot + (size_t)m * dir;
  }
  __host__ __device__ static int states(int iters) { return iters > 2 ? (iters - 1) / 2 : 0; }
};
// message images a half-sweep reads and writes, by direction
struct SweepIO
{
  const float *in[4];
  float *out[4];
};
// half-sweep `it` of the inline job's level from io.in (it = 0: the parents'
// messages) into io.out, skipped cells included
void launch_bp_sweep_io(const Batch &B, int d, int level, int it, const SweepIO &io, KParams kp,
                        int arith, cudaStream_t s);
// Top BP levels in one launch (k_bp_coarse): levels hi down to lo, every one
// with at least two half-sweeps, a cluster of `ctas` blocks per job keeping a
// level in shared memory, `per` cells per block.
constexpr int kCoarseMaxThreads = 1024;
constexpr int kCoarseMaxCtas = 16; // above the portable 8: asked of the device
constexpr int kCoarseAuto = -1; // max_cells of coarse_plan: by the half-sweeps' rounds
struct CoarsePlan
{
  int lo, hi;
  int iters[kMaxLevels];
  int ctas, per, threads;
  int data_smem; // 1: the data term in shared memory too
  int keep;      // 1: the half-sweeps keep their states in hist
  HistLevel hist[kMaxLevels];
};
// Sizes the plan for jobs of d hypotheses, `jobs` jobs of any count and of all
// branches running at once: the top levels with at most max_cells cells in every
// job (cells[l]: the most), two half-sweeps or more, and room in a cluster's shared
// memory.  False: no such level.  plan.keep is read, the rest (but hist) written.
// kCoarseAuto takes the levels of whose cells a colour is one round of a full
// cluster's lane groups, or two where a few streams run: above that a half-sweep in
// the cluster takes longer than a launch over the whole GPU.  Measured (resident
// pass, with the level in the cluster / launched, cells x lanes per cell in
// brackets): one stream 320x240 x 64 (19200) 145 / 152 us, 752x480 x 64 (22560) 210 /
// 212, 320x240 x 96 (38400) 175 / 164, 752x480 x 96 (45120) 256 / 236, 1280x720 x 64
// (57600) 306 / 282; four (their launches are not early) 480x320 x 64 (38400) 233 /
// 239, 1280x720 x 64 (57600) 654 / 675, 320x240 x 64 (76800) 187 / 169; 24 in
// clusters of 8: 752x480 x 64 (22560) 1530 / 1539, 160x128 x 128 (40960) 302 / 241.
bool coarse_plan(CoarsePlan &plan, int d, const long *cells, int levels, const int *iters,
                 long max_cells, int jobs, int arith);
// jobs j0 .. j0 + jobs - 1 of the batch (B.jobs null: the inline job)
void launch_bp_coarse(const Batch &B, int j0, int jobs, int d, const CoarsePlan &plan,
                      KParams kp, int arith, cudaStream_t s);
void launch_extract(const Batch &B, int blocks, int d, int arith, cudaStream_t s,
                    int warps = kCellWarps);
void launch_row_solve(const Batch &B, int blocks, KParams kp, int arith, int max_w,
                      cudaStream_t s, int rows = kRowWarps);
void launch_col_solve(const Batch &B, int blocks, KParams kp, int arith, int max_h,
                      cudaStream_t s, int lines = kColLines);
// Pixels per thread of the fusion update (it walks them as a pipeline) and of
// the transform (1 or 4) when the launch's jobs have `pixels` pixels in all
int fuse_px(long pixels);
int fuse_transform_px(long pixels);
void launch_fuse_transform(const Batch &B, int blocks, int px, int arith, cudaStream_t s);
// hole filling + posterior update (reads the z-buffer keys, leaves them set:
// the next frame's row solve resets them)
void launch_fuse_update(const Batch &B, int blocks, int px, cudaStream_t s);
// out[i] = seeds[i].w (the fused variance sigma^2), n pixels
void launch_seed_variance(const float4 *seeds, float *out, long n, cudaStream_t s);

// Point cloud of one depth map (k_points.cu): out receives (x, y, z,
// intensity) per kept pixel in row-major order, *count (device) their number;
// ws holds point_cloud_workspace(W, H) bytes.
int point_cloud_tiles(int W, int H);
size_t point_cloud_workspace(int W, int H);
void launch_point_cloud(const float *depth, size_t stride, const uint8_t *ref, size_t pitch, int W,
                        int H, const Cam &cam, const float *T_world_ref, float4 *out, int *count,
                        void *ws, cudaStream_t s);

// ---------------------------------------------------------------------------
// Differentiable path (k_diff.cu).

// One BP level of one keyframe for the soft readout and the BP adjoint, with
// messages, adjoints and data terms of real type R: float for the
// differentiable product path, double for the gradient-check mode.
template <class R>
struct DiffBpR
{
  int W, H, D;           // image and hypotheses
  int w, h;              // cells of this level
  int level, parity, qt_max;
  int first;             // half-sweep 0: S holds the parents' messages, pw wide
                         // (null at the coarsest level: zeros)
  int last;              // the level's last half-sweep (adjoint: the first)
  int iters, pw;
  const uint8_t *levels; // quadtree level map
  const R *data;         // data term of this level
  const R *S[4];         // messages read (a kept state, or the finals)
  R *A[4];               // adjoint of the messages, by direction
  float P1, P2;
  double *gP;            // dL/dP1, dL/dP2 (accumulated)
  float tau;             // readout temperature
  double step, min_inv;  // hypothesis depths
  float *sparse;         // readout output (W x H)
  const float *g_sparse; // its adjoint
};
using DiffBp = DiffBpR<float>;
using DiffBp64 = DiffBpR<double>;
template <class R>
struct MsgPtrsR
{
  R *m[4];
};
using MsgPtrs = MsgPtrsR<float>;
using MsgPtrs64 = MsgPtrsR<double>;
// soft readout at level-0 node cells: forward writes sparse; backward writes
// every value of A, the belief adjoint at the four incoming messages of every
// node cell and 0 elsewhere
void launch_soft_readout(const DiffBp &a, int backward, cudaStream_t s);
void launch_soft_readout(const DiffBp64 &a, int backward, cudaStream_t s);
// adjoint of one half-sweep of colour a.parity: consumes A at the updated
// cells and writes the adjoints of the messages they read (a.S, the state the
// forward half-sweep read).  Values of A it has consumed are left stale; they
// are rewritten before they are read again, and launch_msg_downsample skips
// those of the colour of half-sweep 0.
void launch_bp_sweep_bwd(const DiffBp &a, cudaStream_t s);
void launch_bp_sweep_bwd(const DiffBp64 &a, cudaStream_t s);
// parent.m[k] = sum of the (up to four) children's adjoints a.A[k] of the
// starting messages of level a (pw x ph parents)
void launch_msg_downsample(const DiffBp &a, const MsgPtrs &parent, int pw, int ph,
                           cudaStream_t s);
void launch_msg_downsample(const DiffBp64 &a, const MsgPtrs64 &parent, int pw, int ph,
                           cudaStream_t s);
// FP64 BP forward of the gradient-check mode (the product's BP is FP32):
// out[i] = in[i] widened; the pyramid of data terms (children summed x
// offset outer, y offset inner); every cell of a level starting from its
// parent's messages (zeros when parent is null), as the reference's
// copy-down; one half-sweep of colour a.parity updating M in place (a.S
// unused)
void launch_widen(const float *in, double *out, long n, cudaStream_t s);
void launch_pyramid64(const double *fine, int fw, int fh, double *coarse, int cw, int ch, int D,
                      cudaStream_t s);
void launch_msg_inherit_all64(const MsgPtrs64 *parent, int pw, const MsgPtrs64 &child, int cw,
                              int ch, int D, cudaStream_t s);
void launch_bp_sweep_fwd64(const DiffBp64 &a, const MsgPtrs64 &M, cudaStream_t s);

// Weighted upsampling of one image (FP64 line solves).
struct DiffUp
{
  int W, H;
  const uint8_t *img;
  size_t pitch;
  const float *omega;     // W x H edge-weight factors
  double lam, sigma, row_closing, col_closing;
  const float *sparse;    // input
  float *dense;           // output
  double *sd, *si;        // row-pass results (depth, indicator)
  double *td, *ti;        // column-pass results
  double *cp;             // Thomas scratch
  double *ud, *ui;        // adjoint scratch
  const float *g_dense;   // incoming adjoint
  float *g_sparse, *g_omega;
};
void launch_upw_forward(const DiffUp &u, cudaStream_t s);
void launch_upw_backward(const DiffUp &u, cudaStream_t s);

struct DiffFuse
{
  int W, H;
  const float *depth_in;  // upsampled depth before fusion
  const float4 *seeds_in; // the transformed previous seeds
  const int32_t *table;   // source seed per pixel (0 = none)
  const float *g_fused;
  float *g_depth;
};
void launch_fuse_bwd(const DiffFuse &f, cudaStream_t s);

// supported hypothesis-count classes of the BP kernels
bool bp_supported_d(int d);
// cells one warp of the BP sweep / extraction handles for d hypotheses
int bp_cells_per_warp(int d);

} // namespace qm
