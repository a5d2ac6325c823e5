// Hierarchical min-sum belief propagation and depth extraction
// (bp_extract and its kernels, bpextract.cu:37-395 of the reference).
//
// Layout: per pyramid level, the data cost and the four outgoing-message
// images are [h][w][D] float arrays (hypotheses contiguous, the PIXEL_COST
// layout).  A half-sweep updates the cells of one checkerboard colour in
// place; they only read messages of the other colour, so the update is a
// Jacobi step inside the colour, exactly as the reference's launch.
//
// Lane groups: a cell is handled by a group of LPC lanes (32 for 96 and 128
// hypotheses, 16 for 48 and 64, 8 for 32), so a warp updates 32/LPC cells at
// once; a lane holds four consecutive hypotheses (QuadLayout).  The four
// directions are computed from one load of the data cost and the four incoming
// messages.  The normalising sum uses the reference's stride-halving tree
// (bpextract.cu:293-300) over the next power of two P >= D with zero padding.
// The argmin of the extraction uses the same tree with the reference's tie
// rule (the right element wins only when strictly smaller,
// bpextract.cu:347-355).
//
// Bytes per updated cell and half-sweep: 9*D*4 (data + 4 messages read, 4
// messages written).
#include <atomic>
#include <cfloat>
#include <type_traits>

#include "launch.h"

namespace qm
{

namespace
{

constexpr __host__ __device__ int pow2_ceil(int n)
{
  int p = 1;
  while (p < n)
    p <<= 1;
  return p;
}

// Lane g of a cell's group holds the four consecutive hypotheses 4 g .. 4 g + 3
// (one 16-byte access per image; d +- 1 needs two shuffles per direction).  At
// 48 and 96 hypotheses the last quarter of a group's lanes holds padding.
template <int D>
struct QuadLayout
{
  static constexpr int P = pow2_ceil(D); // tree width
  static constexpr int LPC = P / 4;      // lanes per cell
  static constexpr int ACT = D / 4;      // lanes with hypotheses
  static constexpr int G = 32 / LPC;     // cells per warp
  static_assert(D % 4 == 0 && LPC <= 32, "a cell's hypotheses fill lanes of one warp");
};

// sum / (float)DEPTH_NUM (bpextract.cu:302); D is a compile-time constant
// here as DEPTH_NUM is in the reference.
template <int D, int ARITH>
__device__ __forceinline__ float mean_of(float sum)
{
  if (ARITH == QM_ARITH_IEEE)
    return __fdiv_rn(sum, (float)D);
  return sum / (float)D;
}

// The kernels below move whole float4 groups of hypotheses (D is a
// multiple of 16 for every supported count, and every cell row starts on a
// 16-byte boundary); each component keeps its own arithmetic.

// ------------------------------------------------------------- pyramid
// cost_distribute (bpextract.cu:169-198): L_l(x,y) = sum of the existing 2x2
// children, x offset outer, y offset inner, starting from 0; levels `level` ..
// level + n - 1 from level - 1.  A block makes a tile of 4 x 4 cells of the
// first, 2 x 2 of the second and one of the third from 8 x 8 finer cells; the
// levels it has just made are read from shared memory.  A cell that a level
// does not have adds 0 there, which changes no sum.
// Bound: launches where few streams run (a launch per level took three where one
// does: 640x480 x 48 BP alone 126 -> 122 us, one 160x128 keyframe 189 -> 184 us),
// DRAM where many do: 32 x 752x480 x 64 75 us, where a kernel per level took 64 in
// three launches and the gaps between them (this one launched level by level: the
// pass 2.38 ms instead of 2.35).
__global__ void __launch_bounds__(kFlatThreads)
    k_pyramid(const __grid_constant__ Batch B, int level, int n)
{
  after_previous();
  int lb;
  const JobDesc &J = job_of(B, lb);
  const int D4 = J.D / 4, tid = threadIdx.x;
  __shared__ float4 s_a[16 * (kMaxHyp / 4)], s_b[4 * (kMaxHyp / 4)];
  const int tiles = (J.lv[level].w + 3) / 4;
  const int ty = lb / tiles, tx = lb - ty * tiles;
  // cells [4 tx, 4 tx + side) x [4 ty, ..) of a level: v(x, y, q) sums the children
  auto make = [&](const LevelDesc &L, int side, float4 *keep, auto &&child) {
    for (int k = tid; k < side * side * D4; k += kFlatThreads)
    {
      const int c = k / D4, q = k - c * D4, lx = c % side, ly = c / side;
      const int x = tx * side + lx, y = ty * side + ly;
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (x < L.w && y < L.h)
      {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int jj = 0; jj < 2; ++jj)
          {
            const float4 v = child(x, y, lx, ly, i, jj, q);
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
          }
        reinterpret_cast<float4 *>(L.data)[((size_t)y * L.w + x) * D4 + q] = s;
      }
      if (keep)
        keep[k] = s;
    }
  };
  const LevelDesc &F = J.lv[level - 1];
  make(J.lv[level], 4, s_a, [&](int x, int y, int, int, int i, int jj, int q) {
    const int fx = 2 * x + i, fy = 2 * y + jj;
    return fx < F.w && fy < F.h
               ? reinterpret_cast<const float4 *>(F.data)[((size_t)fy * F.w + fx) * D4 + q]
               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  });
  if (n < 2)
    return;
  __syncthreads();
  make(J.lv[level + 1], 2, s_b, [&](int, int, int lx, int ly, int i, int jj, int q) {
    return s_a[((2 * ly + jj) * 4 + 2 * lx + i) * D4 + q];
  });
  if (n < 3)
    return;
  __syncthreads();
  make(J.lv[level + 2], 1, nullptr, [&](int, int, int, int, int i, int jj, int q) {
    return s_b[(jj * 2 + i) * D4 + q];
  });
}

// The reference's quadtree test of the bp kernel (bpextract.cu:214-220): a
// cell of level l is left alone by every sweep of that level when the
// quadtree level at the sample pixel of its pre-checkerboard column (x / 2)
// exceeds l + 2.
__device__ __forceinline__ bool bp_skipped(const JobDesc &J, int level, int x, int y, int qt_max)
{
  const int ilev = level + 2;
  if (ilev > qt_max)
    return false;
  const int size = 1 << ilev;
  const int sx = min((x >> 1) * size, J.W - 1), sy = min(y * size, J.H - 1);
  return (int)J.levels[(size_t)sy * J.W + sx] > ilev;
}

// Message inheritance.  The reference starts every level from a copy of the
// parent messages (upsample, bpextract.cu:374-395), or from zeros at the
// coarsest level (bpextract.cu:87-90), and then sweeps.  Most of those copies
// are never read: the first half-sweep reads the parents directly (the sweep
// kernel's `first` mode), and every cell the sweeps update overwrites its
// copy before anyone reads it.  The copies that ARE read later are written
// here: cells the quadtree test skips at this level, and, with fewer than two
// iterations, the cells no sweep reaches.  With two or more iterations the
// batched pipeline does not launch this pass: half-sweeps 0 and 1 copy the
// skipped cells of their own colour (the sweep kernel's `inherit` mode).
__global__ void __launch_bounds__(kFlatThreads)
    k_msg_inherit(const __grid_constant__ Batch B, int level, int iters, int qt_max)
{
  after_previous();
  int lb;
  const JobDesc &J = job_of(B, lb);
  const LevelDesc &F = J.lv[level];
  const int D4 = J.D / 4;
  const long t = (long)lb * blockDim.x + threadIdx.x;
  if (t >= (long)F.w * F.h * D4)
    return;
  const int cell = (int)(t / D4);
  const int q = (int)(t - (long)cell * D4);
  const int x = cell % F.w, y = cell / F.w;
  // iteration i updates the cells with x + y + i even
  const bool needed = iters <= 0 || (iters == 1 && ((x + y) & 1)) ||
                      bp_skipped(J, level, x, y, qt_max);
  if (!needed)
    return;
  if (level + 1 < J.nlev)
  {
    const LevelDesc &C = J.lv[level + 1];
    const size_t src = ((size_t)(y >> 1) * C.w + (x >> 1)) * D4 + q;
#pragma unroll
    for (int m = 0; m < 4; ++m)
      reinterpret_cast<float4 *>(F.msg[m])[t] = reinterpret_cast<const float4 *>(C.msg[m])[src];
  }
  else
  {
#pragma unroll
    for (int m = 0; m < 4; ++m)
      reinterpret_cast<float4 *>(F.msg[m])[t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// ------------------------------------------------------------- sweep
// bp kernel (bpextract.cu:200-312), one lane group per cell of the active
// colour.  Groups whose cell is skipped or out of range still take part in
// the warp's shuffles (full masks) with zero inputs and store nothing.
__device__ __forceinline__ float4 msg_load(const float *p)
{
  return *reinterpret_cast<const float4 *>(p);
}

// One reduction step across lanes gl and gl ^ o that also halves the values a
// lane holds: lanes with bit o clear go on with lo, the others with hi.
template <int N, class Op>
__device__ __forceinline__ void halve(float (&lo)[N], const float (&hi)[N], bool up, int o, Op op)
{
#pragma unroll
  for (int i = 0; i < N; ++i)
  {
    const float send = up ? lo[i] : hi[i], keep = up ? hi[i] : lo[i];
    lo[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, o));
  }
}

// v[dir] of the group from the lane that holds direction dir's result: the
// directions are split over the two top bits of the lane's index in its group
template <int LPC>
__device__ __forceinline__ float from_dir(float r, int dir)
{
  return __shfl_sync(0xffffffffu, r, (dir >> 1) * (LPC / 2) + (dir & 1) * (LPC / 4), LPC);
}

// The group's minimum of v[dir] for the direction this lane holds.
template <int LPC>
__device__ __forceinline__ float dir_min(const float (&v)[4], int gl)
{
  auto mn = [](float a, float b) { return fminf(a, b); };
  float a[2] = {v[0], v[1]}, b[2] = {v[2], v[3]};
  halve(a, b, (gl & (LPC / 2)) != 0, LPC / 2, mn);
  float c[1] = {a[0]}, d[1] = {a[1]};
  halve(c, d, (gl & (LPC / 4)) != 0, LPC / 4, mn);
  float r = c[0];
#pragma unroll
  for (int o = LPC / 8; o > 0; o >>= 1)
    r = fminf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

// The reference's stride-halving tree sum (bpextract.cu:293-300) of
// m[dir][j] = value(4 g + j) over the group, for the direction this lane
// holds.  Strides of four and more pair lanes: every step adds exactly the
// tree's pairs (addition commutes bit for bit) while the lanes share out the
// directions, then the four j; strides 2 and 1 pair the lanes that hold j and
// j ^ 2, j ^ 1.  Padding is zero.
template <int LPC>
__device__ __forceinline__ float dir_tree_sum(const float (&m)[4][4], int gl)
{
  auto add = [](float a, float b) { return a + b; };
  float a[8], b[8];
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    a[j] = m[0][j], a[4 + j] = m[1][j];
    b[j] = m[2][j], b[4 + j] = m[3][j];
  }
  halve(a, b, (gl & (LPC / 2)) != 0, LPC / 2, add);
  float c[4] = {a[0], a[1], a[2], a[3]}, d[4] = {a[4], a[5], a[6], a[7]};
  halve(c, d, (gl & (LPC / 4)) != 0, LPC / 4, add);
  constexpr int o2 = LPC / 8, o1 = LPC / 16; // lane bits that share out j
  float e[2] = {c[0], c[1]}, f[2] = {c[2], c[3]};
  halve(e, f, (gl & o2) != 0, o2, add);
  if constexpr (o1 == 0)
  {
    // eight lanes: the pair (j, j ^ 2) is in lanes gl, gl ^ 1, j and j ^ 1 here
    const float s0 = e[0] + __shfl_xor_sync(0xffffffffu, e[0], o2);
    const float s1 = e[1] + __shfl_xor_sync(0xffffffffu, e[1], o2);
    return s0 + s1;
  }
  else
  {
    float r[1] = {e[0]}, q[1] = {e[1]};
    halve(r, q, (gl & o1) != 0, o1, add);
    float s = r[0];
#pragma unroll
    for (int o = o1 / 2; o > 0; o >>= 1)
      s += __shfl_xor_sync(0xffffffffu, s, o);
    s += __shfl_xor_sync(0xffffffffu, s, o2);
    s += __shfl_xor_sync(0xffffffffu, s, o1);
    return s;
  }
}

// The update of one cell (bp, bpextract.cu:200-312) from its data term and
// its four incoming messages (zeros where the level ends: the reference leaves
// those terms out, and adding 0 changes no value), every lane of the warp
// taking part (groups without a cell pass zeros): for each outgoing direction,
// emit(dir, v) receives the lane's four values of the message.
// Padding lanes (gl >= ACT) pass anything.
template <int D, int ARITH, class Emit>
__device__ __forceinline__ void cell_update(const float4 &dat, const float4 &fu, const float4 &fd,
                                            const float4 &fl, const float4 &fr, const KParams &kp,
                                            int gl, Emit &&emit)
{
  constexpr int LPC = QuadLayout<D>::LPC, ACT = QuadLayout<D>::ACT;
  const bool pad = ACT < LPC && gl >= ACT;
  const float da[4] = {dat.x, dat.y, dat.z, dat.w}, ua[4] = {fu.x, fu.y, fu.z, fu.w};
  const float ba[4] = {fd.x, fd.y, fd.z, fd.w}, la[4] = {fl.x, fl.y, fl.z, fl.w};
  const float ra[4] = {fr.x, fr.y, fr.z, fr.w};
  // h of every direction: the data term plus the three other incoming
  // messages, in the reference's order (up, down, left, right, the
  // direction's own left out)
  float h[4][4], low[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    const float du = da[j] + ua[j], dud = du + ba[j];
    h[kUp][j] = ((da[j] + ba[j]) + la[j]) + ra[j];
    h[kDown][j] = (du + la[j]) + ra[j];
    h[kLeft][j] = dud + ra[j];
    h[kRight][j] = dud + la[j];
  }
#pragma unroll
  for (int dir = 0; dir < 4; ++dir)
  {
    low[dir] = fminf(fminf(h[dir][0], h[dir][1]), fminf(h[dir][2], h[dir][3]));
    if (pad)
      low[dir] = FLT_MAX;
  }
  // a cell without a finite value counts as FLT_MAX (infinite costs then give
  // the same messages at every count, with padding lanes or without)
  const float cap = fminf(dir_min<LPC>(low, gl), FLT_MAX) + kp.P2;
#pragma unroll
  for (int dir = 0; dir < 4; ++dir)
  {
    // the minimum over h(d), h(d - 1) + P1, h(d + 1) + P1, min h + P2
    const float c = from_dir<LPC>(cap, dir);
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      s[j] = h[dir][j] + kp.P1;
    float prev = __shfl_up_sync(0xffffffffu, s[3], 1, LPC);
    float next = __shfl_down_sync(0xffffffffu, s[0], 1, LPC);
    if (gl == 0)
      prev = c;
    if (gl >= ACT - 1)
      next = c;
    h[dir][0] = fminf(fminf(h[dir][0], prev), fminf(s[1], c));
    h[dir][1] = fminf(fminf(h[dir][1], s[0]), fminf(s[2], c));
    h[dir][2] = fminf(fminf(h[dir][2], s[1]), fminf(s[3], c));
    h[dir][3] = fminf(fminf(h[dir][3], s[2]), fminf(next, c));
    if (pad)
      h[dir][0] = h[dir][1] = h[dir][2] = h[dir][3] = 0.0f;
  }
  // in reference arithmetic the division by the constant count is left beside
  // the subtraction, where the compiler may fuse the two (as it does in
  // m - sum / DEPTH_NUM of one thread); IEEE divides once per direction
  constexpr bool kIeee = ARITH == QM_ARITH_IEEE;
  const float sum = dir_tree_sum<LPC>(h, gl);
  const float mean = kIeee ? mean_of<D, ARITH>(sum) : sum;
#pragma unroll
  for (int dir = 0; dir < 4; ++dir)
  {
    const float got = from_dir<LPC>(mean, dir);
    const float mu = kIeee ? got : mean_of<D, ARITH>(got);
    emit(dir, make_float4(h[dir][0] - mu, h[dir][1] - mu, h[dir][2] - mu, h[dir][3] - mu));
  }
}

// One warp's lane groups of half-sweep `parity` at `level`: items item0 ..
// item0 + G - 1 of the colour's cells (item = y * ceil(w / 2) + x / 2).  The
// neighbours' messages come from the images in[4], the cells' own go to
// out[4], by direction (both the level's own ones, except where the soft BP
// keeps the states between half-sweeps).
template <int D, int ARITH, class In, class Out>
__device__ __forceinline__ void sweep_warp(const JobDesc &J, int level, int parity, int first,
                                           int inherit, const KParams &kp, int item0, const In &in,
                                           const Out &out_img)
{
  using QL = QuadLayout<D>;
  constexpr int LPC = QL::LPC;
  const LevelDesc &L = J.lv[level];
  const int w = L.w, h = L.h, hw = (w + 1) / 2;
  const int lane = threadIdx.x & 31, gl = lane & (LPC - 1);
  const bool lane_on = QL::ACT == LPC || gl < QL::ACT;
  const int item = item0 + lane / LPC;
  int x = 0, y = 0;
  bool act = item < hw * h, skipped = false;
  if (act)
  {
    y = item / hw;
    x = 2 * (item - y * hw) + ((y + parity) & 1); // item - y*hw == x / 2
    skipped = x < w && bp_skipped(J, level, x, y, kp.qt_max);
    act = x < w && !skipped;
  }
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (inherit && skipped && lane_on)
  {
    // message inheritance of a cell the quadtree test skips at this level:
    // its messages keep the parent's (zeros at the coarsest level), as the
    // reference's copied-down images hold them (bpextract.cu:87-90,374-395);
    // half-sweeps 0 and 1 write them for their colour before any later
    // half-sweep reads them
    const size_t c = ((size_t)y * w + x) * D + 4 * gl;
    const bool top = level + 1 >= J.nlev;
    const LevelDesc &C = J.lv[top ? level : level + 1];
    const size_t pc = ((size_t)(y >> 1) * C.w + (x >> 1)) * D + 4 * gl;
#pragma unroll
    for (int m = 0; m < 4; ++m)
      *reinterpret_cast<float4 *>(out_img[m] + c) =
          top ? zero : msg_load(C.msg[m] + pc);
  }
  if (!__any_sync(0xffffffffu, act))
    return;
  const bool on = act && lane_on;
  const bool has_u = on && y > 0, has_d = on && y < h - 1;
  const bool has_l = on && x > 0, has_r = on && x < w - 1;
  const size_t c = ((size_t)y * w + x) * D + 4 * gl;

  // Incoming messages: the neighbours' own ones, or in the first half-sweep
  // of a level the ones their parents ended with (0 at the coarsest level),
  // which is what the reference's copied-down messages hold at that point.
  const float *src_u = nullptr, *src_d = nullptr, *src_l = nullptr, *src_r = nullptr;
  if (!first)
  {
    src_u = in[kDown] + (c - (size_t)w * D);
    src_d = in[kUp] + (c + (size_t)w * D);
    src_l = in[kRight] + (c - D);
    src_r = in[kLeft] + (c + D);
  }
  else if (level + 1 < J.nlev)
  {
    const LevelDesc &C = J.lv[level + 1];
    auto parent = [&](int xn, int yn) {
      return ((size_t)(yn >> 1) * C.w + (xn >> 1)) * D + 4 * gl;
    };
    src_u = C.msg[kDown] + parent(x, y - 1);
    src_d = C.msg[kUp] + parent(x, y + 1);
    src_l = C.msg[kRight] + parent(x - 1, y);
    src_r = C.msg[kLeft] + parent(x + 1, y);
  }
  const bool ld = src_u != nullptr;
  const float4 dat = on ? *reinterpret_cast<const float4 *>(L.data + c) : zero;
  const float4 fu = (ld && has_u) ? msg_load(src_u) : zero;
  const float4 fd = (ld && has_d) ? msg_load(src_d) : zero;
  const float4 fl = (ld && has_l) ? msg_load(src_l) : zero;
  const float4 fr = (ld && has_r) ? msg_load(src_r) : zero;
  cell_update<D, ARITH>(dat, fu, fd, fl, fr, kp, gl, [&](int dir, const float4 &v) {
    if (on)
      *reinterpret_cast<float4 *>(out_img[dir] + c) = v;
  });
}

template <int D, int ARITH>
__global__ void __launch_bounds__(kMaxCellWarps * 32, 4)
    k_bp_sweep(const __grid_constant__ Batch B, int level, int parity, int first, int inherit,
               KParams kp)
{
  after_previous();
  constexpr int G = QuadLayout<D>::G;
  int lb;
  const JobDesc &J = job_of(B, lb);
  if (J.D != D)
    return;
  const LevelDesc &L = J.lv[level];
  const int hw = (L.w + 1) / 2;
  const int item0 = (lb * (int)(blockDim.x >> 5) + (threadIdx.x >> 5)) * G;
  if (item0 >= hw * L.h)
    return; // the whole warp
  sweep_warp<D, ARITH>(J, level, parity, first, inherit, kp, item0, L.msg, L.msg);
}

// Half-sweep `parity` from the message images io.in into io.out (the soft BP,
// which keeps the states its adjoint reads): every cell of the colour is
// written, those the quadtree test skips with their parents' messages.
template <int D, int ARITH>
__global__ void __launch_bounds__(kMaxCellWarps * 32, 4)
    k_bp_sweep_io(const __grid_constant__ Batch B, int level, int parity, int first,
                  const __grid_constant__ SweepIO io, KParams kp)
{
  after_previous();
  constexpr int G = QuadLayout<D>::G;
  const LevelDesc &L = B.one.lv[level];
  const int item0 = ((int)blockIdx.x * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * G;
  if (item0 >= (L.w + 1) / 2 * L.h)
    return; // the whole warp
  sweep_warp<D, ARITH>(B.one, level, parity, first, 1, kp, item0, io.in, io.out);
}

// Every half-sweep of the top levels lo..hi (coarse to fine) in one launch: a
// cluster of plan.ctas blocks per job keeps a level in its shared memory.
//
// Bound: the latency of a half-sweep (a level has a few hundred to a few
// thousand cells).  A launch per half-sweep costs 4 to 5 us, and so did
// half-sweeps of one cluster launch that handed the messages on through L2;
// here a half-sweep is shared-memory reads, the update and one hardware cluster
// barrier (release / acquire, nothing spins).
//
// Layout: block r owns the cells [r per, (r + 1) per) of the level in row-major
// order, with their edges to the right and to the lower neighbour.  An edge
// holds ONE message, the one that will be read next: a half-sweep's cells all
// have one colour, each reads its four edges and overwrites them with what it
// sends, which the other colour reads in the next half-sweep.  That is 2 D
// values per cell instead of 4 D, so 16 blocks hold about 7000 cells of 64
// hypotheses; the data term stays in shared memory where it fits, in L2 where
// not.  A cell's right and lower edge are its block's; its upper and left one
// may be another block's (distributed shared memory).  A cell that the
// quadtree test skips sends its inherited message all along: its edges hold
// that one and are never overwritten.  Only the two last half-sweeps write the
// level's message images (with HIST every one writes its kept state).
// The update is the per-half-sweep kernel's device function, so the messages
// are bit-identical.  Every block of a cluster takes the same barriers: the
// trip counts depend only on the job and the plan.
// Measured (the launch, one stream, messages through L2 with 8 blocks of 512
// threads -> this one): 160x128 (34 half-sweeps) 113 -> 69 us, 752x480 (levels
// 2 and 3) 99 -> 49, 640x480 x 48 92 -> 47; clusters of 8 and 4 blocks: 752x480 76
// and 105 us.  Which levels and how wide a cluster: coarse_plan.
struct CoarseCell
{
  unsigned short local, flags; // index in the block; CoarseFlag bits
  unsigned short up_local, up_rank; // owner of the edge to the upper neighbour
};
enum CoarseFlag
{
  kHas = 1,    // << kUp .. kRight: the neighbour exists
  kOpen = 16,  // << kUp .. kRight: it exists and is not skipped
  kSkip = 256, // the cell itself is skipped
};

__device__ __forceinline__ unsigned cluster_rank()
{
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier()
{
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// the address of p (this block's shared memory) in the block `rank`
__device__ __forceinline__ unsigned cluster_addr(const float *p, unsigned rank)
{
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 cluster_load(unsigned a)
{
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void cluster_store(unsigned a, const float4 &v)
{
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y),
               "f"(v.z), "f"(v.w)
               : "memory");
}

// shared memory of a block with `per` cells, in floats: edges, data term, and
// the cell lists of the two colours, the flags and the list lengths behind it
template <int D>
__host__ __device__ constexpr size_t coarse_smem(int per, bool with_data)
{
  return (size_t)per * (2 + (with_data ? 1 : 0)) * D * sizeof(float) +
         (size_t)per * (2 * sizeof(CoarseCell) + sizeof(unsigned short)) + 32;
}

template <int D, int ARITH, bool HIST>
__global__ void __launch_bounds__(kCoarseMaxThreads, 1)
    k_bp_coarse(const __grid_constant__ Batch B, int j0, const __grid_constant__ CoarsePlan plan,
                KParams kp)
{
  after_previous();
  using QL = QuadLayout<D>;
  constexpr int LPC = QL::LPC, G = 32 / LPC;
  const int threads = blockDim.x, groups = threads / LPC;
  extern __shared__ __align__(16) float s_coarse[];
  const int ctas = plan.ctas;
  const int job = j0 + (int)blockIdx.x / ctas;
  const JobDesc &J = B.jobs ? B.jobs[job] : B.one;
  if (J.D != D)
    return; // the whole cluster
  const int rank = (int)cluster_rank();
  const int tid = threadIdx.x, lane = tid & 31, gl = lane & (LPC - 1), group = tid / LPC;
  const bool lane_on = QL::ACT == LPC || gl < QL::ACT;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float *edges = s_coarse;
  float *data = s_coarse + (size_t)plan.per * 2 * D;
  CoarseCell *lists =
      reinterpret_cast<CoarseCell *>(data + (plan.data_smem ? (size_t)plan.per * D : 0));
  unsigned short *flags = reinterpret_cast<unsigned short *>(lists + 2 * plan.per);
  __shared__ int s_len[2];
  for (int level = plan.hi; level >= plan.lo; --level)
  {
    const LevelDesc &L = J.lv[level];
    const int w = L.w, h = L.h, n = w * h;
    const int per = (n + ctas - 1) / ctas;
    const int c0 = rank * per, cnt = max(0, min(per, n - c0));
    const int iters = plan.iters[level];
    const bool top = level + 1 >= J.nlev;
    const LevelDesc &P = J.lv[top ? level : level + 1];
    // ---- flags of the block's cells
    for (int i = tid; i < cnt; i += threads)
    {
      const int c = c0 + i, y = c / w, x = c - y * w;
      auto skip = [&](int xn, int yn) { return bp_skipped(J, level, xn, yn, kp.qt_max); };
      unsigned f = skip(x, y) ? kSkip : 0;
      if (y > 0)
        f |= (skip(x, y - 1) ? kHas : kHas | kOpen) << kUp;
      if (y < h - 1)
        f |= (skip(x, y + 1) ? kHas : kHas | kOpen) << kDown;
      if (x > 0)
        f |= (skip(x - 1, y) ? kHas : kHas | kOpen) << kLeft;
      if (x < w - 1)
        f |= (skip(x + 1, y) ? kHas : kHas | kOpen) << kRight;
      flags[i] = (unsigned short)f;
    }
    __syncthreads();
    // ---- the cells that are swept, by colour (warps 0 and 1, in order)
    if (tid < 64)
    {
      const int colour = tid >> 5;
      int len = 0;
      for (int i0 = 0; i0 < cnt; i0 += 32)
      {
        const int i = i0 + lane, c = c0 + i, y = c / w, x = c - y * w;
        const bool in = i < cnt && ((x + y) & 1) == colour && !(flags[i] & kSkip);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in)
        {
          const int up = max(c - w, 0), r = up / per;
          lists[colour * plan.per + len + __popc(m & ((1u << lane) - 1u))] =
              CoarseCell{(unsigned short)i, flags[i], (unsigned short)(up - r * per),
                         (unsigned short)r};
        }
        len += __popc(m);
      }
      if (lane == 0)
        s_len[colour] = len;
    }
    // ---- starting messages: an edge gets the message from its odd cell (read
    // by half-sweep 0), or from its even cell where that one is skipped; the
    // parents' final messages, 0 at the coarsest level (what the reference's
    // copied-down messages hold, bpextract.cu:87-90,374-395)
    if (lane_on)
    {
      auto parent = [&](int m, int x, int y) {
        return top ? zero
                   : __ldcg(reinterpret_cast<const float4 *>(
                         P.msg[m] + ((size_t)(y >> 1) * P.w + (x >> 1)) * D + 4 * gl));
      };
      for (int i = group; i < cnt; i += groups)
      {
        const int c = c0 + i, y = c / w, x = c - y * w;
        const unsigned f = flags[i];
        const bool even = ((x + y) & 1) == 0;
#pragma unroll
        for (int e = 0; e < 2; ++e)
        {
          const int to = e == 0 ? kRight : kDown, back = e == 0 ? kLeft : kUp;
          if (!(f & (kHas << to)))
            continue;
          const bool even_skipped = even ? (f & kSkip) != 0 : !(f & (kOpen << to));
          const bool mine = even == even_skipped; // this cell's message, or the neighbour's
          const float4 v = mine ? parent(to, x, y) : parent(back, x + (e == 0), y + (e == 1));
          *reinterpret_cast<float4 *>(edges + ((size_t)i * 2 + e) * D + 4 * gl) = v;
        }
        if (plan.data_smem)
          *reinterpret_cast<float4 *>(data + (size_t)i * D + 4 * gl) =
              *reinterpret_cast<const float4 *>(L.data + (size_t)c * D + 4 * gl);
        if (f & kSkip)
        {
#pragma unroll
          for (int m = 0; m < 4; ++m)
          {
            const float4 v = parent(m, x, y);
            const size_t o = (size_t)c * D + 4 * gl;
            *reinterpret_cast<float4 *>(L.msg[m] + o) = v;
            if constexpr (HIST)
              for (int it = iters - 3; it >= 0; it -= 2)
                *reinterpret_cast<float4 *>(plan.hist[level].at(it, iters, m, L.msg[m]) + o) = v;
          }
        }
      }
    }
    cluster_barrier();
    // ---- half-sweeps
    for (int it = 0; it < iters; ++it)
    {
      const CoarseCell *list = lists + (it & 1) * plan.per;
      const int len = s_len[it & 1];
      const bool out_on = HIST || it >= iters - 2;
      float *out[4];
#pragma unroll
      for (int m = 0; m < 4; ++m)
        out[m] = HIST ? plan.hist[level].at(it, iters, m, L.msg[m]) : L.msg[m];
      for (int k0 = (tid >> 5) * G; k0 < len; k0 += threads / LPC)
      {
        const int k = k0 + lane / LPC;
        const bool on = k < len && lane_on;
        const CoarseCell q = list[min(k, len - 1)];
        const unsigned f = q.flags;
        const int i = q.local;
        float *own = edges + (size_t)i * 2 * D + 4 * gl;
        // the edges to the left (the previous cell's first) and up
        const bool far_l = i == 0, far_u = (int)q.up_rank != rank;
        float *left = edges + (size_t)(far_l ? per - 1 : i - 1) * 2 * D + 4 * gl;
        float *up = edges + ((size_t)q.up_local * 2 + 1) * D + 4 * gl;
        const unsigned left_a = far_l ? cluster_addr(left, max(rank - 1, 0)) : 0u;
        const unsigned up_a = far_u ? cluster_addr(up, q.up_rank) : 0u;
        float4 fu = zero, fd = zero, fl = zero, fr = zero, dat = zero;
        if (on)
        {
          dat = plan.data_smem
                    ? *reinterpret_cast<const float4 *>(data + (size_t)i * D + 4 * gl)
                    : __ldg(reinterpret_cast<const float4 *>(L.data + (size_t)(c0 + i) * D +
                                                             4 * gl));
          if (f & (kHas << kUp))
            fu = far_u ? cluster_load(up_a) : *reinterpret_cast<const float4 *>(up);
          if (f & (kHas << kLeft))
            fl = far_l ? cluster_load(left_a) : *reinterpret_cast<const float4 *>(left);
          if (f & (kHas << kRight))
            fr = *reinterpret_cast<const float4 *>(own);
          if (f & (kHas << kDown))
            fd = *reinterpret_cast<const float4 *>(own + D);
        }
        cell_update<D, ARITH>(dat, fu, fd, fl, fr, kp, gl, [&](int dir, const float4 &v) {
          if (!on)
            return;
          if (f & (kOpen << dir))
          {
            if (dir == kRight)
              *reinterpret_cast<float4 *>(own) = v;
            else if (dir == kDown)
              *reinterpret_cast<float4 *>(own + D) = v;
            else if (dir == kLeft ? far_l : far_u)
              cluster_store(dir == kLeft ? left_a : up_a, v);
            else
              *reinterpret_cast<float4 *>(dir == kLeft ? left : up) = v;
          }
          if (out_on)
            *reinterpret_cast<float4 *>(out[dir] + (size_t)(c0 + i) * D + 4 * gl) = v;
        });
      }
      cluster_barrier();
    }
  }
}

// ------------------------------------------------------------- extract
// The reference's stride-halving argmin (bpextract.cu:340-355) of
// b[j] = value(4 g + j) over the group: a right element replaces the left one
// only when strictly smaller.  Strides of four and more pair lanes; the first
// two also share out the four j over the lanes, so strides 2 and 1 pair lanes
// as well.  Padding must never be smaller than anything (infinity).  Every
// lane ends with the result.
template <int LPC>
__device__ __forceinline__ void quad_argmin(const float (&b)[4], int gl, float &best_v, int &best_i)
{
  // lanes with bit o clear hold the left element
  auto pick = [&](float own, int oi, float other, int ti, bool right, float &v, int &i) {
    const float l = right ? other : own, r = right ? own : other;
    const bool take = r < l;
    v = take ? r : l;
    i = take == right ? oi : ti;
  };
  const bool h1 = (gl & (LPC / 2)) != 0, h2 = (gl & (LPC / 4)) != 0;
  const int mate = gl ^ (LPC / 2);
  float v[2];
  int i[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
  {
    const float send = h1 ? b[j] : b[2 + j], keep = h1 ? b[2 + j] : b[j];
    const float got = __shfl_xor_sync(0xffffffffu, send, LPC / 2);
    const int jj = h1 ? 2 + j : j;
    pick(keep, 4 * gl + jj, got, 4 * mate + jj, h1, v[j], i[j]);
  }
  float r;
  int ri;
  {
    const float send = h2 ? v[0] : v[1], keep = h2 ? v[1] : v[0];
    const int si = h2 ? i[0] : i[1], ki = h2 ? i[1] : i[0];
    const float got = __shfl_xor_sync(0xffffffffu, send, LPC / 4);
    const int gi = __shfl_xor_sync(0xffffffffu, si, LPC / 4);
    pick(keep, ki, got, gi, h2, r, ri);
  }
  auto step = [&](int o) {
    const float got = __shfl_xor_sync(0xffffffffu, r, o);
    const int gi = __shfl_xor_sync(0xffffffffu, ri, o);
    pick(r, ri, got, gi, (gl & o) != 0, r, ri);
  };
#pragma unroll
  for (int o = LPC / 8; o > 0; o >>= 1)
    step(o);
  step(LPC / 2); // stride 2: j and j ^ 2
  step(LPC / 4); // stride 1: j and j ^ 1
  best_v = r;
  best_i = ri;
}

// Extraction, one lane group per level-0 cell, 16 bytes per lane and image as
// in the half-sweeps (five images read, 4 bytes per leaf written).
// Measured, one hypothesis every 8 to 32 per lane -> four consecutive ones:
// 32 x 752x480 x 64 180 -> 152 us, 8 x 1920x1080 x 128 457 -> 316 us (2.65 GB if
// every cell were a leaf origin; the others are not read).
template <int D, int ARITH>
__global__ void __launch_bounds__(kMaxCellWarps * 32)
    k_extract(const __grid_constant__ Batch B)
{
  after_previous();
  using QL = QuadLayout<D>;
  constexpr int LPC = QL::LPC, G = 32 / LPC;
  int lb;
  const JobDesc &J = job_of(B, lb);
  if (J.D != D)
    return;
  const LevelDesc &L = J.lv[0];
  const int w = L.w, h = L.h;
  const int lane = threadIdx.x & 31, gl = lane & (LPC - 1);
  const int cell0 = (lb * (int)(blockDim.x >> 5) + (threadIdx.x >> 5)) * G;
  if (cell0 >= w * h)
    return; // the whole warp
  const int cell = cell0 + lane / LPC;
  int x = 0, y = 0;
  bool act = cell < w * h;
  if (act)
  {
    x = cell % w;
    y = cell / w;
    const int lvl = J.levels[(size_t)min(y * 4, J.H - 1) * J.W + min(x * 4, J.W - 1)];
    const int size = 1 << lvl;
    if ((x * 4) % size != 0 || (y * 4) % size != 0)
    {
      if (gl == 0 && J.labels)
        J.labels[cell] = -1;
      act = false;
    }
  }
  if (!__any_sync(0xffffffffu, act))
    return;
  const bool on = act && (QL::ACT == LPC || gl < QL::ACT);
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const size_t c = (size_t)cell * D + 4 * gl;
  auto msg = [&](int dir, bool has, long off) {
    return on && has ? msg_load(L.msg[dir] + (c + off * D)) : zero;
  };
  const float4 dat = on ? *reinterpret_cast<const float4 *>(L.data + c) : zero;
  const float4 fl = msg(kRight, x > 0, -1), fr = msg(kLeft, x < w - 1, 1);
  const float4 fu = msg(kDown, y > 0, -w), fd = msg(kUp, y < h - 1, w);
  // the reference's order: from the left, the right, above, below
  float b[4] = {(((dat.x + fl.x) + fr.x) + fu.x) + fd.x, (((dat.y + fl.y) + fr.y) + fu.y) + fd.y,
                (((dat.z + fl.z) + fr.z) + fu.z) + fd.z, (((dat.w + fl.w) + fr.w) + fu.w) + fd.w};
  if (QL::ACT < LPC && gl >= QL::ACT)
    b[0] = b[1] = b[2] = b[3] = __int_as_float(0x7f800000);
  float bmin;
  int best;
  quad_argmin<LPC>(b, gl, bmin, best);
  // neighbours of the winner for the parabola
  auto at = [&](int d) {
    const float lo = (d & 1) ? b[1] : b[0], hi = (d & 1) ? b[3] : b[2];
    return __shfl_sync(0xffffffffu, (d & 2) ? hi : lo, d >> 2, LPC);
  };
  const float pre = at(best > 0 ? best - 1 : 0), post = at(best < D - 1 ? best + 1 : D - 1);
  if (gl != 0 || !act)
    return;
  float disparity = (float)best;
  if (best > 0 && best < D - 1)
  {
    if (ARITH == QM_ARITH_IEEE)
    {
      const float a = __fadd_rn(__fsub_rn(pre, __fmul_rn(2.0f, bmin)), post);
      const float bb = __fadd_rn(-pre, post);
      const float b_a = __fdiv_rn(bb, a);
      if (isfinite(b_a))
        disparity = __fsub_rn((float)best, __fdiv_rn(b_a, 2.0f));
    }
    else
    {
      const float a = pre - 2.0f * bmin + post;
      const float bb = -pre + post;
      const float b_a = bb / a;
      if (isfinite(b_a))
        disparity = (float)best - b_a / 2.0f;
    }
  }
  float depth;
  if (ARITH == QM_ARITH_IEEE)
    depth = (float)__ddiv_rn(1.0, __dadd_rn(__dmul_rn(J.step, (double)disparity), J.min_inv));
  else
    depth = 1.0 / (J.step * disparity + J.min_inv);
  J.sparse[(size_t)(y * 4) * J.W + x * 4] = depth;
  if (J.labels)
    J.labels[cell] = best;
}

template <int D>
void sweep_d(const Batch &B, int blocks, int level, int parity, int first, int inherit,
             KParams kp, int arith, int warps, cudaStream_t s)
{
  if (arith == QM_ARITH_IEEE)
    launch_kernel(k_bp_sweep<D, QM_ARITH_IEEE>, blocks, warps * 32, 0, s, B.early, B, level,
                  parity, first, inherit, kp);
  else
    launch_kernel(k_bp_sweep<D, QM_ARITH_REFERENCE>, blocks, warps * 32, 0, s, B.early, B, level,
                  parity, first, inherit, kp);
}

// Opt-ins of one k_bp_coarse instance on the current device (large shared
// memory, clusters of 16); returns how many clusters of 16 full blocks the
// device runs at once (0: it has none; a B200 runs 7).
template <int D, int ARITH, bool HIST>
int coarse_prepare()
{
  static std::atomic<unsigned long long> done{0};
  static std::atomic<int> wide[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess)
    return 0;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(done.load(std::memory_order_acquire) & bit))
  {
    const auto k = k_bp_coarse<D, ARITH, HIST>;
    check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxBlockSmem - 64),
          "BP cluster kernel");
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kCoarseMaxCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    c.gridDim = dim3(kCoarseMaxCtas);
    c.blockDim = dim3(kCoarseMaxThreads);
    c.dynamicSmemBytes = kMaxBlockSmem - 64;
    c.attrs = at;
    c.numAttrs = 1;
    int clusters = 0;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveClusters(&clusters, k, &c);
    if (e != cudaSuccess)
    {
      cudaGetLastError(); // a device without such clusters is no error
      clusters = 0;
    }
    wide[dev & 63].store(clusters, std::memory_order_relaxed);
    done.fetch_or(bit, std::memory_order_acq_rel);
  }
  return wide[dev & 63].load(std::memory_order_relaxed);
}

template <int D, int ARITH, bool HIST>
void coarse_k(const Batch &B, int j0, int jobs, const CoarsePlan &plan, KParams kp, cudaStream_t s)
{
  coarse_prepare<D, ARITH, HIST>();
  cudaLaunchConfig_t c = {};
  cudaLaunchAttribute at[2];
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = plan.ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  c.gridDim = dim3(jobs * plan.ctas);
  c.blockDim = dim3(plan.threads);
  c.dynamicSmemBytes = coarse_smem<D>(plan.per, plan.data_smem != 0);
  c.stream = s;
  c.attrs = at;
  c.numAttrs = B.early ? 2 : 1;
  check(cudaLaunchKernelEx(&c, k_bp_coarse<D, ARITH, HIST>, B, j0, plan, kp), "kernel launch");
}

template <int D>
void coarse_d(const Batch &B, int j0, int jobs, const CoarsePlan &plan, KParams kp, int arith,
              cudaStream_t s)
{
  constexpr int R = QM_ARITH_REFERENCE, I = QM_ARITH_IEEE;
  if (arith == QM_ARITH_IEEE)
    plan.keep ? coarse_k<D, I, true>(B, j0, jobs, plan, kp, s)
              : coarse_k<D, I, false>(B, j0, jobs, plan, kp, s);
  else
    plan.keep ? coarse_k<D, R, true>(B, j0, jobs, plan, kp, s)
              : coarse_k<D, R, false>(B, j0, jobs, plan, kp, s);
}

// clusters of 16 blocks that run at once, as coarse_prepare
template <int D>
int coarse_wide_d(bool keep, int arith)
{
  constexpr int R = QM_ARITH_REFERENCE, I = QM_ARITH_IEEE;
  if (arith == QM_ARITH_IEEE)
    return keep ? coarse_prepare<D, I, true>() : coarse_prepare<D, I, false>();
  return keep ? coarse_prepare<D, R, true>() : coarse_prepare<D, R, false>();
}

template <int D>
bool coarse_fit_d(CoarsePlan &plan, long cells, int ctas, bool shared_sm)
{
  const long per = (cells + ctas - 1) / ctas;
  constexpr size_t room = kMaxBlockSmem - 64; // 64: s_len
  if (per > 4096 || coarse_smem<D>((int)per, false) > room)
    return false;
  plan.ctas = ctas;
  plan.per = (int)per;
  // two blocks per SM: half the threads each, and half the shared memory if
  // that is possible without the data term
  const size_t half = kMaxBlockSmem / 2 - 2048;
  const bool split = shared_sm && coarse_smem<D>((int)per, false) <= half;
  plan.threads = split ? 512 : kCoarseMaxThreads;
  plan.data_smem = coarse_smem<D>((int)per, true) <= (split ? half : room) ? 1 : 0;
  return true;
}

template <int D>
void sweep_io_d(const Batch &B, int blocks, int level, int it, const SweepIO &io, KParams kp,
                int arith, cudaStream_t s)
{
  if (arith == QM_ARITH_IEEE)
    launch_kernel(k_bp_sweep_io<D, QM_ARITH_IEEE>, blocks, kCellWarps * 32, 0, s, B.early, B,
                  level, it & 1, it == 0, io, kp);
  else
    launch_kernel(k_bp_sweep_io<D, QM_ARITH_REFERENCE>, blocks, kCellWarps * 32, 0, s, B.early, B,
                  level, it & 1, it == 0, io, kp);
}

template <int D>
void extract_d(const Batch &B, int blocks, int arith, int warps, cudaStream_t s)
{
  if (arith == QM_ARITH_IEEE)
    launch_kernel(k_extract<D, QM_ARITH_IEEE>, blocks, warps * 32, 0, s, B.early, B);
  else
    launch_kernel(k_extract<D, QM_ARITH_REFERENCE>, blocks, warps * 32, 0, s, B.early, B);
}

} // namespace

namespace
{
// f(std::integral_constant<int, d>) for a supported hypothesis count
template <class F>
void by_d(int d, F &&f)
{
  switch (d)
  {
  case 32: f(std::integral_constant<int, 32>()); break;
  case 48: f(std::integral_constant<int, 48>()); break;
  case 64: f(std::integral_constant<int, 64>()); break;
  case 96: f(std::integral_constant<int, 96>()); break;
  case 128: f(std::integral_constant<int, 128>()); break;
  default: break;
  }
}
} // namespace

bool bp_supported_d(int d) { return d == 32 || d == 48 || d == 64 || d == 96 || d == 128; }

int bp_cells_per_warp(int d)
{
  switch (d)
  {
  case 32: return QuadLayout<32>::G;
  case 48: return QuadLayout<48>::G;
  case 64: return QuadLayout<64>::G;
  case 96: return QuadLayout<96>::G;
  case 128: return QuadLayout<128>::G;
  default: return 1;
  }
}

int pyramid_blocks(int w, int h) { return (w + 3) / 4 * ((h + 3) / 4); }

void launch_pyramid(const Batch &B, int blocks, int level, int n, cudaStream_t s)
{
  launch_kernel(k_pyramid, blocks, kFlatThreads, 0, s, B.early, B, level, n);
}

void launch_msg_inherit(const Batch &B, int blocks, int level, int iters, int qt_max,
                        cudaStream_t s)
{
  launch_kernel(k_msg_inherit, blocks, kFlatThreads, 0, s, B.early, B, level, iters, qt_max);
}

// A batch with mixed hypothesis counts launches one sweep per count present;
// each launch skips the jobs of other counts.
void launch_bp_sweep(const Batch &B, int blocks, int d, int level, int it, KParams kp, int arith,
                     cudaStream_t s, int warps, int inherit)
{
  by_d(d, [&](auto dc) {
    sweep_d<decltype(dc)::value>(B, blocks, level, it & 1, it == 0 ? 1 : 0,
                                 inherit && it < 2 ? 1 : 0, kp, arith, warps, s);
  });
}

void launch_bp_sweep_io(const Batch &B, int d, int level, int it, const SweepIO &io, KParams kp,
                        int arith, cudaStream_t s)
{
  const LevelDesc &L = B.one.lv[level];
  const int per = kCellWarps * bp_cells_per_warp(d);
  const int blocks = ((L.w + 1) / 2 * L.h + per - 1) / per;
  if (blocks > 0)
    by_d(d, [&](auto dc) {
      sweep_io_d<decltype(dc)::value>(B, blocks, level, it, io, kp, arith, s);
    });
}

bool coarse_plan(CoarsePlan &plan, int d, const long *cells, int levels, const int *iters,
                 long max_cells, int jobs, int arith)
{
  plan.lo = levels;
  plan.hi = levels - 1;
  for (int l = 0; l < levels; ++l)
    plan.iters[l] = iters[l];
  // As wide a cluster for each job as lets those of all jobs run at once: 16
  // blocks of 1024 threads (a half-sweep's latency counts), above what the
  // device holds of these 16 of 512, two on an SM, if the level fits them so,
  // and above twice as many 8 of 512.  Measured (resident pass, 16 of 1024 / 16
  // of 512 / 8 of 512): 160x128 x 64, 8 streams 215 / 161 / 171 us, 12 225 / 172
  // / 181, 16 294 / 236 / 198; 320x240 8 267 / 255 / 272, 12 331 / 306 / 316;
  // 752x480 12 951 / 943 / 937, 24 1858 / 1809 / 1783.
  for (int l = levels - 1; l >= 0 && iters[l] >= 2; --l)
  {
    bool ok = false;
    by_d(d, [&](auto dc) {
      constexpr int D = decltype(dc)::value;
      const int wide = coarse_wide_d<D>(plan.keep != 0, arith);
      // lane groups of a cluster x 2 colours x rounds
      const long most = max_cells != kCoarseAuto ? max_cells
                                                 : kCoarseMaxCtas * kCoarseMaxThreads /
                                                       QuadLayout<D>::LPC * 2L *
                                                       (jobs > 1 && jobs <= wide ? 2 : 1);
      const int first = jobs <= 2 * wide ? kCoarseMaxCtas : 8;
      for (int ctas : {first, kCoarseMaxCtas + 8 - first})
        ok = ok || (cells[l] <= most && (ctas <= 8 || wide > 0) &&
                    coarse_fit_d<D>(plan, cells[l], ctas, jobs > wide));
    });
    if (!ok)
      break;
    plan.lo = l;
  }
  return plan.lo < levels;
}

void launch_bp_coarse(const Batch &B, int j0, int jobs, int d, const CoarsePlan &plan,
                      KParams kp, int arith, cudaStream_t s)
{
  by_d(d, [&](auto dc) { coarse_d<decltype(dc)::value>(B, j0, jobs, plan, kp, arith, s); });
}

void launch_extract(const Batch &B, int blocks, int d, int arith, cudaStream_t s, int warps)
{
  by_d(d, [&](auto dc) { extract_d<decltype(dc)::value>(B, blocks, arith, warps, s); });
}

} // namespace qm
