// Differentiable path (the training-side pattern of the pipeline): a
// temperature-softened BP belief readout and the adjoints of the BP
// half-sweeps, of an edge-aware upsampling with per-pixel weight factors, and
// of the fusion update.  The product path keeps the hard argmin; these
// kernels serve parameter fitting (BP penalties P1, P2 and the upsampling
// weight factors) against ground-truth depth.
//
// Soft readout, per node cell (the node test of depth_extract,
// bpextract.cu:314-372): beliefs b(d) = data + the four incoming messages in
// the extraction's order, p(d) = softmax(-b(d)/tau), disparity = sum p(d) d,
// depth = 1 / (step * disparity + min) (FP64).
//
// BP adjoint.  A half-sweep writes, for every updated cell c and direction,
// m(d) = min(h(d), h(d-1)+P1, h(d+1)+P1, min_k h(k)+P2) - mean_d(...), where h
// is the data term plus three incoming messages.  Reverse mode follows the
// selected term of each minimum (ties go to the earliest candidate, the
// forward's order) and subtracts the mean of the adjoint.  The adjoint state
// A holds dL/d(message) for every cell and direction; the backward of a
// half-sweep consumes A at the cells it updated (their earlier values were
// overwritten) and writes A at the neighbours' messages those cells read, each
// read by exactly one cell (no atomics).  dL/dP1 and dL/dP2 are accumulated in
// FP64.  The messages come from the states the forward half-sweeps left (a
// half-sweep only reads the other colour, so two of them share one state).
//
// Weighted upsampling: the row and column systems of global_upsample
// (depth_upsample.cu:20-302) with every inner edge weight multiplied by a
// per-pixel factor omega (the edge between a pixel and its left / upper
// neighbour takes that pixel's factor), solved per line in FP64 by the Thomas
// algorithm (its recurrences scanned by a warp per line).  The systems are
// symmetric, so the adjoint solve is the same solve; dL/dw for the edge (k-1, k)
// is -lambda (g(k) - g(k-1)) (s(k) - s(k-1)) summed over the two right-hand sides.
//
// Fusion adjoint: the update of fuse_currentmap evaluated on dual numbers
// (value, derivative with respect to the upsampled depth).
#include <atomic>
#include <cfloat>
#include <type_traits>

#include "launch.h"

namespace qm
{

namespace
{

constexpr int kDiffWarps = 8;

// Arithmetic of a real type: float for the product path, double for the
// gradient-check mode.
template <class R>
struct Real;
template <>
struct Real<float>
{
  static __device__ __forceinline__ float big() { return FLT_MAX; }
  static __device__ __forceinline__ float min(float a, float b) { return fminf(a, b); }
  static __device__ __forceinline__ float exp(float a) { return expf(a); }
};
template <>
struct Real<double>
{
  static __device__ __forceinline__ double big() { return DBL_MAX; }
  static __device__ __forceinline__ double min(double a, double b) { return fmin(a, b); }
  static __device__ __forceinline__ double exp(double a) { return ::exp(a); }
};

template <class R>
__device__ __forceinline__ R warp_sum(R v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <class R>
__device__ __forceinline__ R warp_min(R v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = Real<R>::min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// value at hypothesis d-1 / d+1 of a per-lane register array (lane l holds
// d = l + 32k), one shuffle per register; lanes at the ends of the range get
// their own value back (callers mask them)
template <int NV, class R>
__device__ __forceinline__ void neighbours(const R (&v)[NV], int lane, int k, R &prev, R &next)
{
  const R up_src = (lane == 31 && k > 0) ? v[k > 0 ? k - 1 : 0] : v[k];
  const R dn_src = (lane == 0 && k + 1 < NV) ? v[k + 1 < NV ? k + 1 : k] : v[k];
  prev = __shfl_sync(0xffffffffu, up_src, (lane + 31) & 31);
  next = __shfl_sync(0xffffffffu, dn_src, (lane + 1) & 31);
}

template <class R>
__device__ __forceinline__ bool skipped(const DiffBpR<R> &a, int x, int y)
{
  const int ilev = a.level + 2;
  if (ilev > a.qt_max)
    return false;
  const int size = 1 << ilev;
  const int sx = min((x >> 1) * size, a.W - 1), sy = min(y * size, a.H - 1);
  return (int)a.levels[(size_t)sy * a.W + sx] > ilev;
}

template <class R>
__device__ __forceinline__ bool is_node(const DiffBpR<R> &a, int x, int y)
{
  const int lvl = a.levels[(size_t)min(y * 4, a.H - 1) * a.W + min(x * 4, a.W - 1)];
  const int size = 1 << lvl;
  return (x * 4) % size == 0 && (y * 4) % size == 0;
}

// ------------------------------------------------------------ soft readout
template <int D, class R>
__global__ void __launch_bounds__(kDiffWarps * 32)
    k_soft_readout(const DiffBpR<R> a, int backward)
{
  after_previous();
  using M = Real<R>;
  constexpr int NV = (D + 31) / 32;
  const int cell = blockIdx.x * kDiffWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int w = a.w, h = a.h;
  if (cell >= w * h)
    return;
  const int x = cell % w, y = cell / w;
  const size_t c = (size_t)cell;
  const size_t px = (size_t)(y * 4) * a.W + x * 4;
  const bool node = is_node(a, x, y);
  const float g = backward && node ? a.g_sparse[px] : 0.0f;
  if (backward)
  {
    // messages that leave the image have no reader
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      const int d = lane + 32 * k;
      if (d >= D)
        continue;
      if (x == 0)
        a.A[kLeft][c * D + d] = (R)0;
      if (x == w - 1)
        a.A[kRight][c * D + d] = (R)0;
      if (y == 0)
        a.A[kUp][c * D + d] = (R)0;
      if (y == h - 1)
        a.A[kDown][c * D + d] = (R)0;
    }
  }
  // adjoint of the four messages the cell reads (each read by this cell only)
  auto put = [&](int d, R v) {
    if (x != 0)
      a.A[kRight][(c - 1) * D + d] = v;
    if (x != w - 1)
      a.A[kLeft][(c + 1) * D + d] = v;
    if (y != 0)
      a.A[kDown][(c - w) * D + d] = v;
    if (y != h - 1)
      a.A[kUp][(c + w) * D + d] = v;
  };
  if (backward && g == 0.0f)
  {
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane + 32 * k < D)
        put(lane + 32 * k, (R)0);
    return;
  }
  if (!node)
    return;
  R b[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    const int d = lane + 32 * k;
    R v = M::big();
    if (d < D)
    {
      v = a.data[c * D + d];
      if (x != 0)
        v += a.S[kRight][(c - 1) * D + d];
      if (x != w - 1)
        v += a.S[kLeft][(c + 1) * D + d];
      if (y != 0)
        v += a.S[kDown][(c - w) * D + d];
      if (y != h - 1)
        v += a.S[kUp][(c + w) * D + d];
    }
    b[k] = v;
  }
  R lmin = M::big();
#pragma unroll
  for (int k = 0; k < NV; ++k)
    lmin = M::min(lmin, b[k]);
  const R bmin = warp_min<R>(lmin);
  const R tau = (R)a.tau;
  R e[NV], z = 0, s = 0;
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    const int d = lane + 32 * k;
    e[k] = d < D ? M::exp(-(b[k] - bmin) / tau) : (R)0;
    z += e[k];
    s += e[k] * (R)d;
  }
  z = warp_sum<R>(z);
  s = warp_sum<R>(s);
  const R disp = s / z;
  const double depth = 1.0 / (a.step * (double)disp + a.min_inv);
  if (!backward)
  {
    if (lane == 0)
      a.sparse[px] = (float)depth;
    return;
  }
  // d depth / d disparity = -step * depth^2; d disparity / d b(d) =
  // -(1/tau) p(d) (d - disparity)
  const R g_disp = (R)(-a.step * depth * depth * (double)g);
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    const int d = lane + 32 * k;
    if (d >= D)
      continue;
    put(d, g_disp * (-(e[k] / z) * ((R)d - disp) / tau));
  }
}

// ------------------------------------------------------------ BP adjoint
// The adjoint of one cell's update; adds to the lane's dL/dP1 and dL/dP2.
template <int D, class R>
__device__ __forceinline__ void bwd_cell(const DiffBpR<R> &a, int x, int y, int lane, R &gp1,
                                         R &gp2)
{
  using M = Real<R>;
  constexpr int NV = (D + 31) / 32;
  const int w = a.w, h = a.h;
  const bool has_u = y > 0, has_d = y < h - 1, has_l = x > 0, has_r = x < w - 1;
  if (skipped(a, x, y))
    return;
  const bool sk_u = has_u && skipped(a, x, y - 1), sk_d = has_d && skipped(a, x, y + 1);
  const bool sk_l = has_l && skipped(a, x - 1, y), sk_r = has_r && skipped(a, x + 1, y);
  const size_t c = (size_t)y * w + x;
  // where the neighbours' messages to this cell lie
  auto at = [&](int xn, int yn) {
    return (a.first ? (size_t)(yn >> 1) * a.pw + (xn >> 1) : (size_t)yn * w + xn) * D;
  };
  const bool ld = a.S[0] != nullptr;
  const size_t ou = ld && has_u ? at(x, y - 1) : 0, od = ld && has_d ? at(x, y + 1) : 0;
  const size_t ol = ld && has_l ? at(x - 1, y) : 0, orr = ld && has_r ? at(x + 1, y) : 0;
  R dat[NV], fu[NV], fd[NV], fl[NV], fr[NV], am[4][NV];
  R gu[NV], gd[NV], gl[NV], gr[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    const int d = lane + 32 * k;
    const bool in = d < D;
    dat[k] = in ? a.data[c * D + d] : (R)0;
    fu[k] = (in && ld && has_u) ? a.S[kDown][ou + d] : (R)0;
    fd[k] = (in && ld && has_d) ? a.S[kUp][od + d] : (R)0;
    fl[k] = (in && ld && has_l) ? a.S[kRight][ol + d] : (R)0;
    fr[k] = (in && ld && has_r) ? a.S[kLeft][orr + d] : (R)0;
#pragma unroll
    for (int m = 0; m < 4; ++m)
      am[m][k] = in ? a.A[m][c * D + d] : (R)0;
    gu[k] = gd[k] = gl[k] = gr[k] = (R)0;
  }
  const R P1 = (R)a.P1, P2 = (R)a.P2;
#pragma unroll
  for (int dir = 0; dir < 4; ++dir)
  {
    R hv[NV];
    R lmin = M::big();
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      R v = dat[k];
      if (dir != kUp && has_u)
        v += fu[k];
      if (dir != kDown && has_d)
        v += fd[k];
      if (dir != kLeft && has_l)
        v += fl[k];
      if (dir != kRight && has_r)
        v += fr[k];
      hv[k] = (lane + 32 * k < D) ? v : M::big();
      lmin = M::min(lmin, hv[k]);
    }
    const R hmin = warp_min<R>(lmin);
    // the first hypothesis attaining the minimum
    int amin = D;
#pragma unroll
    for (int k = NV - 1; k >= 0; --k)
    {
      const unsigned bal = __ballot_sync(0xffffffffu, hv[k] == hmin);
      if (bal)
        amin = 32 * k + __ffs(bal) - 1;
    }
    // adjoint of the outgoing message, minus its mean
    R gm[NV], gsum = 0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      gm[k] = am[dir][k];
      gsum += gm[k];
    }
    const R gmean = warp_sum<R>(gsum) / (R)D;
    // selected term of every minimum: 0 own, 1 from d-1, 2 from d+1, 3 P2
    int sel[NV];
    R own[NV], to_prev[NV], to_next[NV], s3 = 0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      const int d = lane + 32 * k;
      R prev, next;
      neighbours<NV>(hv, lane, k, prev, next);
      gm[k] = d < D ? gm[k] - gmean : (R)0;
      R best = hv[k];
      int s = 0;
      if (d > 0 && prev + P1 < best)
      {
        best = prev + P1;
        s = 1;
      }
      if (d < D - 1 && next + P1 < best)
      {
        best = next + P1;
        s = 2;
      }
      if (hmin + P2 < best)
        s = 3;
      sel[k] = d < D ? s : 0;
      own[k] = sel[k] == 0 ? gm[k] : (R)0;
      to_prev[k] = sel[k] == 1 ? gm[k] : (R)0; // lands on h(d-1)
      to_next[k] = sel[k] == 2 ? gm[k] : (R)0; // lands on h(d+1)
      if (sel[k] == 1 || sel[k] == 2)
        gp1 += gm[k];
      if (sel[k] == 3)
      {
        gp2 += gm[k];
        s3 += gm[k];
      }
    }
    s3 = warp_sum<R>(s3);
    R gh[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      // h(d) receives to_prev from d+1 and to_next from d-1
      R from_next, unused, from_prev;
      neighbours<NV>(to_prev, lane, k, unused, from_next);
      neighbours<NV>(to_next, lane, k, from_prev, unused);
      const int d = lane + 32 * k;
      R v = own[k];
      if (d + 1 < D)
        v += from_next;
      if (d > 0)
        v += from_prev;
      if (d == amin)
        v += s3;
      gh[k] = d < D ? v : (R)0;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      if (dir != kUp)
        gu[k] += gh[k];
      if (dir != kDown)
        gd[k] += gh[k];
      if (dir != kLeft)
        gl[k] += gh[k];
      if (dir != kRight)
        gr[k] += gh[k];
    }
  }
  auto put = [&](bool there, bool add, R *p, const R(&v)[NV]) {
    if (!there)
      return;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (lane + 32 * k < D)
        p[lane + 32 * k] = add ? p[lane + 32 * k] + v[k] : v[k];
  };
  // the cell's own messages that no cell of this level reads
  const R zero[NV] = {};
  put(!has_u || sk_u, false, a.A[kUp] + c * D, zero);
  put(!has_d || sk_d, false, a.A[kDown] + c * D, zero);
  put(!has_l || sk_l, false, a.A[kLeft] + c * D, zero);
  put(!has_r || sk_r, false, a.A[kRight] + c * D, zero);
  put(has_u, a.last || sk_u, a.A[kDown] + (c - w) * D, gu);
  put(has_d, a.last || sk_d, a.A[kUp] + (c + w) * D, gd);
  put(has_l, a.last || sk_l, a.A[kRight] + (c - 1) * D, gl);
  put(has_r, a.last || sk_r, a.A[kLeft] + (c + 1) * D, gr);
}

// One warp per cell of the colour.  Bound: its bytes, 13 D values per cell
// (data, four messages and four adjoints read, four adjoints written), from
// L2 at the coarser levels.  Between two half-sweeps every adjoint of the
// other colour is consumed, so the adjoints of the messages read are stored,
// not added (nor is A cleared), with three exceptions: after the level's last
// half-sweep they hold the readout's (or the finer level's) adjoint of the
// final messages; a cell that the quadtree test skips is never consumed
// before the start of the level, its adjoint collects every reader's; and a
// message to a skipped cell or out of the image has no reader at this level
// (only the finer one's copy-down), so its cell clears it once consumed.
// dL/dP1 and dL/dP2 leave a block as one atomic each.  Measured at 752x480 with
// 64 hypotheses (34 half-sweeps): 0.395 -> 0.257 ms.
template <int D, class R>
__global__ void __launch_bounds__(kDiffWarps * 32) k_bp_sweep_bwd(const DiffBpR<R> a)
{
  after_previous();
  __shared__ double s_gp[2][kDiffWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int w = a.w, h = a.h, hw = (w + 1) / 2;
  const int item = blockIdx.x * kDiffWarps + warp;
  const int y = item / hw;
  const int x = 2 * (item - y * hw) + ((y + a.parity) & 1);
  R gp1 = 0, gp2 = 0;
  if (y < h && x < w)
    bwd_cell<D, R>(a, x, y, lane, gp1, gp2);
  const double t1 = warp_sum<double>((double)gp1), t2 = warp_sum<double>((double)gp2);
  if (lane == 0)
  {
    s_gp[0][warp] = t1;
    s_gp[1][warp] = t2;
  }
  __syncthreads();
  if (threadIdx.x < 2)
  {
    double t = 0.0;
    for (int i = 0; i < kDiffWarps; ++i)
      t += s_gp[threadIdx.x][i];
    atomicAdd(a.gP + threadIdx.x, t);
  }
}

// Adjoint of the copy-down: a parent message's is the sum of the adjoints of
// its (up to four) children's starting messages.  Half-sweep 0 overwrites the
// cells with x + y even before anything reads them: their starting messages
// count only where the quadtree test skips the cell (or nothing is swept).
template <class R>
__global__ void __launch_bounds__(256)
    k_msg_downsample(const DiffBpR<R> a, const MsgPtrsR<R> parent, int pw, int ph)
{
  after_previous();
  const int D = a.D;
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)pw * ph * D)
    return;
  const int p = (int)(t / D), d = (int)(t - (long)p * D);
  const int px = p % pw, py = p / pw;
  R s[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i)
    {
      const int x = 2 * px + i, y = 2 * py + j;
      if (x >= a.w || y >= a.h || !(a.iters == 0 || ((x + y) & 1) || skipped(a, x, y)))
        continue;
#pragma unroll
      for (int m = 0; m < 4; ++m)
        s[m] += a.A[m][((size_t)y * a.w + x) * D + d];
    }
#pragma unroll
  for (int m = 0; m < 4; ++m)
    parent.m[m][(size_t)p * D + d] = s[m];
}

// ------------------------------------------- FP64 BP forward (gradient check)
__global__ void __launch_bounds__(256) k_widen(const float *in, double *out, long n)
{
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n)
    out[t] = (double)in[t];
}

// cost_distribute (bpextract.cu:169-198) in FP64: children summed x offset
// outer, y offset inner
__global__ void __launch_bounds__(256)
    k_pyramid64(const double *fine, int fw, int fh, double *coarse, int cw, int ch, int D)
{
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)cw * ch * D)
    return;
  const int p = (int)(t / D), d = (int)(t - (long)p * D);
  const int x = p % cw, y = p / cw;
  double s = 0.0;
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j)
      if (2 * x + i < fw && 2 * y + j < fh)
        s += fine[((size_t)(2 * y + j) * fw + (2 * x + i)) * D + d];
  coarse[t] = s;
}

// the reference's copy-down of the parent's messages (upsample,
// bpextract.cu:374-395), zeros at the coarsest level (bpextract.cu:87-90)
__global__ void __launch_bounds__(256)
    k_msg_inherit_all64(const MsgPtrs64 parent, int has_parent, int pw, const MsgPtrs64 child,
                        int cw, int ch, int D)
{
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)cw * ch * D)
    return;
  const int p = (int)(t / D), d = (int)(t - (long)p * D);
  const int x = p % cw, y = p / cw;
  const size_t src = ((size_t)(y >> 1) * pw + (x >> 1)) * D + d;
#pragma unroll
  for (int m = 0; m < 4; ++m)
    child.m[m][t] = has_parent ? parent.m[m][src] : 0.0;
}

// one half-sweep (bp, bpextract.cu:200-312) in FP64, a warp per cell of the
// colour, messages M updated in place
template <int D>
__global__ void __launch_bounds__(kDiffWarps * 32)
    k_bp_sweep_fwd64(const DiffBp64 a, const MsgPtrs64 M)
{
  using RM = Real<double>;
  constexpr int NV = (D + 31) / 32;
  const int lane = threadIdx.x & 31;
  const int w = a.w, h = a.h, hw = (w + 1) / 2;
  const int item = blockIdx.x * kDiffWarps + (threadIdx.x >> 5);
  if (item >= hw * h)
    return;
  const int y = item / hw;
  const int x = 2 * (item - y * hw) + ((y + a.parity) & 1);
  if (x >= w || skipped(a, x, y))
    return;
  const bool has_u = y > 0, has_d = y < h - 1, has_l = x > 0, has_r = x < w - 1;
  const size_t c = (size_t)y * w + x;
  double dat[NV], fu[NV], fd[NV], fl[NV], fr[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k)
  {
    const int d = lane + 32 * k;
    const bool in = d < D;
    dat[k] = in ? a.data[c * D + d] : 0.0;
    fu[k] = (in && has_u) ? M.m[kDown][(c - w) * D + d] : 0.0;
    fd[k] = (in && has_d) ? M.m[kUp][(c + w) * D + d] : 0.0;
    fl[k] = (in && has_l) ? M.m[kRight][(c - 1) * D + d] : 0.0;
    fr[k] = (in && has_r) ? M.m[kLeft][(c + 1) * D + d] : 0.0;
  }
  const double P1 = a.P1, P2 = a.P2;
#pragma unroll
  for (int dir = 0; dir < 4; ++dir)
  {
    double hv[NV];
    double lmin = RM::big();
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      double v = dat[k];
      if (dir != kUp && has_u)
        v += fu[k];
      if (dir != kDown && has_d)
        v += fd[k];
      if (dir != kLeft && has_l)
        v += fl[k];
      if (dir != kRight && has_r)
        v += fr[k];
      hv[k] = (lane + 32 * k < D) ? v : RM::big();
      lmin = fmin(lmin, hv[k]);
    }
    const double hmin = warp_min<double>(lmin);
    double m[NV], msum = 0.0;
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      const int d = lane + 32 * k;
      double prev, next;
      neighbours<NV>(hv, lane, k, prev, next);
      double v = hv[k];
      if (d > 0)
        v = fmin(v, prev + P1);
      if (d < D - 1)
        v = fmin(v, next + P1);
      m[k] = fmin(v, hmin + P2);
      if (d < D)
        msum += m[k];
    }
    const double mean = warp_sum<double>(msum) / (double)D;
#pragma unroll
    for (int k = 0; k < NV; ++k)
    {
      const int d = lane + 32 * k;
      if (d < D)
        M.m[dir][c * D + d] = m[k] - mean;
    }
  }
}

// ------------------------------------------------------ weighted upsampling
// Edge weight factor: exp(-(Ia - Ib)^2 / sigma) in FP64.
__device__ __forceinline__ double edge_exp(double a, double b, double sigma)
{
  const double diff = a - b;
  return exp(-diff * diff / sigma);
}

// weight of the edge (k-1, k) of a line of n samples: k = 0 -> 0, k = n ->
// the closing weight, else omega * exp term
struct LineW
{
  const uint8_t *img;
  size_t step_img; // image elements between consecutive samples
  const float *omega;
  size_t step;     // pixel elements between consecutive samples
  int n;
  double closing, sigma;
  __device__ double w(int k, double *expo = nullptr) const
  {
    if (k <= 0)
      return 0.0;
    if (k >= n)
      return closing;
    const double e = edge_exp((double)img[k * step_img], (double)img[(k - 1) * step_img], sigma);
    if (expo)
      *expo = e;
    return (double)omega[k * step] * e;
  }
};

// Solves (I + lam L_w) s = r along one line for two right-hand sides (FP64
// Thomas); cp is scratch of n doubles.  r and s may alias.
__device__ void thomas2(const LineW &L, double lam, const double *r0, const double *r1,
                        double *s0, double *s1, double *cp, size_t step)
{
  const int n = L.n;
  double wl = L.w(0), wr = L.w(1);
  double den = 1.0 + lam * (wl + wr);
  double c = -lam * wr / den;
  double d0 = r0[0] / den, d1 = r1[0] / den;
  cp[0] = c;
  s0[0] = d0;
  s1[0] = d1;
  for (int k = 1; k < n; ++k)
  {
    wl = wr;
    wr = L.w(k + 1);
    const double a = -lam * wl;
    den = 1.0 + lam * (wl + wr) - a * c;
    c = -lam * wr / den;
    d0 = (r0[k * step] - a * d0) / den;
    d1 = (r1[k * step] - a * d1) / den;
    cp[k * step] = c;
    s0[k * step] = d0;
    s1[k * step] = d1;
  }
  for (int k = n - 2; k >= 0; --k)
  {
    s0[k * step] -= cp[k * step] * s0[(k + 1) * step];
    s1[k * step] -= cp[k * step] * s1[(k + 1) * step];
  }
}

// ---- line in shared memory, one warp per line
//
// Bound: the latency of the FP64 recurrences (a 752x480 image has 480 rows
// and 752 columns of a few hundred dependent steps; its bytes take 10 us at
// the copy bandwidth).  A lane owns a segment of m = ceil(n / 32) samples and
// every recurrence of the Thomas algorithm runs as a segment composition, a
// warp scan and a walk of the segment: the pivots c' as 2x2 Moebius products
// (rescaled by powers of two every eight samples, so no factor omega or
// lambda overflows them), the two right-hand sides and the back substitution
// as affine maps, all in FP64.  The serial chain is 4 m steps instead of 2 n,
// and global memory is read and written along the rows (column pass: a
// stripe of up to four columns per block, one 32-byte sector per row) instead
// of one line per thread.  Measured (forward + backward, four launches, one
// thread per line before): 752x480 5.81 -> 0.089 ms, 160x128 1.23 -> 0.032 ms.
// Per line four double arrays of 32 segments with an odd pitch (8-byte
// accesses of consecutive lanes then fall on different bank pairs).
constexpr int kUpwTableBytes = 256 * (int)sizeof(double);

__host__ __device__ __forceinline__ int upw_seg(int n) { return (n + 31) / 32; }
__host__ __device__ __forceinline__ int upw_pitch(int n) { return upw_seg(n) | 1; }
__host__ __device__ __forceinline__ int upw_line_doubles(int n) { return 4 * 32 * upw_pitch(n); }

struct UpwLine
{
  double *w, *r0, *r1, *cp; // edge weights (k - 1, k), right-hand sides, c'
  int n, m, mp;
  unsigned m_inv; // ceil(2^32 / m): k / m = umulhi(k, m_inv), exact for k < 2^20
  __device__ __forceinline__ UpwLine(double *base, int n_) : n(n_)
  {
    m = upw_seg(n);
    mp = upw_pitch(n);
    m_inv = m == 1 ? 0u : 0xffffffffu / (unsigned)m + 1u;
    w = base;
    r0 = w + 32 * mp;
    r1 = r0 + 32 * mp;
    cp = r1 + 32 * mp;
  }
  __device__ __forceinline__ int pos(int k) const
  {
    const int l = m == 1 ? k : (int)__umulhi((unsigned)k, m_inv);
    return l * mp + (k - l * m);
  }
};

// largest entry scaled to [1, 2) by a power of two (exact); zero, subnormal,
// huge, infinite or NaN entries are left as they are
__device__ __forceinline__ void upw_renorm(double (&P)[4])
{
  const double mx = fmax(fmax(fabs(P[0]), fabs(P[1])), fmax(fabs(P[2]), fabs(P[3])));
  const int e = (__double2hiint(mx) >> 20) & 0x7ff;
  if (e == 0 || e >= 2046)
    return;
  const double s = __hiloint2double((2046 - e) << 20, 0);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    P[i] *= s;
}

// Solves (I + lam L_w) s = r for both right-hand sides of the line; the
// solutions replace r0 and r1, w and cp are scratch afterwards.  closing is
// the weight after the last sample.  Whole warp, the line already stored.
__device__ void upw_solve(const UpwLine &L, double lam, double closing)
{
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int s = min(lane * L.m, L.n), len = min(s + L.m, L.n) - s;
  double *w = L.w + lane * L.mp, *r0 = L.r0 + lane * L.mp, *r1 = L.r1 + lane * L.mp,
         *cp = L.cp + lane * L.mp;
  __syncwarp();
  // weight right of the segment's last sample: the next segment's first one
  const double wend = len == 0 ? 0.0 : s + len < L.n ? w[L.mp] : closing;
  __syncwarp(); // before the next lane overwrites it
  // pivots: c'_k = c_k / (b_k - a_k c'_{k-1}), [[P0 P1], [P2 P3]] the
  // segment's product
  double P[4] = {1.0, 0.0, 0.0, 1.0};
  double wl = len > 0 ? w[0] : 0.0;
  for (int j = 0; j < len; ++j)
  {
    const double wr = j + 1 < len ? w[j + 1] : wend;
    const double a = -lam * wl, c = -lam * wr, b = 1.0 + lam * (wl + wr);
    const double q2 = b * P[2] - a * P[0], q3 = b * P[3] - a * P[1];
    P[0] = c * P[2];
    P[1] = c * P[3];
    P[2] = q2;
    P[3] = q3;
    wl = wr;
    if ((j & 7) == 7)
      upw_renorm(P);
  }
  upw_renorm(P);
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    double Q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      Q[i] = __shfl_up_sync(full, P[i], off);
    if (lane >= off)
    {
      const double t[4] = {P[0] * Q[0] + P[1] * Q[2], P[0] * Q[1] + P[1] * Q[3],
                           P[2] * Q[0] + P[3] * Q[2], P[2] * Q[1] + P[3] * Q[3]};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        P[i] = t[i];
      upw_renorm(P);
    }
  }
  const double pb = __shfl_up_sync(full, P[1], 1), pd = __shfl_up_sync(full, P[3], 1);
  double c = lane == 0 ? 0.0 : pb / pd; // c' before the segment
  // c' of the segment; forward values d'_k = alpha_k d'_{k-1} + r_k / den_k
  // composed over the segment (alpha replaces w, r / den replaces r)
  double g = 1.0, h0 = 0.0, h1 = 0.0;
  wl = len > 0 ? w[0] : 0.0;
  for (int j = 0; j < len; ++j)
  {
    const double wr = j + 1 < len ? w[j + 1] : wend;
    const double a = -lam * wl;
    const double inv = 1.0 / (1.0 + lam * (wl + wr) - a * c);
    c = -lam * wr * inv;
    cp[j] = c;
    const double alpha = -a * inv, q0 = r0[j] * inv, q1 = r1[j] * inv;
    w[j] = alpha;
    r0[j] = q0;
    r1[j] = q1;
    g *= alpha;
    h0 = alpha * h0 + q0;
    h1 = alpha * h1 + q1;
    wl = wr;
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    const double og = __shfl_up_sync(full, g, off), o0 = __shfl_up_sync(full, h0, off),
                 o1 = __shfl_up_sync(full, h1, off);
    if (lane >= off)
    {
      h0 += g * o0;
      h1 += g * o1;
      g *= og;
    }
  }
  double d0 = __shfl_up_sync(full, h0, 1), d1 = __shfl_up_sync(full, h1, 1);
  if (lane == 0)
    d0 = d1 = 0.0;
  // forward values; back substitution s_k = d'_k - c'_k s_{k+1} composed
  g = 1.0;
  h0 = h1 = 0.0;
  for (int j = 0; j < len; ++j)
  {
    d0 = w[j] * d0 + r0[j];
    d1 = w[j] * d1 + r1[j];
    r0[j] = d0;
    r1[j] = d1;
    h0 += g * d0;
    h1 += g * d1;
    g *= -cp[j];
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    const double og = __shfl_down_sync(full, g, off), o0 = __shfl_down_sync(full, h0, off),
                 o1 = __shfl_down_sync(full, h1, off);
    if (lane + off < 32)
    {
      h0 += g * o0;
      h1 += g * o1;
      g *= og;
    }
  }
  double z0 = __shfl_down_sync(full, h0, 1), z1 = __shfl_down_sync(full, h1, 1);
  if (lane == 31)
    z0 = z1 = 0.0;
  for (int j = len - 1; j >= 0; --j)
  {
    z0 = r0[j] - cp[j] * z0;
    z1 = r1[j] - cp[j] * z1;
    r0[j] = z0;
    r1[j] = z1;
  }
  __syncwarp();
}

extern __shared__ __align__(16) unsigned char g_upw_smem[];

// exp(-d^2 / sigma) for every intensity difference (the per-edge expression,
// so the values are the per-edge ones); whole block
__device__ __forceinline__ double *upw_table(double sigma)
{
  double *tab = reinterpret_cast<double *>(g_upw_smem);
  for (int t = threadIdx.x; t < 256; t += blockDim.x)
    tab[t] = edge_exp((double)t, 0.0, sigma);
  __syncthreads();
  return tab;
}
__device__ __forceinline__ double *upw_line_base(int i, int n)
{
  return reinterpret_cast<double *>(g_upw_smem + kUpwTableBytes) + (size_t)i * upw_line_doubles(n);
}

// row pass, one row per warp
template <bool BWD>
__global__ void __launch_bounds__(64) k_upw_rows(const DiffUp u)
{
  const double *tab = upw_table(u.sigma);
  after_previous();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int y = blockIdx.x * (int)(blockDim.x >> 5) + warp, n = u.W;
  if (y >= u.H)
    return;
  const UpwLine L(upw_line_base(warp, n), n);
  const uint8_t *img = u.img + (size_t)y * u.pitch;
  const size_t o = (size_t)y * n;
#pragma unroll 4
  for (int k = lane; k < n; k += 32)
  {
    const int p = L.pos(k);
    L.w[p] =
        k > 0 ? (double)u.omega[o + k] * tab[abs((int)img[k] - (int)img[k - 1])] : 0.0;
    if (BWD)
    {
      L.r0[p] = u.ud[o + k];
      L.r1[p] = u.ui[o + k];
    }
    else
    {
      const double d = u.sparse[o + k];
      L.r0[p] = d;
      L.r1[p] = d > 0.0 ? 1.0 : 0.0;
    }
  }
  upw_solve(L, u.lam, u.row_closing);
#pragma unroll 4
  for (int k = lane; k < n; k += 32)
  {
    const int p = L.pos(k);
    const size_t q = o + k;
    if (!BWD)
    {
      u.sd[q] = L.r0[p];
      u.si[q] = L.r1[p];
      continue;
    }
    u.g_sparse[q] = (float)L.r0[p];
    if (k == 0)
      continue;
    const int p1 = L.pos(k - 1);
    const double gw = -u.lam * ((L.r0[p] - L.r0[p1]) * (u.sd[q] - u.sd[q - 1]) +
                                (L.r1[p] - L.r1[p1]) * (u.si[q] - u.si[q - 1]));
    u.g_omega[q] += (float)(gw * tab[abs((int)img[k] - (int)img[k - 1])]);
  }
}

// column pass, a stripe of blockDim.x / 32 columns per block, loaded and
// stored row by row by the whole block (thread t: column t % C, rows t / C +
// 32 j)
template <bool BWD>
__global__ void __launch_bounds__(128) k_upw_cols(const DiffUp u)
{
  const double *tab = upw_table(u.sigma);
  after_previous();
  const int C = blockDim.x >> 5, n = u.H;
  const int kt = (int)threadIdx.x / C, ct = (int)threadIdx.x - kt * C;
  const int xt = blockIdx.x * C + ct;
  const size_t W = u.W;
  const UpwLine Lt(upw_line_base(ct, n), n);
  if (xt < u.W)
  {
#pragma unroll 4
    for (int k = kt; k < n; k += 32)
    {
      const int p = Lt.pos(k);
      const size_t o = (size_t)k * W + xt;
      const uint8_t *i = u.img + (size_t)k * u.pitch + xt;
      Lt.w[p] = k > 0 ? (double)u.omega[o] * tab[abs((int)i[0] - (int)*(i - u.pitch))] : 0.0;
      if (BWD)
      {
        const double g = u.g_dense[o], ti = u.ti[o];
        Lt.r0[p] = g / ti;
        Lt.r1[p] = -g * u.td[o] / (ti * ti);
      }
      else
      {
        Lt.r0[p] = u.sd[o];
        Lt.r1[p] = u.si[o];
      }
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  if (blockIdx.x * C + warp < u.W)
    upw_solve(UpwLine(upw_line_base(warp, n), n), u.lam, u.col_closing);
  __syncthreads();
  if (xt >= u.W)
    return;
#pragma unroll 4
  for (int k = kt; k < n; k += 32)
  {
    const int p = Lt.pos(k);
    const size_t o = (size_t)k * W + xt;
    const double s0 = Lt.r0[p], s1 = Lt.r1[p];
    if (!BWD)
    {
      u.td[o] = s0;
      u.ti[o] = s1;
      u.dense[o] = (float)(s0 / s1);
      continue;
    }
    u.ud[o] = s0;
    u.ui[o] = s1;
    if (k == 0)
    {
      u.g_omega[o] = 0.0f;
      continue;
    }
    const int p1 = Lt.pos(k - 1);
    const uint8_t *i = u.img + (size_t)k * u.pitch + xt;
    const double gw = -u.lam * ((s0 - Lt.r0[p1]) * (u.td[o] - u.td[o - W]) +
                                (s1 - Lt.r1[p1]) * (u.ti[o] - u.ti[o - W]));
    u.g_omega[o] = (float)(gw * tab[abs((int)i[0] - (int)*(i - u.pitch))]);
  }
}

// ---- lines longer than shared memory holds (above about 7200 samples): one
// thread per line over global memory
// row pass: one thread per row
__global__ void k_upw_rows_fwd(DiffUp u)
{
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  if (y >= u.H)
    return;
  const size_t o = (size_t)y * u.W;
  LineW L{u.img + (size_t)y * u.pitch, 1, u.omega + o, 1, u.W, u.row_closing, u.sigma};
  for (int x = 0; x < u.W; ++x)
  {
    const double d = u.sparse[o + x];
    u.sd[o + x] = d;
    u.si[o + x] = d > 0.0 ? 1.0 : 0.0;
  }
  thomas2(L, u.lam, u.sd + o, u.si + o, u.sd + o, u.si + o, u.cp + o, 1);
}

// column pass: one thread per column (coalesced across threads)
__global__ void k_upw_cols_fwd(DiffUp u)
{
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= u.W)
    return;
  LineW L{u.img + x, u.pitch, u.omega + x, (size_t)u.W, u.H, u.col_closing, u.sigma};
  thomas2(L, u.lam, u.sd + x, u.si + x, u.td + x, u.ti + x, u.cp + x, (size_t)u.W);
  for (int y = 0; y < u.H; ++y)
  {
    const size_t o = (size_t)y * u.W + x;
    u.dense[o] = (float)(u.td[o] / u.ti[o]);
  }
}

// column adjoint: u = B^-1 g_t, g_omega from the column edges
__global__ void k_upw_cols_bwd(DiffUp u)
{
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= u.W)
    return;
  const size_t W = u.W;
  for (int y = 0; y < u.H; ++y)
  {
    const size_t o = (size_t)y * W + x;
    const double g = u.g_dense[o], ti = u.ti[o];
    u.ud[o] = g / ti;
    u.ui[o] = -g * u.td[o] / (ti * ti);
  }
  LineW L{u.img + x, u.pitch, u.omega + x, W, u.H, u.col_closing, u.sigma};
  thomas2(L, u.lam, u.ud + x, u.ui + x, u.ud + x, u.ui + x, u.cp + x, W);
  for (int y = 1; y < u.H; ++y)
  {
    const size_t o = (size_t)y * W + x, p = o - W;
    double e = 0.0;
    L.w(y, &e);
    const double gw = -u.lam * ((u.ud[o] - u.ud[p]) * (u.td[o] - u.td[p]) +
                                (u.ui[o] - u.ui[p]) * (u.ti[o] - u.ti[p]));
    u.g_omega[o] = (float)(gw * e);
  }
  u.g_omega[x] = 0.0f;
}

// row adjoint: v = A^-1 u, g_sparse = v_d, g_omega += row edges
__global__ void k_upw_rows_bwd(DiffUp u)
{
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  if (y >= u.H)
    return;
  const size_t o = (size_t)y * u.W;
  LineW L{u.img + (size_t)y * u.pitch, 1, u.omega + o, 1, u.W, u.row_closing, u.sigma};
  thomas2(L, u.lam, u.ud + o, u.ui + o, u.ud + o, u.ui + o, u.cp + o, 1);
  for (int x = 0; x < u.W; ++x)
  {
    u.g_sparse[o + x] = (float)u.ud[o + x];
    if (x == 0)
      continue;
    double e = 0.0;
    L.w(x, &e);
    const size_t q = o + x, p = q - 1;
    const double gw = -u.lam * ((u.ud[q] - u.ud[p]) * (u.sd[q] - u.sd[p]) +
                                (u.ui[q] - u.ui[p]) * (u.si[q] - u.si[p]));
    u.g_omega[q] += (float)(gw * e);
  }
}

// ------------------------------------------------------------ fusion adjoint
struct Dual
{
  double v, g;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.g + b.g}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.g - b.g}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b)
{
  return {a.v * b.v, a.g * b.v + a.v * b.g};
}
__device__ __forceinline__ Dual operator/(Dual a, Dual b)
{
  const double q = a.v / b.v;
  return {q, (a.g - q * b.g) / b.v};
}
__device__ __forceinline__ Dual cst(double v) { return {v, 0.0}; }
__device__ __forceinline__ Dual dexp(Dual a)
{
  const double e = exp(a.v);
  return {e, e * a.g};
}
__device__ __forceinline__ Dual dsqrt(Dual a)
{
  const double s = sqrt(a.v);
  return {s, a.g / (2.0 * s)};
}

// d(fused depth)/d(upsampled depth) times the incoming gradient, with the
// prior of the pixel (table and transformed seeds of the forward fusion)
__global__ void __launch_bounds__(256) k_fuse_bwd(DiffFuse f)
{
  after_previous();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)f.W * f.H)
    return;
  const Dual dep{(double)f.depth_in[idx], 1.0};
  Dual unc = dep.v * 0.2 > 0.5 ? dep * cst(0.2) : cst(0.5);
  unc = unc * unc;
  if (dep.v <= 0.0)
    unc = cst(1e9);
  const int pre = f.table[idx];
  Dual a = cst(10.0), b = cst(10.0), mu = dep, s2 = cst(2500.0);
  if (pre > 0)
  {
    const float4 s = f.seeds_in[pre];
    a = cst(s.x);
    b = cst(s.y);
    mu = cst(s.z);
    s2 = cst(s.w);
  }
  if (((dep - mu) * (dep - mu)).v > (unc + s2).v)
  {
    a = cst(10.0);
    b = cst(10.0);
    mu = dep;
    s2 = cst(2500.0);
  }
  const Dual var = unc + s2;
  const Dual new_mu = (dep * s2 + mu * unc) / var;
  const Dual dm = dep - mu;
  const Dual pdf = dexp(cst(0.0) - dm * dm / (cst(2.0) * var)) / dsqrt(cst(2.0 * M_PI) * var);
  const double ratio = a.v / (a.v + b.v);
  Dual c1 = cst(ratio) * pdf;
  Dual c2 = cst(b.v / (a.v + b.v) / 50.0);
  const Dual norm = c1 + c2;
  c1 = c1 / norm;
  c2 = c2 / norm;
  const Dual mu_p = c1 * new_mu + c2 * mu;
  f.g_depth[idx] = ratio > 0.60 ? (float)(mu_p.g * (double)f.g_fused[idx]) : 0.0f;
}

template <int D, class R>
void readout_d(const DiffBpR<R> &a, int backward, cudaStream_t s)
{
  const int cells = a.w * a.h;
  launch_kernel(k_soft_readout<D, R>, (cells + kDiffWarps - 1) / kDiffWarps, kDiffWarps * 32, 0, s,
                1, a, backward);
}

template <int D, class R>
void bwd_d(const DiffBpR<R> &a, cudaStream_t s)
{
  const int items = ((a.w + 1) / 2) * a.h;
  launch_kernel(k_bp_sweep_bwd<D, R>, (items + kDiffWarps - 1) / kDiffWarps, kDiffWarps * 32, 0, s,
                1, a);
}

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

void launch_soft_readout(const DiffBp &a, int backward, cudaStream_t s)
{
  by_d(a.D, [&](auto dc) { readout_d<decltype(dc)::value>(a, backward, s); });
}

void launch_soft_readout(const DiffBp64 &a, int backward, cudaStream_t s)
{
  by_d(a.D, [&](auto dc) { readout_d<decltype(dc)::value>(a, backward, s); });
}

void launch_bp_sweep_bwd(const DiffBp &a, cudaStream_t s)
{
  by_d(a.D, [&](auto dc) { bwd_d<decltype(dc)::value>(a, s); });
}

void launch_bp_sweep_bwd(const DiffBp64 &a, cudaStream_t s)
{
  by_d(a.D, [&](auto dc) { bwd_d<decltype(dc)::value>(a, s); });
}

namespace
{
template <class R>
void downsample(const DiffBpR<R> &a, const MsgPtrsR<R> &parent, int pw, int ph, cudaStream_t s)
{
  const long n = (long)pw * ph * a.D;
  if (n > 0)
    launch_kernel(k_msg_downsample<R>, (unsigned)((n + 255) / 256), 256, 0, s, 1, a, parent, pw,
                  ph);
}
} // namespace

void launch_msg_downsample(const DiffBp &a, const MsgPtrs &parent, int pw, int ph, cudaStream_t s)
{
  downsample(a, parent, pw, ph, s);
}

void launch_msg_downsample(const DiffBp64 &a, const MsgPtrs64 &parent, int pw, int ph,
                           cudaStream_t s)
{
  downsample(a, parent, pw, ph, s);
}

void launch_widen(const float *in, double *out, long n, cudaStream_t s)
{
  if (n > 0)
    k_widen<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, out, n);
}

void launch_pyramid64(const double *fine, int fw, int fh, double *coarse, int cw, int ch, int D,
                      cudaStream_t s)
{
  const long n = (long)cw * ch * D;
  if (n > 0)
    k_pyramid64<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(fine, fw, fh, coarse, cw, ch, D);
}

void launch_msg_inherit_all64(const MsgPtrs64 *parent, int pw, const MsgPtrs64 &child, int cw,
                              int ch, int D, cudaStream_t s)
{
  const long n = (long)cw * ch * D;
  MsgPtrs64 none{};
  if (n > 0)
    k_msg_inherit_all64<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        parent ? *parent : none, parent ? 1 : 0, pw, child, cw, ch, D);
}

void launch_bp_sweep_fwd64(const DiffBp64 &a, const MsgPtrs64 &M, cudaStream_t s)
{
  const int items = ((a.w + 1) / 2) * a.h;
  by_d(a.D, [&](auto dc) {
    k_bp_sweep_fwd64<decltype(dc)::value>
        <<<(items + kDiffWarps - 1) / kDiffWarps, kDiffWarps * 32, 0, s>>>(a, M);
  });
}

namespace
{
// lines of n samples per block: at most `most`, as many as shared memory
// holds; 0 when not even one fits
int upw_lines(int n, int most)
{
  const int line = upw_line_doubles(n) * (int)sizeof(double);
  int c = most;
  while (c > 0 && kUpwTableBytes + c * line > kMaxBlockSmem)
    c >>= 1;
  return c;
}

// more than 48 KB of dynamic shared memory is an opt-in per device
std::atomic<unsigned long long> g_upw_prepared{0};
void upw_prepare()
{
  int dev = 0;
  const bool known = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
  const unsigned long long bit = known ? 1ull << dev : 0ull;
  if (known && (g_upw_prepared.load(std::memory_order_acquire) & bit))
    return;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaFuncSetAttribute(k_upw_rows<false>, attr, kMaxBlockSmem);
  cudaFuncSetAttribute(k_upw_rows<true>, attr, kMaxBlockSmem);
  cudaFuncSetAttribute(k_upw_cols<false>, attr, kMaxBlockSmem);
  cudaFuncSetAttribute(k_upw_cols<true>, attr, kMaxBlockSmem);
  g_upw_prepared.fetch_or(bit, std::memory_order_acq_rel);
}

template <bool BWD>
void upw_rows(const DiffUp &u, cudaStream_t s)
{
  const int c = upw_lines(u.W, 2);
  if (c > 0)
    launch_kernel(k_upw_rows<BWD>, (u.H + c - 1) / c, 32 * c,
                  kUpwTableBytes + c * upw_line_doubles(u.W) * sizeof(double), s, 1, u);
  else if (BWD)
    k_upw_rows_bwd<<<(u.H + 63) / 64, 64, 0, s>>>(u);
  else
    k_upw_rows_fwd<<<(u.H + 63) / 64, 64, 0, s>>>(u);
}

template <bool BWD>
void upw_cols(const DiffUp &u, cudaStream_t s)
{
  const int c = upw_lines(u.H, 4);
  if (c > 0)
    launch_kernel(k_upw_cols<BWD>, (u.W + c - 1) / c, 32 * c,
                  kUpwTableBytes + c * upw_line_doubles(u.H) * sizeof(double), s, 1, u);
  else if (BWD)
    k_upw_cols_bwd<<<(u.W + 63) / 64, 64, 0, s>>>(u);
  else
    k_upw_cols_fwd<<<(u.W + 63) / 64, 64, 0, s>>>(u);
}
} // namespace

void launch_upw_forward(const DiffUp &u, cudaStream_t s)
{
  upw_prepare();
  upw_rows<false>(u, s);
  upw_cols<false>(u, s);
}

void launch_upw_backward(const DiffUp &u, cudaStream_t s)
{
  upw_prepare();
  upw_cols<true>(u, s);
  upw_rows<true>(u, s);
}

void launch_fuse_bwd(const DiffFuse &f, cudaStream_t s)
{
  const long n = (long)f.W * f.H;
  if (n > 0)
    launch_kernel(k_fuse_bwd, (unsigned)((n + 255) / 256), 256, 0, s, 1, f);
}

} // namespace qm
