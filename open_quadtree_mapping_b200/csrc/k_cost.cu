// Multi-view matching cost at quadtree nodes (image_to_cost +
// normalize_the_cost, depth_extract.cu:135-244 of the reference).
//
// A block owns a tile of kCostCells consecutive cells of one cell row (or its
// share of the tile's hypotheses).  Warp
// 0 finds the tile's node cells (ballot) and stages, per node, its ray and
// 3x3 reference patch in shared memory; the block also stages the slot poses
// and the hypothesis depths.  Thread t then owns node t % n (n nodes in the
// tile) and every (256 / n)-th hypothesis from t / n on, so the lanes of a
// warp evaluate neighbouring nodes at one depth: their projections are
// neighbours in the slot image and a gather touches few cache lines; the
// node's ray and patch stay in registers.  Each pair loops over the
// measurement slots and accumulates the 3x3 SAD as an integer: every term is
// an integer intensity difference, so the sum is exact and equal to the
// reference's shared-memory tree over slots.  The projection follows the
// reference's arithmetic (ArithRef) or IEEE rounding (ArithIeee).  The tile's
// costs are assembled in shared memory and written as one contiguous run.
//
// Cells that are not node origins, or touch the border (x <= 0, y <= 0,
// x >= W-1, y >= H-1), get cost 0 for every hypothesis, as the reference's
// zeroed cost image does.  A node with no valid slot gets 100.  Every node
// cost is then divided by the cell's writer count, which in the reference is
// the number of hypotheses: each hypothesis thread of slot row 0 adds 1 to it
// (depth_extract.cu:219-228), and normalize_the_cost divides by it
// (depth_extract.cu:231-244).
//
// Bytes per cell: 9 reference pixels + D*F*9 measurement gathers (u8, mostly
// L1/L2 hits along the epipolar segment) + 4*D written.
#include "launch.h"

namespace qm
{

namespace
{

// Packed pairs (x, y) of floats: one instruction for both coordinates.
typedef unsigned long long F2;
__device__ __forceinline__ F2 pack2(float x, float y)
{
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(F2 v, float &x, float &y)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
  F2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b)
{
  F2 r;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// floor(c + 0.5) for -0.5 <= c < 2^23 - 0.5, which equals the reference's
// (int)((double)c + 0.5) there, in one rounded operation: 2^23 + 0.5 is not
// a float, but it is the exact product 24929 * 336.5 (24929 = 97 * 257,
// 336.5 = 673 / 2), so a fused multiply-add rounded down evaluates
// RD(2^23 + 0.5 + c) with a single rounding.  That sum lies in [2^23, 2^24),
// where floats are spaced 1 apart, so the result is 2^23 + floor(c + 0.5)
// exactly, and its bit pattern minus kBias = bits(2^23) is the integer; kBias
// is subtracted (folded into the image offset) by the caller.
__device__ __forceinline__ F2 round2(F2 c)
{
  F2 r;
  asm("fma.rm.ftz.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(pack2(24929.0f, 24929.0f)), "l"(pack2(336.5f, 336.5f)), "l"(c));
  return r;
}
constexpr unsigned kBias = 0x4B000000u;
__device__ __forceinline__ unsigned offset_of(F2 r, unsigned pitch, unsigned bias)
{
  // y * pitch + x in 32-bit wrap-around arithmetic (the true offset is below
  // 2^31)
  const unsigned hx = (unsigned)r, hy = (unsigned)(r >> 32);
  return hy * pitch + hx + bias;
}

// SAD of three bytes packed in a word each, plus s
__device__ __forceinline__ unsigned sad3(unsigned a, unsigned b, unsigned s)
{
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %0;" : "+r"(s) : "r"(a), "r"(b));
  return s;
}

// The 3x3 SAD at (u, v), every pixel at its own rounded position.  The
// reference computes (u + a*i) + b*j for i, j in {-1, 0, 1} (i the patch
// column, j the row).  The products are exact (a*(+-1) = +-a, a*0 = +-0, and
// c +- 0 = c), so in both arithmetic modes the nine values are these correctly
// rounded sums: three column bases, then three rows each.  row[j]: the
// reference patch's row, three bytes.
// The slot poses are validated as rigid on the host (|r00|+|r01| and
// |r10|+|r11| <= 1.5), so every patch coordinate + 0.5 lies in [0.5, W-0.5) x
// [0.5, H-0.5): no clamp needed.
__device__ __forceinline__ unsigned patch_sad(const uint8_t *m, unsigned pitch, unsigned bias,
                                              F2 uv, F2 a, F2 b, const unsigned (&row)[3])
{
  const F2 col[3] = {sub2(uv, a), uv, add2(uv, a)};
  unsigned s = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
  {
    unsigned px[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
      const F2 c = j == 0 ? sub2(col[i], b) : j == 1 ? col[i] : add2(col[i], b);
      px[i] = __ldg(m + offset_of(round2(c), pitch, bias));
    }
    s = sad3(px[0] | (px[1] << 8) | (px[2] << 16), row[j], s);
  }
  return s;
}

// A slot whose rotation barely turns the patch: at most places the nine rounded
// positions are the 3x3 pixels around the rounded centre.  They certainly are
// when the centre lies within `margin` of its pixel's centre in x and y:
// position (i, j) is off the grid by the centre's own offset plus at most
// |a - 1| + |b| (x; |c| + |d - 1| in y), plus two roundings of at most half an
// ulp each.
struct __align__(16) SlotParam
{
  const uint8_t *img;
  float margin;
  unsigned weight;
};

// Hypotheses [lo, hi] (real numbers of the line 0 .. last, lo > hi: none) outside
// of which a node's projection into a slot is certainly not in view.  With inverse
// depth w the projected point is, up to scale, q(w) = R ray + t w, and in view
// means (q_x / q_z, q_y / q_z) within four bounds: four linear forms in w that
// are all >= 0 where q_z > 0, or all <= 0 where q_z < 0 (the projection does not
// ask on which side of the camera the point lies).  Every form is widened by
// kViewSlack of the sum of its terms' magnitudes (the rays are unit vectors), far
// above what float rounding moves the compared coordinates by in either arithmetic
// (a dozen roundings, 1e-6); a bound that comes out NaN does not narrow anything.
constexpr float kViewSlack = 1e-5f;
__device__ __forceinline__ void view_range(const float4 &t0, const float4 &t1, const float4 &t2,
                                           const float3 &ray, const Cam &cam, float W, float H,
                                           float w0, float dw, float last, int &first, int &end)
{
  const float ax = t0.x * ray.x + t0.y * ray.y + t0.z * ray.z;
  const float ay = t1.x * ray.x + t1.y * ray.y + t1.z * ray.z;
  const float az = t2.x * ray.x + t2.y * ray.y + t2.z * ray.z;
  const float w_max = fmaxf(fabsf(w0), fabsf(w0 + dw * last));
  const float slack = kViewSlack *
                      (fabsf(cam.fx) + fabsf(cam.fy) + fabsf(cam.cx) + fabsf(cam.cy) +
                       2.0f * (W + H)) *
                      (fabsf(t0.x) + fabsf(t0.y) + fabsf(t0.z) + fabsf(t1.x) + fabsf(t1.y) +
                       fabsf(t1.z) + fabsf(t2.x) + fabsf(t2.y) + fabsf(t2.z) +
                       (fabsf(t0.w) + fabsf(t1.w) + fabsf(t2.w)) * w_max);
  float lo[2] = {0.0f, 0.0f}, hi[2] = {last, last};
  // the form p + q w >= 0, and <= 0 for the points behind the camera
  auto form = [&](float p, float q) {
    const float a = p + q * w0, b = q * dw; // in the hypothesis index
    const float inv = __fdividef(1.0f, b);
#pragma unroll
    for (int side = 0; side < 2; ++side)
    {
      const float c = (side ? -a : a) + slack, m = side ? -b : b;
      const float at = (side ? c : -c) * inv;
      if (m > 0.0f)
        lo[side] = fmaxf(lo[side], at);
      else if (m < 0.0f)
        hi[side] = fminf(hi[side], at);
      else if (c < 0.0f)
        hi[side] = -1e9f;
    }
  };
  auto axis = [&](float f, float c, float size, float p, float q) {
    const float below = c - 1.25f, above = size - 2.25f - c; // a quarter pixel wide of the bounds
    form(f * p + below * az, f * q + below * t2.w);
    form(above * az - f * p, above * t2.w - f * q);
  };
  axis(cam.fx, cam.cx, W, ax, t0.w);
  axis(cam.fy, cam.cy, H, ay, t1.w);
  // a hypothesis to either side for the rounding of the bounds themselves
  first = 1 << 20;
  end = -1;
#pragma unroll
  for (int side = 0; side < 2; ++side)
    if (!(lo[side] > hi[side] + 2.0f))
    {
      first = min(first, (int)floorf(fminf(lo[side], 1e6f)) - 1);
      end = max(end, (int)ceilf(fminf(hi[side], 1e6f)) + 1);
    }
}

// Share of the centres that must lie within the margin, else the slot's patches
// are taken pixel by pixel at once: a deferred patch costs about 1.3 of those and
// an aligned one 0.7, so the list pays up to about a quarter.  (Frames up to 18
// steps of 1.7 degrees apart: 0.9 and more at nine of ten.)
constexpr float kMinAligned = 0.8f;
constexpr int kCostWarps = kFlatThreads / 32;

// MINB resident blocks of 256 threads per SM (at most 48, 64 or 80
// registers for 5, 4 or 3): more resident warps against fewer spilled
// values.  The balance depends on the hypothesis and slot counts, so the
// engine's autotuner picks it per stream set.
//
// Bound: instruction issue (71 to 75 % busy; with nine byte gathers per node,
// hypothesis and slot it was 133 instructions each, and L1 80 % busy).  Where
// the patch is aligned (SlotParam) its three rows come as two aligned words each
// and three byte-wise SADs, from one address; coordinates are packed pairs, and
// two hypotheses share a slot's parameters: about 100 instructions.  A patch
// that is not aligned, in a slot where most are, would hold up its warp: its
// position goes to the warp's list, and the list is worked off 32 at a time,
// every lane busy.  Slots that turn further take every pixel at its own
// position.  The sums are integers, so all ways give the same.  Measured, nine
// gathers for every patch before, on views of which all patches are aligned (the
// scenes of perf/cases.py): 32 x 752x480 x 64, 5 slots 0.838 -> 0.724 ms, 8 x
// 1920x1080 x 128, 20 slots 4.93 -> 4.36, one 1280x720, 10 slots 0.144 -> 0.123,
// one 1920x1080 x 128, 18 slots 0.870 -> 0.689.  The gain is the scene's: on
// bench.py's views, which turn by 1 to 2 degrees a frame (94 to 97 % aligned), the
// first is 0.881 -> 0.842 in eager launches, where the others' is 0.900 -> 0.752.
// WORDS: the slot images' rows all start on a word, so that a patch's rows are
// offset alike.  VIEW: the hypotheses out of a slot's view are found first
// (kViewWork).
template <class A, int MINB, bool WORDS, bool VIEW>
__global__ void __launch_bounds__(kFlatThreads, MINB)
    k_cost(const __grid_constant__ Batch B, int split)
{
  after_previous();
  // sum of absolute differences (low 20 bits: at most 32 slots * 9 * 255) and
  // number of valid slots of the tile, [kCostCells][D + 1] (the padding keeps
  // lanes that add to one hypothesis of different cells on different banks)
  extern __shared__ unsigned s_acc[];
  __shared__ float4 s_pose[kMaxSlots * 3];
  __shared__ SlotParam s_slot[kMaxSlots];
  __shared__ float s_depth[kMaxHyp];
  // node cells of the tile, in x order: tile column, ray, rows of the 3x3 patch
  __shared__ int s_col[kCostCells];
  __shared__ float s_dir[3][kCostCells];
  __shared__ unsigned s_row[3][kCostCells];
  __shared__ unsigned s_nodes;
  __shared__ int s_fast;
  // hypotheses at which any node of the tile may be in view of a slot, and per
  // hypothesis the slots
  __shared__ int2 s_range[VIEW ? kMaxSlots : 1];
  __shared__ unsigned s_view[VIEW ? kMaxHyp : 1];
  // per warp: patches to be taken pixel by pixel (position; node, hypothesis
  // and slot)
  __shared__ float4 s_late[kCostWarps][96];
  int lb;
  const JobDesc &J = job_of(B, lb);
  // the block's share of the tile's hypotheses: [h0, h0 + D)
  const int all_d = J.D, D = all_d / split, h0 = (lb % split) * D;
  lb /= split;
  const int F = J.F, W = J.W, H = J.H;
  const int segs = (J.cw + kCostCells - 1) / kCostCells;
  const int cy = lb / segs, cx0 = (lb - cy * segs) * kCostCells;
  const int ncells = min(kCostCells, J.cw - cx0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned pitch = (unsigned)J.slot_pitch;
  // the job's (deduplicated) slots, those with aligned patches first, and the
  // hypothesis depths, once per block
  if (warp == kCostWarps - 1)
  {
    const bool in = lane < F; // F <= kMaxSlots = 32
    const float *T = slot_pose(B, J.slot_base + (in ? lane : 0));
    const uint8_t *img = slot_image(B, J.slot_base + (in ? lane : 0));
    const float eps = (float)max(W, H) * 0x1p-22f + 0x1p-20f;
    const float margin =
        0.5f - eps -
        fmaxf(fabsf(T[0] - 1.0f) + fabsf(T[1]), fabsf(T[4]) + fabsf(T[5] - 1.0f));
    const bool fast = in && margin > 0.0f && 4.0f * margin * margin >= kMinAligned;
    const unsigned m = __ballot_sync(0xffffffffu, fast), below = (1u << lane) - 1u;
    if (in)
    {
      const int at = fast ? __popc(m & below) : __popc(m) + __popc(~m & below);
      s_slot[at] = SlotParam{img, margin, (unsigned)slot_weight(B, J.slot_base + lane)};
#pragma unroll
      for (int r = 0; r < 3; ++r)
        s_pose[3 * at + r] = make_float4(T[4 * r], T[4 * r + 1], T[4 * r + 2], T[4 * r + 3]);
    }
    if (lane == 0)
      s_fast = __popc(m);
  }
  for (int d = tid; d < D; d += blockDim.x)
    s_depth[d] = A::hyp_depth(J.step, J.min_inv, h0 + d);
  const int sd = D + 1;
  for (int i = tid; i < ncells * sd; i += blockDim.x)
    s_acc[i] = 0u;
  const Cam cam{J.fx, J.fy, J.cx, J.cy};
  if (tid < 32)
  {
    // node test of cell cx0 + tid: quadtree node origin away from the border
    const int x = (cx0 + tid) * 4, y = cy * 4;
    bool node = false;
    if (tid < ncells && x > 0 && y > 0 && x < W - 1 && y < H - 1)
    {
      const int size = 1 << J.levels[(size_t)y * W + x];
      node = x % size == 0 && y % size == 0;
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, node);
    if (node)
    {
      const int k = __popc(ballot & ((1u << tid) - 1u));
      s_col[k] = tid;
      const float3 dir = A::ray((float)x, (float)y, cam);
      s_dir[0][k] = dir.x;
      s_dir[1][k] = dir.y;
      s_dir[2][k] = dir.z;
      const uint8_t *r = J.ref + (size_t)(y - 1) * J.ref_pitch + (x - 1);
#pragma unroll
      for (int jj = 0; jj < 3; ++jj)
      {
        const uint8_t *q = r + (size_t)jj * J.ref_pitch;
        s_row[jj][k] = (unsigned)__ldg(q) | ((unsigned)__ldg(q + 1) << 8) |
                       ((unsigned)__ldg(q + 2) << 16);
      }
    }
    if (tid == 0)
      s_nodes = ballot;
  }
  __syncthreads();
  const unsigned nodes = s_nodes;
  const int n = __popc(nodes);
  // (int)(u + 0.5) in [2, W-2) exactly when u in [1.5, W-2.5) (both bounds
  // are floats, the comparisons exact; NaN fails)
  const float ulo = 1.5f, uhi = (float)W - 2.5f, vhi = (float)H - 2.5f;
  const unsigned bias = 0u - kBias * (pitch + 1u);
  if constexpr (VIEW)
  {
    for (int f = warp; f < F; f += kCostWarps)
    {
      const int k = min(lane, n - 1);
      int first = 1 << 20, end = -1;
      if (n > 0)
        view_range(s_pose[3 * f], s_pose[3 * f + 1], s_pose[3 * f + 2],
                   make_float3(s_dir[0][k], s_dir[1][k], s_dir[2][k]), cam, (float)W, (float)H,
                   (float)J.min_inv, (float)J.step, (float)(all_d - 1), first, end);
      first = __reduce_min_sync(0xffffffffu, first);
      end = __reduce_max_sync(0xffffffffu, end);
      if (lane == 0)
        s_range[f] = make_int2(first, end);
    }
    __syncthreads();
    for (int d = tid; d < D; d += blockDim.x)
    {
      unsigned m = 0;
      for (int f = 0; f < F; ++f)
      {
        const int2 r = s_range[f];
        m |= (h0 + d >= r.x && h0 + d <= r.y ? 1u : 0u) << f;
      }
      s_view[d] = m;
    }
    __syncthreads();
  }
  // Thread t evaluates node k = t % n at hypotheses g, g + per, g + 2 per,
  // ... (g = t / n, per = threads per node): consecutive lanes hold
  // neighbouring nodes at one depth, whose projections are neighbours in the
  // slot images.  The node's ray and 3x3 patch stay in registers across the
  // thread's hypotheses and slots.  All lanes of a warp walk the loops
  // together (the lists are the warp's).
  const int per = n > 0 ? (int)blockDim.x / n : 0;
  if (n > 0 && warp * 32 < min(per, D) * n)
  {
    const bool mine = tid < per * n;
    const int k = tid % n, g = tid / n;
    const float3 dir = make_float3(s_dir[0][k], s_dir[1][k], s_dir[2][k]);
    const unsigned row[3] = {s_row[0][k], s_row[1][k], s_row[2][k]};
    const int col = s_col[k] * sd;
    int late = 0; // entries of the warp's list
    // takes the last `cnt` (<= 32) entries of the list
    auto work_off = [&](int cnt) {
      __syncwarp();
      late -= cnt;
      if (lane < cnt)
      {
        const float4 e = s_late[warp][late + lane];
        const F2 uv = pack2(e.x, e.y);
        const unsigned id = __float_as_uint(e.z);
        const int f = id & 0xffu, kk = (id >> 8) & 0xffu, d = id >> 16;
        const float4 t0 = s_pose[3 * f], t1 = s_pose[3 * f + 1];
        const unsigned r[3] = {s_row[0][kk], s_row[1][kk], s_row[2][kk]};
        const unsigned s = patch_sad(s_slot[f].img, pitch, bias, uv, pack2(t0.x, t1.x),
                                     pack2(t0.y, t1.y), r);
        atomicAdd(&s_acc[s_col[kk] * sd + d], s_slot[f].weight * s);
      }
      __syncwarp();
    };
    const int fast = s_fast;
    auto project = [&](const float4 &t0, const float4 &t1, const float4 &t2, const float3 &p) {
      const float T[12] = {t0.x, t0.y, t0.z, t0.w, t1.x, t1.y,
                           t1.z, t1.w, t2.x, t2.y, t2.z, t2.w};
      return A::project(A::apply(T, p), cam);
    };
    auto inside = [&](const float2 &uv) {
      return uv.x >= ulo && uv.x < uhi && uv.y >= ulo && uv.y < vhi;
    };
    // two hypotheses at a time: they share the slot's parameters
    for (int d0 = 0; d0 < D; d0 += 2 * per)
    {
      const int da = d0 + g, db = da + per;
      const bool on_a = mine && da < D, on_b = mine && db < D;
      const float3 pa = A::scale(dir, s_depth[min(da, D - 1)]);
      const float3 pb = A::scale(dir, s_depth[min(db, D - 1)]);
      // the slots that any of the warp's pairs may be in view of
      unsigned view = 0u;
      if constexpr (VIEW)
        view = __reduce_or_sync(0xffffffffu,
                                (on_a ? s_view[da] : 0u) | (on_b ? s_view[db] : 0u));
      unsigned acc_a = 0, acc_b = 0;
      const unsigned id_a = ((unsigned)k << 8) | ((unsigned)da << 16);
      const unsigned id_b = ((unsigned)k << 8) | ((unsigned)db << 16);
      for (int f = 0; f < fast; ++f)
      {
        if constexpr (VIEW)
        {
          const bool any = view & 1u;
          view >>= 1;
          if (!any)
            continue;
        }
        const float4 t0 = s_pose[3 * f], t1 = s_pose[3 * f + 1], t2 = s_pose[3 * f + 2];
        const SlotParam sp = s_slot[f];
        const float2 ua = project(t0, t1, t2, pa), ub = project(t0, t1, t2, pb);
        // true: deferred
        auto take = [&](const float2 &uv, bool on, unsigned &acc) {
          const bool seen = on && inside(uv);
          const F2 c = pack2(uv.x, uv.y), r = round2(c);
          float fx, fy;
          unpack2(sub2(c, sub2(r, pack2(0x1p23f, 0x1p23f))), fx, fy);
          const bool aligned = fmaxf(fabsf(fx), fabsf(fy)) <= sp.margin;
          if (seen)
            acc += sp.weight << 20;
          if (seen && aligned)
          {
            // the rows' first bytes are (x - 1, y - 1 .. y + 1); two words hold
            // three bytes wherever they start (the second one stays inside the
            // image: rows y + 1 <= H - 2)
            const uint8_t *at = sp.img + (offset_of(r, pitch, bias) - pitch - 1u);
            unsigned s = 0;
            unsigned sh = (unsigned)(reinterpret_cast<uintptr_t>(at) & 3u) * 8u;
            const unsigned *w =
                reinterpret_cast<const unsigned *>(reinterpret_cast<uintptr_t>(at) & ~(uintptr_t)3);
#pragma unroll
            for (int j = 0; j < 3; ++j)
            {
              const unsigned lo = __ldg(w), hi = __ldg(w + 1);
              s = sad3(__funnelshift_r(lo, hi, sh) & 0xffffffu, row[j], s);
              if (WORDS) // every row is offset alike within its words
                w = reinterpret_cast<const unsigned *>(reinterpret_cast<const uint8_t *>(w) +
                                                       pitch);
              else
              {
                at += pitch;
                sh = (unsigned)(reinterpret_cast<uintptr_t>(at) & 3u) * 8u;
                w = reinterpret_cast<const unsigned *>(reinterpret_cast<uintptr_t>(at) &
                                                       ~(uintptr_t)3);
              }
            }
            acc += sp.weight * s;
          }
          return seen && !aligned;
        };
        const bool late_a = take(ua, on_a, acc_a), late_b = take(ub, on_b, acc_b);
        const unsigned wa = __ballot_sync(0xffffffffu, late_a);
        const unsigned wb = __ballot_sync(0xffffffffu, late_b);
        if (wa | wb)
        {
          const unsigned below = (1u << lane) - 1u;
          if (late_a)
            s_late[warp][late + __popc(wa & below)] =
                make_float4(ua.x, ua.y, __uint_as_float(id_a + f), 0.0f);
          late += __popc(wa);
          if (late_b)
            s_late[warp][late + __popc(wb & below)] =
                make_float4(ub.x, ub.y, __uint_as_float(id_b + f), 0.0f);
          late += __popc(wb);
          while (late >= 32)
            work_off(32);
        }
      }
      for (int f = fast; f < F; ++f)
      {
        if constexpr (VIEW)
        {
          const bool any = view & 1u;
          view >>= 1;
          if (!any)
            continue;
        }
        const float4 t0 = s_pose[3 * f], t1 = s_pose[3 * f + 1], t2 = s_pose[3 * f + 2];
        const SlotParam sp = s_slot[f];
        const F2 a = pack2(t0.x, t1.x), b = pack2(t0.y, t1.y);
#pragma unroll 1
        for (int h = 0; h < 2; ++h)
        {
          const float2 uv = project(t0, t1, t2, h ? pb : pa);
          if (!((h ? on_b : on_a) && inside(uv)))
            continue;
          const unsigned s = patch_sad(sp.img, pitch, bias, pack2(uv.x, uv.y), a, b, row);
          const unsigned v = (sp.weight << 20) + sp.weight * s;
          if (h)
            acc_b += v;
          else
            acc_a += v;
        }
      }
      if (on_a)
        atomicAdd(&s_acc[col + da], acc_a);
      if (on_b)
        atomicAdd(&s_acc[col + db], acc_b);
    }
    if (late > 0)
      work_off(late);
  }
  __syncthreads();
  // the tile's cells are consecutive in the [cell][all_d] layout.  Element i is
  // s_acc[i + i / D]; i / D = umulhi(i, ceil(2^32 / D)), exact for i < 2^20.
  // D is a multiple of 4, so when the tile starts on a 16-byte boundary
  // (always in the engine's arena; a caller's cost buffer may not) four
  // hypotheses of one cell go out per store.
  float *out = J.lv[0].data + ((size_t)cy * J.cw + cx0) * all_d + h0;
  const unsigned dinv = 0xffffffffu / (unsigned)D + 1u;
  const float add_num = (float)all_d; // writer count of the cell (see above)
  auto value = [&](unsigned v, bool node) {
    const unsigned nvalid = v >> 20;
    const float c = nvalid > 0 ? A::sad_norm((float)(v & 0xfffffu), (float)nvalid) : 100.0f;
    return node ? A::div(c, add_num) : 0.0f;
  };
  if ((reinterpret_cast<uintptr_t>(out) & 15u) == 0)
  {
    for (int i4 = tid; i4 < ncells * D / 4; i4 += blockDim.x)
    {
      const int i = 4 * i4, cell = (int)__umulhi((unsigned)i, dinv);
      const unsigned *src = s_acc + i + cell;
      const bool node = (nodes >> cell) & 1u;
      *reinterpret_cast<float4 *>(out + cell * (all_d - D) + i) =
          make_float4(value(src[0], node), value(src[1], node), value(src[2], node),
                      value(src[3], node));
    }
  }
  else
  {
    for (int i = tid; i < ncells * D; i += blockDim.x)
    {
      const int cell = (int)__umulhi((unsigned)i, dinv);
      out[cell * (all_d - D) + i] = value(s_acc[i + cell], (nodes >> cell) & 1u);
    }
  }
}

} // namespace

int cost_tiles(int cw, int ch) { return ch * ((cw + kCostCells - 1) / kCostCells); }

// Few tiles leave SMs or warp slots idle: their hypotheses are then shared among
// 4 blocks (up to one tile per SM) or 2 (up to three); every count is a multiple
// of 16.  Measured, 64 hypotheses and 5 slots, 1 / 2 / 4 blocks per tile:
// 160x128 (64 tiles) 16.9 / 10.8 / 8.0 us, 320x240 (180) 20.0 / 14.5 / 15.0,
// 480x320 (320) 24.5 / 21.2 / 22.4, 640x480 x 48 (600) 25.5 / 30.0 / 35.5.
int cost_split(long tiles) { return tiles <= 148 ? 4 : tiles <= 444 ? 2 : 1; }

namespace
{
template <int MINB, bool WORDS>
void cost_minb(const Batch &B, int blocks, int arith, int split, bool view, size_t sm,
               cudaStream_t s)
{
  auto go = [&](auto k) { launch_kernel(k, blocks, kFlatThreads, sm, s, B.early, B, split); };
  if (arith == QM_ARITH_IEEE)
    view ? go(k_cost<ArithIeee, MINB, WORDS, true>) : go(k_cost<ArithIeee, MINB, WORDS, false>);
  else
    view ? go(k_cost<ArithRef, MINB, WORDS, true>) : go(k_cost<ArithRef, MINB, WORDS, false>);
}

// Slot images whose rows all start on a word: always in the engine's frame
// pools (widths are multiples of 16); a caller's may not.
bool word_rows(const Batch &B)
{
  if (B.jobs)
    return true;
  unsigned long long all = (unsigned)B.one.slot_pitch;
  for (int f = 0; f < B.one.F; ++f)
    all |= reinterpret_cast<uintptr_t>(B.slots.ptr[f]);
  return (all & 3u) == 0;
}
} // namespace

void launch_cost(const Batch &B, int blocks, int arith, int max_d, int split, bool view,
                 cudaStream_t s, int blocks_per_sm)
{
  const size_t sm = sizeof(unsigned) * kCostCells * (max_d / split + 1);
  if (!word_rows(B)) // single calls only: the default budget
    cost_minb<kCostBlocks, false>(B, blocks, arith, split, view, sm, s);
  else if (blocks_per_sm == 3)
    cost_minb<3, true>(B, blocks, arith, split, view, sm, s);
  else if (blocks_per_sm == 4)
    cost_minb<4, true>(B, blocks, arith, split, view, sm, s);
  else
    cost_minb<5, true>(B, blocks, arith, split, view, sm, s);
}

} // namespace qm
