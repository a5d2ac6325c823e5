// Host engine of the dense pipeline: owns the device buffers of N keyframe
// jobs and runs quadtree -> cost -> BP -> extraction -> upsampling -> fusion
// for any subset of them, one kernel launch per stage, optionally replayed
// from a captured CUDA graph.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <memory>
#include <string>
#include <vector>

#include "launch.h"

namespace qm
{

// thread-local error message behind qm_last_error()
void set_error(const std::string &msg);
const char *get_error();

struct CudaError
{
  int status;
  std::string msg;
};

// Kernel kinds, for per-kind timing (qm_batch_profile).
enum KernelKind
{
  kQuadtree = 0,
  kCost,
  kPyramid,
  kMsgInit, // levels with fewer than two half-sweeps only
  kSweep,
  kExtract,
  kRowSolve,
  kColSolve,
  kFuseTransform,
  kFuseFill, // not launched (hole filling runs inside kFuseUpdate); keeps the
             // kind indices of qm_batch_profile stable
  kFuseUpdate,
  kNumKinds
};

// Default L2 budget of a BP job range: 0, every level over all jobs at once.
// Ranges that fit in L2 (e.g. 64 MiB) keep a range's costs and messages
// resident between its half-sweeps, but on a B200 the smaller launches lose
// more to tails and launch gaps than L2 residency saves (752x480, 64
// hypotheses, 32 streams: 4.60 ms per batch ungrouped, 4.72 ms at 64 MiB,
// 5.23 ms at 24 MiB).
constexpr size_t kDefaultGroupBytes = 0;

// Default number of concurrent pipeline branches per batch (consecutive ranges
// of the active jobs, bit-identical results).  submit + wait / resident, two
// and three branches: 32 x 752x480 3.45 / 2.48 and 3.32 / 2.50 ms, 8 x 752x480
// 0.96 / 0.73 and 0.92 / 0.72, 8 x 1920x1080 9.73 / 8.93 and 9.47 / 8.88; four:
// 3.34 / 2.61 and 9.24 / 8.82.
#ifndef QM_DEFAULT_BRANCHES
#define QM_DEFAULT_BRANCHES 3
#endif
constexpr int kMaxBranches = 4;

struct LaunchProfile
{
  struct Mark
  {
    int kind;
    cudaEvent_t e0, e1;
  };
  std::vector<Mark> marks;
};

struct Shape
{
  int W, H, D, F;
  Cam cam;
};

struct JobBuffers
{
  uint8_t *levels = nullptr;
  float *data[kMaxLevels] = {};
  float *msg[kMaxLevels][4] = {};
  int lw[kMaxLevels] = {}, lh[kMaxLevels] = {};
  int32_t *labels = nullptr;
  float *sparse = nullptr;
  float *dense[2] = {}; // by step parity (a step's result can be read
                        // back while the next step runs)
  float2 *rowres = nullptr;
  float4 *seeds[2] = {};
  unsigned long long *zkey = nullptr;  // fusion z-buffer (reset by the row solve)
  unsigned long long *sdkey = nullptr; // semi-dense z-buffer (all ones between its steps)
};

// Byte layout of one job's buffers (offsets from a 256-byte aligned base).
struct JobLayout
{
  size_t bytes = 0;
  size_t off_levels, off_data[kMaxLevels], off_msg[kMaxLevels][4], off_labels, off_sparse,
      off_dense[2], off_rowres, off_seeds[2], off_zkey, off_sdkey;
  int lw[kMaxLevels], lh[kMaxLevels];
  static JobLayout make(const Shape &s, int nlev);
};

// Fills a JobDesc (geometry, parameters, buffer pointers) for one job.
JobDesc make_job_desc(const Shape &s, const qm_params &p, const JobBuffers &b, int seeds_cur);

// Validates a parameter struct and a shape; returns an empty string when OK.
std::string validate(const qm_params &p);
std::string validate(const Shape &s, const qm_params &p);

KParams kparams(const qm_params &p);

// True when the 3x4 pose is finite and its rotation rows satisfy
// |r00| + |r01| <= 1.5 and |r10| + |r11| <= 1.5 (every rotation does): the
// cost kernel's rotated 3x3 patch then stays inside the measurement image.
bool rigid_enough(const float *T);

// Merges measurement slots with the same image and pose: writes the unique
// slots (first-occurrence order) with their multiplicities and returns how
// many there are.  Throws CudaError(QM_ERR_INVALID_ARG) for a pose that is
// not rigid_enough.
int dedupe_slots(int F, const uint8_t *const *ptrs, const float *T, const uint8_t **out_ptrs,
                 float *out_T, int *out_w);

// Stage plan of one active job set: block prefix per stage, in one device
// buffer, plus the captured graph.
struct Plan;
struct TableBuf;

// Validates launch shapes for lines up to max_w / max_h samples.
std::string validate(const Tune &t, int max_w, int max_h);

class Engine
{
public:
  Engine(int device, const qm_params &p, const std::vector<Shape> &shapes);
  ~Engine();
  Engine(const Engine &) = delete;
  Engine &operator=(const Engine &) = delete;

  int njobs() const { return (int)shapes_.size(); }
  const Shape &shape(int j) const { return shapes_[j]; }
  const JobBuffers &buffers(int j) const { return bufs_[j]; }
  const qm_params &params() const { return params_; }
  cudaStream_t stream() const { return stream_; }
  int device() const { return device_; }

  // Step parity: selects the output buffer and the pinned descriptor and
  // slot tables that set_inputs / launch use, so that the host can prepare
  // step t+1 while step t (the other parity) is still in flight.
  void set_parity(int p) { parity_ = p & 1; }
  int parity() const { return parity_; }
  // fused depth buffer of job j for the current parity
  float *dense(int j) const { return bufs_[j].dense[parity_]; }

  // Inputs of job j for the next run.  Device pointers; T_slot_ref is
  // F*12 floats (host), T_fuse 12 floats T_income<-lastfuse (host).
  void set_inputs(int j, const uint8_t *ref, int ref_pitch, const uint8_t *const *slots,
                  int slot_pitch, const float *T_slot_ref, const float *T_fuse);
  // Current seed buffer of job j (after the last run).
  float4 *seeds(int j) const { return bufs_[j].seeds[seeds_cur_[j]]; }
  void reset_seeds(int j);

  // Enqueues the pipeline for `active` job indices without waiting; stream()
  // is behind it.  Throws CudaError.  Graph capture is used when `graphs` is
  // set.  ready[i] (may be null): event branch i waits for before it starts.
  void launch(const std::vector<int> &active, const cudaEvent_t *ready = nullptr);
  // The branches of the next launch of `active`: branch i runs the jobs
  // order[cuts[i]] .. order[cuts[i + 1] - 1].  After the launch,
  // branch_done(i) marks its end.
  void layout(const std::vector<int> &active, std::vector<int> &order, std::vector<int> &cuts);
  cudaEvent_t branch_done(int i) const { return ev_branch_[i]; }
  // launch() and wait for it
  void run(const std::vector<int> &active);
  void set_graphs(bool on) { graphs_ = on; }
  // L2 budget of a BP job range (0: every level over all jobs at once)
  void set_group_bytes(size_t bytes) { group_bytes_ = bytes; }
  // k (1..4): the pipeline runs as k concurrent branches over consecutive
  // ranges of the active jobs (graph branches, or streams when launching
  // eagerly); 1: one sequence over all jobs.  Results do not depend on it.
  void set_branches(int k);
  int branches() const { return branches_; }
  size_t group_bytes() const { return group_bytes_; }
  // coarse BP levels (at most `cells` cells in every active job) in one
  // cluster launch; 0: one launch per half-sweep at every level; kCoarseAuto
  // until it is called.  Results do not depend on it.
  void set_coarse_cells(int cells) { coarse_cells_ = cells < 0 ? 0 : cells; }
  // true: branch i + 1 starts once branch i's cost volume is done, so the
  // issue-bound cost kernel of one branch runs beside the bandwidth-bound
  // BP of the previous one; false (the default; resident pass with three
  // branches, off / on: 4 x 752x480 401 / 434 us, 32 x 752x480 2.36 / 2.40 ms, 8 x
  // 1920x1080 6.64 / 8.04): all branches start together.  Results do not depend
  // on it.
  void set_stagger(bool on) { stagger_ = on; }
  bool stagger() const { return stagger_; }
  int coarse_cells() const { return coarse_cells_; }
  int last_launches() const { return last_launches_; }
  // 1: the sparse buffers arrive filled with the semi-dense tracker's depths
  // (the quadtree pass keeps them instead of clearing)
  void set_keep_sparse(bool on)
  {
    for (auto &J : master_)
      J.keep_sparse = on ? 1 : 0;
  }
  // Launch shapes of the BP and line-solver kernels.  With autotune on (the
  // default) each active job set times three candidates per kernel family
  // on its first run and keeps the fastest; set_tune fixes the shapes for
  // every set (autotune off).  Results do not depend on the shapes.
  void set_autotune(bool on);
  bool autotune() const { return autotune_; }
  void set_tune(const Tune &t);
  // shapes of the last launched or profiled set
  Tune last_tune() const { return last_tune_; }
  // Events bracketing the device work of the last run (for timing).
  float last_run_ms() const;
  // Runs the pipeline once with eager launches, each bracketed by events;
  // ms[k] / launches[k] receive the summed device time and launch count per
  // KernelKind.
  void profile(const std::vector<int> &active, float *ms, int *launches);

private:
  Plan &plan_for(const std::vector<int> &active);
  std::vector<int> branch_cuts(const std::vector<int> &order) const;
  std::unique_ptr<TableBuf> build_table(const std::vector<int> &active, const Tune &tune);
  void tune_plan(Plan &pl);
  // packs the descriptors of `active` into the pinned run array
  void pack(const std::vector<int> &active);
  // enqueues the descriptor and slot-table uploads; returns the batch
  Batch upload(int n, cudaStream_t s);
  // runs stages [first, last] of branch i on s, from its graph when graphs are
  // on (part: which of the plan's graphs)
  void run_part(Plan &pl, const Batch &B, int i, int part, int first, int last, cudaStream_t s);

  int device_;
  qm_params params_;
  std::vector<Shape> shapes_;
  std::vector<JobLayout> layouts_;
  std::vector<JobBuffers> bufs_;
  std::vector<int> seeds_cur_;
  void *arena_ = nullptr;
  // One step's descriptors -- the packed job descriptors, then the slot tables
  // of all jobs (image, pose, multiplicity) -- as one block: pinned per parity,
  // and its device copy
  std::vector<int> slot_base_;
  int total_slots_ = 0;
  struct StepBlock
  {
    char *base = nullptr;
    JobDesc *run = nullptr;
    const uint8_t **slot_ptr = nullptr;
    float *slot_T = nullptr;
    int *slot_w = nullptr;
  };
  size_t block_bytes_ = 0;
  StepBlock h_block_[2], d_block_;
  std::vector<JobDesc> master_; // host master copies of the descriptors
  cudaStream_t stream_ = nullptr;
  cudaStream_t branch_[kMaxBranches - 1] = {}; // streams of branches 2..k
  cudaEvent_t ev_fork_ = nullptr, ev_branch_[kMaxBranches] = {}; // branch i done
  cudaEvent_t ev_stage_[kMaxBranches - 1] = {}; // branch i's cost stage done
  bool stagger_ = false;
  int branches_ = QM_DEFAULT_BRANCHES;
  cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
  bool graphs_ = true;
  int parity_ = 0;
  size_t group_bytes_ = kDefaultGroupBytes;
  int coarse_cells_ = kCoarseAuto;
  int last_launches_ = 0;
  bool autotune_ = true;
  Tune fixed_tune_, last_tune_;
  std::map<std::vector<int>, std::unique_ptr<Plan>> plans_;
};

} // namespace qm
