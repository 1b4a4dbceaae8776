// gd_common.h -- host-side internals shared by gd_api.cu and gd_ensemble.cu:
// the opaque handle types, error reporting and launch-shape selection.
#pragma once

#include <atomic>
#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "gd_internal.h"

namespace gd {

gd_status fail(gd_status st, const char *fmt, ...);

#define GD_CUDA(call)                                                                   \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return ::gd::fail(e_ == cudaErrorMemoryAllocation ? GD_ENOMEM : GD_ECUDA,          \
                        "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__,      \
                        __LINE__);                                                      \
  } while (0)

#define GD_TRY(call)            \
  do {                          \
    gd_status s_ = (call);      \
    if (s_ != GD_OK) return s_; \
  } while (0)

constexpr float kPI = 3.1415926535f;  // size.h:86

// NVTX range over a host call (shown by profilers that attach a tool; free
// otherwise).
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// Launch shape of the energy kernel: A atom groups x P tile groups of warps,
// NA ligand atoms per warp.
struct Tile {
  int A = 0, P = 0, NA = 0;
  bool valid() const { return A > 0 && P > 0 && NA > 0; }
};

// Candidate atoms-per-warp values compiled into the kernel.
// Even: the pair loop handles two atoms per packed f32x2 instruction.
constexpr int kNAValues[] = {2, 4, 6, 8, 10};

Tile default_tile(int lna);
int round_na(int na);  // smallest compiled NA >= na (0 if none)
// Resident staging when the tiles of one CTA (of a split's busiest CTA) fit
// in shared memory, else the streaming ring.
// lists: as in dock_smem_bytes
void pick_stages(const KTables &T, const Tile &t, int *n_stages, int *resident, int split,
                 bool lists);

}  // namespace gd

// Most bytes of workspace kept between calls on a device, and the bytes of a
// context's pinned staging.
namespace gd {
constexpr size_t kKeepBytes = 64 << 20;
constexpr size_t kStageBytes = 256 << 10;
}

// Handles are reference counted: a complex keeps its context (and a shared
// protein's owner) alive, a REMC run or batch keeps its complexes alive, so
// callers may destroy them in any order.
struct gd_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // pinned host memory that kernels access directly: the error word (read once
  // the stream has ended, no copy), then kStageBytes through which small
  // results and pose calls pass, used under stage_mu
  int *h_err = nullptr;
  unsigned char *stage = nullptr;
  void *shared = nullptr;  // its lease of them (gd_shared.h)
  std::mutex stage_mu;
  uint64_t launches = 0;
  int n_sm = 148;
  int sched_mode = 0;      // GD_SCHED_*
  int sched_machines = 0;  // persistent CTAs (0: SMs x occupancy)
  int sched_tail = 2;      // last MC steps of every unit left to the shared queue
  int split_mode = 0;      // CTAs per unit of MC launches (0: split_for's rule)
  uint32_t wait_limit = 0; // polls of a dependency wait before it gives up (0: default)
  int wait_bias = 0;       // added to every dependency wait's target (test hook)
  std::atomic<int> alloc_fail_in{0};  // > 0: that many device allocations from now,
                                      // the last one fails (test hook)
  std::atomic<int> refs{1};
  // autotuned launch shapes keyed by (ligand-size bucket, protein tiles)
  std::mutex tile_mu;
  std::map<std::pair<int, int>, gd::Tile> tiles;
  // side streams: launches of different shapes run side by side on them
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> side_done;
  cudaEvent_t forked = nullptr;
  // address of the library's fixed pose-scratch array in the CUDA context
  // that was current when this gd_ctx was created (gd_energy_poses_noalloc)
  unsigned char *noalloc_scratch = nullptr;
};

struct gd_dcomplex {
  gd_ctx *ctx = nullptr;
  gd::KTables T{};
  std::vector<void *> allocs;
  size_t bytes = 0;
  std::atomic<int> refs{1};
  gd_dcomplex *protein_owner = nullptr;  // when the protein arrays are shared
  double far_share = 0.0;  // share of the protein's points that are far of the
                           // ligand at its start place, however it is turned
  // device position -> caller's point index: points whose type can form an
  // H-bond come first, so a 32-point chunk rarely mixes the two kinds
  std::vector<int> point_order;
};

namespace gd {
void ctx_retain(gd_ctx *c);
void ctx_release(gd_ctx *c);
void dcx_retain(gd_dcomplex *d);
void dcx_release(gd_dcomplex *d);
gd_status ctx_check(gd_ctx *c);
// Status for a nonzero kernel error word (KRun.err).
gd_status kernel_error(int code);
// Loads the module that holds the fixed pose-scratch array of
// gd_energy_poses_noalloc on c's device (current) and stores the array's
// address in c->noalloc_scratch (gd_noalloc.cu).  Called by gd_ctx_create.
gd_status noalloc_attach(gd_ctx *c);
// Test hook of gd_ctx_set_alloc_fail: true (and the hook off again) when
// this device allocation through c is the one set to fail.
inline bool injected_alloc_failure(gd_ctx *c) {
  int n = c->alloc_fail_in.load();
  while (n > 0 && !c->alloc_fail_in.compare_exchange_weak(n, n - 1)) {
  }
  return n == 1;
}
// The device memory of one call, all of whose work is on the context's stream
// (poses, similarity): a slab that the device's contexts keep (gd_shared.h), so
// that a repeated call makes no allocation.  (Each took 50 .. 100 us from the
// device's default pool, which unmaps at every synchronisation; from a pool
// shared by the device's contexts a call took longer with every context that had
// used it: 0.10 ms with one, 0.55 with 24.)  A call under capture, whose graph may
// run beside later calls, one that finds no slab and what is beyond kKeepBytes
// take memory of their own from the default pool.
class Workspace {
 public:
  // expect: what the call is likely to need in all
  Workspace(gd_ctx *c, size_t expect) : c_(c), expect_(expect) {}
  ~Workspace();
  Workspace(const Workspace &) = delete;
  Workspace &operator=(const Workspace &) = delete;
  static size_t padded(size_t bytes) { return (bytes + 255) & ~size_t(255); }
  cudaError_t get(void **p, size_t bytes);

 private:
  void take(size_t bytes);
  gd_ctx *c_;
  const size_t expect_;
  bool asked_ = false;
  void *slab_ = nullptr;  // (DeviceShared::Slab)
  unsigned char *base_ = nullptr;
  size_t room_ = 0, used_ = 0, want_ = 0;
  static constexpr int kOwn = 12;
  void *own_[kOwn];
  int n_own_ = 0;
};
// Ligand-size bucket: sizes are rounded up to a multiple of 8 atoms; launch
// shapes are chosen (and autotuned) per bucket and cover its largest size.
int lna_bucket(int lna);
Tile tile_for(gd_ctx *ctx, const KTables &T);
// The energy launch of a pose call (gd_api.cu): poses, terms and raw are
// device pointers, work pose_work_bytes of device memory (nullptr without).
gd_status poses_launch(gd_ctx *ctx, const gd_dcomplex *d, int prt_conf, int lig_conf, int n_pose,
                       const float *poses, float *terms, double *raw, void *work);
// CTAs (a thread-block cluster) that share each 32-replica unit of a complex
// in MC launches.  The order of the FP64 sums, and so a run's last bits, depend on
// it.  split_rule: a function of the complex (ligand-size bucket x protein points)
// and of run_units, the units that want SMs with it; for a server request those
// of its own run, never of what else runs, so a request's results do not depend on
// the server's load.  In a run or batch, run_splits (gd_ensemble.cu) deals the
// SMs over all its complexes, the costliest first: a complex's split there follows
// from the sizes of the others too.
// min_cost: pairs per CTA that a split must leave.  Runs and batches have the GPU
// to themselves: kRunSplitCost.  Server requests share it with one another:
// kServeSplitCost, so that splitting under load costs little throughput.
constexpr double kRunSplitCost = 4500.0;
constexpr double kServeSplitCost = 42500.0;
int split_rule(gd_ctx *ctx, const KTables &T, int run_units, double min_cost);
// The split of an MC run: the context's own (gd_ctx_set_split), else the rule's.
int split_for(gd_ctx *ctx, const KTables &T, int run_units, double min_cost);
// 32-replica units of a complex's replicas (n_prt x n_lig x n_tmp): whole
// exchange groups per unit when n_tmp divides 32.
int units_of(int n_prt, int n_lig, int n_tmp);
// What an idle server lane launches next: the initialisation of its new
// requests (true), or MC steps of those it has.  Never two initialisations in
// a row while it has some: under steady arrivals they would take no step.
inline bool lane_inits_next(bool has_fresh, bool has_members, bool last_was_init) {
  return has_fresh && !(has_members && last_was_init);
}
// MC launches whose complexes have a smaller share of far points (far_share)
// take them all in the full form (KFORM_NEAR, the same bits).  20 steps of 160
// units, near form against near / far: share 0.01 (96 atoms x 700 points) 7.59
// against 8.14 ms, 0.08 (24 x 700) 2.38 and 2.52, 0.17 (96 x 1,500) 13.9 and 14.4;
// 0.29 (48 x 1,500) 7.18 and 7.10, 0.43 (24 x 1,500) 3.83 and 3.61.
constexpr double kFarShareMc = 0.25;
// Whether each of those units has at most 16 replicas (KRun.packed).  One full
// unit keeps the ordered kernel for all of them: the packed one forms its sums
// in another order, and the run ends with its full units either way.
bool all_packed_units(int n_lig, int n_tmp);

// Launches of different shapes (one per launch plan) are independent; each
// kernel holds one CTA per SM, so a plan with fewer CTAs than SMs leaves the
// rest idle unless the next plan runs beside it.  fork_streams returns n
// streams (n <= kMaxSide; the first is ctx->stream) that start after the work
// already queued on ctx->stream; join_streams makes ctx->stream wait for all
// of them.  Both work inside a stream capture, which turns the plans into
// parallel graph branches.  Plans beyond kMaxSide share streams (and run
// after the plan they share one with), so it covers every launch-shape class
// a batch can have in practice.
constexpr int kMaxSide = 32;
gd_status fork_streams(gd_ctx *c, int n, cudaStream_t *out);
gd_status join_streams(gd_ctx *c, int n);
}  // namespace gd
