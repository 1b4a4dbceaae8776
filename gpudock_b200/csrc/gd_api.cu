// gd_api.cu -- host side of the C-ABI in include/gpudock.h: errors, force
// field and temperature tables, validation, contexts, the device layout of a
// complex, pose energies, launch-shape selection and test entry points.
//
// Boundary replaced: the table staging of Run() in
// gpudocksm-rem-1.2/src/run.cu:114-256 (cudaMemcpy / cudaMemcpyToSymbol into
// __constant__ globals, exit() on any error).  Here every call returns a
// status and device memory belongs to reference-counted handles.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <new>
#include <string>
#include <vector>

#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "gd_common.h"
#include "gd_shared.h"

using namespace gd;

namespace gd {

static thread_local std::string g_err;

gd_status fail(gd_status st, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return st;
}

int round_na(int na) {
  for (int v : kNAValues)
    if (v >= na) return v;
  return 0;
}

// Default launch shape (used until the autotuner has timed a size class):
// atom groups to cover the ligand and as many tile groups as fit in
// MAX_WARPS (resident or streamed, the groups split the protein's chunks).
Tile default_tile(int lna) {
  // A warp's time per protein point is about NA + 1.5 pair-slots (its atoms
  // plus the per-point loads and test), and the A x P warps share the points
  // P ways: pick the shape with the smallest (NA + 1.5) / P.
  Tile best;
  double best_cost = 1e30;
  for (int na : kNAValues) {
    const int A = (lna + na - 1) / na;
    if (A > MAX_WARPS) continue;
    const int NA = round_na((lna + A - 1) / A);
    const int P = std::max(1, MAX_WARPS / A);
    const double cost = (NA + 1.5) / P;
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best.A = A;
      best.P = P;
      best.NA = NA;
    }
  }
  return best;
}

void pick_stages(const KTables &T, const Tile &t, int *n_stages, int *resident, int split,
                 bool lists) {
  const int n_tiles = (T.pnp + TILE_PTS - 1) / TILE_PTS;
  const int own = (n_tiles + split - 1) / split;  // tiles of a split's busiest CTA
  const size_t limit = 227 * 1024;
  if (own <= MAX_RESIDENT_TILES && dock_smem_bytes(t.A, t.P, t.NA, own, split, lists) <= limit) {
    *n_stages = own;
    *resident = 1;
  } else {
    *n_stages = STREAM_STAGES;
    *resident = 0;
  }
}

int lna_bucket(int lna) { return std::min(((lna + 7) / 8) * 8, MAX_LNA); }

int split_for(gd_ctx *ctx, const KTables &T, int run_units, double min_cost) {
  return ctx->split_mode > 0 ? ctx->split_mode : split_rule(ctx, T, run_units, min_cost);
}

int split_rule(gd_ctx *ctx, const KTables &T, int run_units, double min_cost) {
  // the largest power of two <= cost / min_cost and <= SMs / units, at most
  // 8: a run that fills the GPU with units gains nothing from splitting
  const double cost = (double)lna_bucket(T.lna) * T.pnp;
  const int free = ctx->n_sm / std::max(1, run_units);
  int k = 1;
  while (k < MAX_SPLIT && cost >= min_cost * 2.0 * k && 2 * k <= free) k *= 2;
  return k;
}

int units_of(int n_prt, int n_lig, int n_tmp) {
  if (32 % n_tmp == 0) {
    const int G = 32 / n_tmp;  // ligand conformations per unit
    return n_prt * ((n_lig + G - 1) / G);
  }
  return n_prt * ((n_lig * n_tmp + 31) / 32);
}

bool all_packed_units(int n_lig, int n_tmp) {
  // every unit but the last of a protein conformation is full
  const int full = 32 % n_tmp == 0 ? 32 / n_tmp * n_tmp : 32;
  return packed_reps(std::min(full, n_lig * n_tmp)) < 32;
}

Tile tile_for(gd_ctx *ctx, const KTables &T) {
  const int n_tiles = (T.pnp + TILE_PTS - 1) / TILE_PTS;
  const int hi = lna_bucket(T.lna);
  {
    std::lock_guard<std::mutex> g(ctx->tile_mu);
    auto it = ctx->tiles.find({hi, n_tiles});
    if (it != ctx->tiles.end()) return it->second;
  }
  return default_tile(hi);
}

// The runtime behind what a device's contexts share (gd_shared.h).
struct CudaShared {
  using Error = cudaError_t;
  using Stream = cudaStream_t;
  using Event = cudaEvent_t;
  static bool ok(Error e) { return e == cudaSuccess; }
  // Serial number of the device's CUDA context, which no later one of the
  // process has (0: this driver does not tell).
  static uint64_t serial() {
    static const std::pair<PFN_cuCtxGetCurrent_v4000, PFN_cuCtxGetId_v12000> fn = [] {
      void *cur = nullptr, *id = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &cur, 4000, cudaEnableDefault, &q) !=
          cudaSuccess)
        cur = nullptr;
      if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &id, 12000, cudaEnableDefault, &q) !=
          cudaSuccess)
        id = nullptr;
      cudaGetLastError();
      return std::make_pair((PFN_cuCtxGetCurrent_v4000)cur, (PFN_cuCtxGetId_v12000)id);
    }();
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!fn.first || !fn.second || fn.first(&c) != CUDA_SUCCESS || !c ||
        fn.second(c, &id) != CUDA_SUCCESS)
      return 0;
    return (uint64_t)id + 1;
  }
  static Error pin(void **p, size_t bytes) { return cudaHostAlloc(p, bytes, cudaHostAllocDefault); }
  static void unpin(void *p) { cudaFreeHost(p); }
  static Error alloc(void **p, size_t bytes, Stream s) {
    const cudaError_t e = cudaMallocAsync(p, bytes, s);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
  }
  static void free(void *p, Stream s) { cudaFreeAsync(p, s); }
  static Error event(Event *e) { return cudaEventCreateWithFlags(e, cudaEventDisableTiming); }
  static Error record(Event e, Stream s) { return cudaEventRecord(e, s); }
  static bool done(Event e) {
    const cudaError_t q = cudaEventQuery(e);
    if (q != cudaSuccess && q != cudaErrorNotReady) cudaGetLastError();
    return q == cudaSuccess;
  }
  static void drop(Event e) { cudaEventDestroy(e); }
};

// Never destroyed: a handle may be released while the process ends.
using Shared = DeviceShared<CudaShared>;
static Shared &shared() {
  static auto *s = new Shared(256 + kStageBytes, kKeepBytes);
  return *s;
}
static Shared::Group *group_of(gd_ctx *c) { return static_cast<Shared::Lease *>(c->shared)->group; }

// The context's error word and staging.
static cudaError_t shared_attach(gd_ctx *c) {
  Shared::Lease *l = nullptr;
  cudaError_t e = cudaErrorMemoryAllocation;
  try {
    l = new Shared::Lease;
    e = shared().acquire(c->device, l);
  } catch (const std::bad_alloc &) {
  }
  if (e != cudaSuccess) {
    delete l;
    return e;
  }
  c->shared = l;
  c->h_err = static_cast<int *>(l->block);
  c->stage = static_cast<unsigned char *>(l->block) + 256;
  std::memset(l->block, 0, 256);
  return cudaSuccess;
}

static void shared_detach(gd_ctx *c) {
  auto *l = static_cast<Shared::Lease *>(c->shared);
  if (!l) return;
  shared().release(l, c, c->stream);
  delete l;
  c->shared = nullptr;
}

// A slab for this call, unless the stream is under capture.
void Workspace::take(size_t bytes) {
  asked_ = true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(c_->stream, &cap) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (cap != cudaStreamCaptureStatusNone) return;
  Shared::Slab *b = shared().lend(group_of(c_), c_, c_->stream, bytes);
  if (!b) return;
  slab_ = b;
  base_ = b->p;
  room_ = b->bytes;
}

Workspace::~Workspace() {
  for (int k = 0; k < n_own_; ++k) cudaFreeAsync(own_[k], c_->stream);
  if (slab_)
    shared().give_back(group_of(c_), static_cast<Shared::Slab *>(slab_), c_, c_->stream, want_);
}

cudaError_t Workspace::get(void **p, size_t bytes) {
  *p = nullptr;
  if (injected_alloc_failure(c_)) return cudaErrorMemoryAllocation;
  bytes = padded(std::max<size_t>(bytes, 1));
  if (!asked_) take(std::max(expect_, bytes));
  want_ += bytes;
  if (used_ + bytes <= room_) {
    *p = base_ + used_;
    used_ += bytes;
    return cudaSuccess;
  }
  if (n_own_ == kOwn) return cudaErrorMemoryAllocation;
  const cudaError_t e = cudaMallocAsync(p, bytes, c_->stream);
  if (e == cudaSuccess)
    own_[n_own_++] = *p;
  else
    *p = nullptr;
  return e;
}

void ctx_retain(gd_ctx *c) {
  if (c) c->refs++;
}

gd_status fork_streams(gd_ctx *c, int n, cudaStream_t *out) {
  n = std::max(1, std::min(n, kMaxSide));
  out[0] = c->stream;
  if (n == 1) return GD_OK;
  if (!c->forked) GD_CUDA(cudaEventCreateWithFlags(&c->forked, cudaEventDisableTiming));
  while ((int)c->side.size() < n - 1) {
    cudaStream_t s = nullptr;
    cudaEvent_t e = nullptr;
    GD_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    c->side.push_back(s);
    GD_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    c->side_done.push_back(e);
  }
  GD_CUDA(cudaEventRecord(c->forked, c->stream));
  for (int k = 1; k < n; ++k) {
    GD_CUDA(cudaStreamWaitEvent(c->side[k - 1], c->forked, 0));
    out[k] = c->side[k - 1];
  }
  return GD_OK;
}

gd_status join_streams(gd_ctx *c, int n) {
  n = std::max(1, std::min(n, kMaxSide));
  for (int k = 1; k < n; ++k) {
    GD_CUDA(cudaEventRecord(c->side_done[k - 1], c->side[k - 1]));
    GD_CUDA(cudaStreamWaitEvent(c->stream, c->side_done[k - 1], 0));
  }
  return GD_OK;
}

void ctx_release(gd_ctx *c) {
  if (!c || --c->refs > 0) return;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  for (cudaStream_t s : c->side) {
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
  }
  for (cudaEvent_t e : c->side_done) cudaEventDestroy(e);
  if (c->forked) cudaEventDestroy(c->forked);
  shared_detach(c);
  if (c->own_stream) cudaStreamDestroy(c->stream);
  delete c;
}

void dcx_retain(gd_dcomplex *d) {
  if (d) d->refs++;
}

// The last reference frees the tables in stream order on the context stream
// (work of the library's side streams is joined into it; the server frees a
// request only after its lane's launches have ended).
void dcx_release(gd_dcomplex *d) {
  if (!d || --d->refs > 0) return;
  if (d->ctx) {
    cudaSetDevice(d->ctx->device);
    for (void *p : d->allocs) cudaFreeAsync(p, d->ctx->stream);
  }
  gd_ctx *c = d->ctx;
  gd_dcomplex *owner = d->protein_owner;
  delete d;
  dcx_release(owner);
  ctx_release(c);
}

gd_status kernel_error(int code) {
  if (code == 3)
    return fail(GD_ECUDA, "internal: a warp needs more H-bond atom pairs than its launch "
                          "shape evaluates");
  if (code == 4)
    return fail(GD_ETIMEDOUT, "a persistent CTA gave up waiting for the earlier MC steps of "
                              "its unit (code 4)");
  return fail(GD_ETIMEDOUT, "a bounded barrier wait gave up in a kernel (code %d)", code);
}

gd_status ctx_check(gd_ctx *c) {
  GD_CUDA(cudaStreamSynchronize(c->stream));
  const int code = *(volatile int *)c->h_err;
  if (code == 0) return GD_OK;
  *(volatile int *)c->h_err = 0;
  return kernel_error(code);
}

}  // namespace gd

extern "C" const char *gd_last_error(void) { return gd::g_err.c_str(); }
extern "C" const char *gd_version(void) { return "gpudock-b200 0.2 (sm_100a)"; }

// ---------------------------------------------------------------------------
// Force-field tables (OptimizeEnepara, util.C:405-458) and temperatures
// (SetTemperature, util.C:491-532): host arithmetic in single precision with
// the same libm calls, so the tables match the reference's bit for bit.
// ---------------------------------------------------------------------------
extern "C" gd_status gd_enepara_optimize(const gd_enepara_raw *r, gd_enepara *e) {
  if (!r || !e) return fail(GD_EINVAL, "gd_enepara_optimize: NULL argument");
  const float sqrt_2_pi = sqrtf(2.0f * kPI);
  std::memset(e, 0, sizeof(*e));
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) {
      const float tmp = r->vdw[j][i][0] * r->lj[2];
      e->p1a[i][j] = 2.0f * r->vdw[j][i][1] * powf(tmp, 9.0f);
      e->p2a[i][j] = 3.0f * r->vdw[j][i][1] * powf(tmp, 6.0f);
    }
  e->lj0 = r->lj[0];
  e->lj1 = r->lj[1];
  e->el0 = r->el[0];
  e->a1 = 4.0f - 3.0f * r->el[0];
  e->b1 = 2.0f * r->el[0] - 3.0f;
  e->el1 = r->el[1];
  for (int i = 0; i < GD_NELE; ++i) e->ele[i] = r->ele[i];
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) {
      e->pmf0[i][j] = r->pmf[j][i][0];
      e->pmf1[i][j] = r->pmf[j][i][1];
      e->hdb0[i][j] = r->hdb[j][i][0];
      e->hdb1[i][j] = 1.0f / r->hdb[j][i][1];
      e->hdb2[i][j] = -1.0f / (r->hdb[j][i][1] * sqrt_2_pi);
    }
  for (int i = 0; i < GD_NRES; ++i) e->hpp[i] = r->hpp[i];
  for (int i = 0; i < GD_NLT; ++i) {
    e->hpl0[i] = r->hpl[i][0];
    e->hpl1[i] = r->hpl[i][1];
    e->hpl2[i] = logf(1.0f / (e->hpl1[i] * sqrt_2_pi));
  }
  e->kde2 = -0.5f / (r->kde * r->kde);
  e->kde3 = powf(r->kde * sqrt_2_pi, 3.0f);
  for (int i = 0; i < GD_NTERM; ++i) {
    e->w[i] = r->w[i];
    e->a_para[i] = r->a_para[i];
    e->b_para[i] = r->b_para[i];
  }
  return GD_OK;
}

extern "C" gd_status gd_set_temperature(int n, float floor_t, float ceil_t, float *temps,
                                        float *minus_beta) {
  if (n < 1 || !minus_beta) return fail(GD_EINVAL, "gd_set_temperature: n=%d", n);
  if (!(floor_t > 0.f) || !(ceil_t > 0.f))
    return fail(GD_EINVAL, "gd_set_temperature: temperatures must be > 0");
  if (n == 1) {
    const float beta = 1.0f / (1.0f * floor_t);
    if (temps) temps[0] = floor_t;
    minus_beta[0] = 0.0f - beta;
    return GD_OK;
  }
  const float ratio = expf(logf(ceil_t / floor_t) / (float)(n - 1));
  float a = floor_t;
  for (int i = 0; i < n; ++i) {
    const float beta = 1.0f / (1.0f * a);
    if (temps) temps[i] = a;
    minus_beta[i] = 0.0f - beta;
    a *= ratio;
  }
  return GD_OK;
}

// Rigid poses given as a translation and a rotation quaternion, as the
// move vectors of Move_d (move_d.cu:90-105): R = Rz(m3) Ry(m4) Rx(m5), so
// r00 = cos m3 cos m4, r10 = sin m3 cos m4, r20 = -sin m4, r21 = cos m4 sin m5,
// r22 = cos m4 cos m5.  Where cos m4 vanishes only m5 - m3 (m4 = pi/2) or
// m5 + m3 (m4 = -pi/2) is fixed; m3 = 0 then.  Double precision throughout.
extern "C" gd_status gd_poses_from_quaternions(int n_pose, const float *quat_poses,
                                               float *poses) {
  if (n_pose < 0 || (n_pose > 0 && (!quat_poses || !poses)))
    return fail(GD_EINVAL, "gd_poses_from_quaternions: n_pose=%d", n_pose);
  for (int i = 0; i < n_pose; ++i) {
    const float *q = quat_poses + (size_t)i * 7;
    for (int k = 0; k < 7; ++k)
      if (!std::isfinite(q[k])) return fail(GD_EINVAL, "pose %d: non-finite value", i);
    double w = q[3], x = q[4], y = q[5], z = q[6];
    const double nrm = std::sqrt(w * w + x * x + y * y + z * z);
    if (!(nrm > 0.0)) return fail(GD_EINVAL, "pose %d: zero quaternion", i);
    w /= nrm, x /= nrm, y /= nrm, z /= nrm;
    const double r00 = 1.0 - 2.0 * (y * y + z * z), r01 = 2.0 * (x * y - w * z);
    const double r10 = 2.0 * (x * y + w * z), r11 = 1.0 - 2.0 * (x * x + z * z);
    const double r20 = 2.0 * (x * z - w * y), r21 = 2.0 * (y * z + w * x);
    const double r22 = 1.0 - 2.0 * (x * x + y * y);
    const double m4 = -std::asin(std::min(1.0, std::max(-1.0, r20)));
    double m3, m5;
    if (std::hypot(r00, r10) > 1e-9) {
      m3 = std::atan2(r10, r00);
      m5 = std::atan2(r21, r22);
    } else {
      m3 = 0.0;
      m5 = r20 < 0.0 ? std::atan2(r01, r11) : std::atan2(-r01, r11);
    }
    float *m = poses + (size_t)i * 6;
    m[0] = q[0], m[1] = q[1], m[2] = q[2];
    m[3] = (float)m3, m[4] = (float)m4, m[5] = (float)m5;
  }
  return GD_OK;
}

// ---------------------------------------------------------------------------
// Validation
// ---------------------------------------------------------------------------
extern "C" gd_status gd_complex_validate(const gd_complex *cx) {
  if (!cx) return fail(GD_EINVAL, "complex is NULL");
  const gd_ligand &L = cx->lig;
  const gd_protein &P = cx->prt;
  if (!cx->ff) return fail(GD_EINVAL, "force field is NULL");
  if (L.lna < 1 || L.lna > MAX_WARPS * MAX_NA || L.lna > MAX_LNA)
    return fail(GD_EINVAL, "ligand atoms lna=%d outside [1, %d]", L.lna,
                std::min(MAX_WARPS * MAX_NA, MAX_LNA));
  if (L.n_conf < 1) return fail(GD_EINVAL, "ligand conformations n_conf=%d", L.n_conf);
  if (!L.x || !L.y || !L.z || !L.t || !L.c || !L.n) return fail(GD_EINVAL, "ligand array NULL");
  if (P.pnp < 1 || P.n_conf < 1)
    return fail(GD_EINVAL, "protein pnp=%d n_conf=%d", P.pnp, P.n_conf);
  if (!P.x || !P.y || !P.z || !P.t || !P.c || !P.ele || !P.seq3r || !P.c0_and_d12_or_c2 || !P.hpp)
    return fail(GD_EINVAL, "protein array NULL");
  if (cx->psp.n_col < 1 || !cx->psp.psp) return fail(GD_EINVAL, "psp table missing");
  for (int a = 0; a < L.lna; ++a) {
    if (L.t[a] < 0 || L.t[a] >= GD_NLT)
      return fail(GD_EINVAL, "ligand atom %d type %d outside [0, %d)", a, L.t[a], GD_NLT);
    if (cx->mcs.pos > 0 && (L.n[a] < 0 || L.n[a] + 1 >= cx->mcs.n_field))
      return fail(GD_EINVAL, "ligand atom %d number %d: MCS field n+1 outside [0, %d)", a, L.n[a],
                  cx->mcs.n_field);
  }
  for (int p = 0; p < P.pnp; ++p) {
    if (P.t[p] < 0 || P.t[p] >= GD_NPT)
      return fail(GD_EINVAL, "protein point %d type %d outside [0, %d)", p, P.t[p], GD_NPT);
    if (P.c[p] < 0 || P.c[p] > 3) return fail(GD_EINVAL, "protein point %d class %d", p, P.c[p]);
    if (P.seq3r[p] < 0 || P.seq3r[p] >= cx->psp.n_col || P.seq3r[p] > MAX_SEQ3R)
      return fail(GD_EINVAL, "protein point %d seq3r %d outside [0, %d)", p, P.seq3r[p],
                  std::min(cx->psp.n_col, MAX_SEQ3R + 1));
  }
  if (cx->kde.pnk < 0) return fail(GD_EINVAL, "kde pnk=%d", cx->kde.pnk);
  if (cx->kde.pnk > 0) {
    if (!cx->kde.x || !cx->kde.y || !cx->kde.z || !cx->kde.t) return fail(GD_EINVAL, "kde NULL");
    for (int k = 0; k < cx->kde.pnk; ++k)
      if (cx->kde.t[k] < 0 || cx->kde.t[k] >= GD_NLT)
        return fail(GD_EINVAL, "kde point %d type %d", k, cx->kde.t[k]);
  }
  if (cx->mcs.pos < 0) return fail(GD_EINVAL, "mcs pos=%d", cx->mcs.pos);
  if (cx->mcs.pos > 0 && (!cx->mcs.x || !cx->mcs.y || !cx->mcs.z || !cx->mcs.tcc))
    return fail(GD_EINVAL, "mcs arrays NULL");
  return GD_OK;
}

// ---------------------------------------------------------------------------
// Context
// ---------------------------------------------------------------------------
extern "C" gd_status gd_ctx_create(int device, void *stream, gd_ctx **out) {
  if (!out) return fail(GD_EINVAL, "gd_ctx_create: out is NULL");
  *out = nullptr;
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0)
    return fail(GD_ENODEV, "no CUDA device (%s)", cudaGetErrorString(e));
  if (device < 0 || device >= n) return fail(GD_EINVAL, "device %d of %d", device, n);
  GD_CUDA(cudaSetDevice(device));
  // single attributes (cudaGetDeviceProperties queries them all: slow)
  int major = 0, minor = 0, n_sm = 0;
  GD_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
  GD_CUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
  GD_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device));
  if (major != 10)
    return fail(GD_ENODEV, "device %d is sm_%d%d; this build targets sm_100a", device, major,
                minor);
  gd_ctx *c = new (std::nothrow) gd_ctx;
  if (!c) return fail(GD_ENOMEM, "host allocation");
  c->device = device;
  c->n_sm = n_sm;
  if (stream) {
    c->stream = (cudaStream_t)stream;
  } else {
    e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      delete c;
      return fail(GD_ECUDA, "cudaStreamCreate: %s", cudaGetErrorString(e));
    }
    c->own_stream = true;
  }
  e = shared_attach(c);
  if (e != cudaSuccess) {
    if (c->own_stream) cudaStreamDestroy(c->stream);
    delete c;
    return fail(GD_ENOMEM, "pinned host memory: %s", cudaGetErrorString(e));
  }
  // the fixed scratch of gd_energy_poses_noalloc is committed now, not on
  // that entry point's first call
  const gd_status st = noalloc_attach(c);
  if (st != GD_OK) {
    shared_detach(c);
    if (c->own_stream) cudaStreamDestroy(c->stream);
    delete c;
    return st;
  }
  *out = c;
  return GD_OK;
}

extern "C" gd_status gd_ctx_destroy(gd_ctx *c) {
  ctx_release(c);
  return GD_OK;
}

extern "C" gd_status gd_ctx_sync(gd_ctx *c) {
  if (!c) return fail(GD_EINVAL, "ctx is NULL");
  GD_CUDA(cudaSetDevice(c->device));
  return ctx_check(c);
}

extern "C" uint64_t gd_ctx_launch_count(const gd_ctx *c) { return c ? c->launches : 0; }

// ---------------------------------------------------------------------------
// Device layout of a complex
// ---------------------------------------------------------------------------
// The tables of a complex, collected on the host and placed in one device
// allocation by one copy (a request's upload: 18 allocations and copies of a
// few hundred bytes to a few hundred KB took about 150 us).  Stream-ordered on
// the context stream: neither this nor the matching cudaFreeAsync in dcx_release
// synchronises the device, so a server uploading and releasing requests never
// stalls the kernels of other streams.
struct TableUpload {
  gd_dcomplex *d;
  std::vector<unsigned char> host;
  std::vector<std::pair<const void **, size_t>> at;  // pointer to set, offset
};

template <typename T>
static gd_status upload(TableUpload &U, const std::vector<T> &h, const T **out) {
  const size_t n = std::max<size_t>(h.size(), 1) * sizeof(T);
  const size_t o = (U.host.size() + 255) & ~size_t(255);
  U.host.resize(o + n);
  if (!h.empty()) std::memcpy(U.host.data() + o, h.data(), h.size() * sizeof(T));
  U.at.emplace_back(reinterpret_cast<const void **>(out), o);
  U.d->bytes += n;
  return GD_OK;
}

static gd_status upload_finish(TableUpload &U) {
  gd_ctx *c = U.d->ctx;
  const auto injected = [&] {
    return fail(GD_ENOMEM, "cudaMallocAsync of %zu bytes: out of memory (injected)",
                U.host.size());
  };
  unsigned char *p = nullptr;
  if (injected_alloc_failure(c)) return injected();
  GD_CUDA(cudaMallocAsync((void **)&p, U.host.size(), c->stream));
  U.d->allocs.push_back(p);
  for (const auto &x : U.at) {
    // each table counts as an allocation: a failure with the memory taken
    if (injected_alloc_failure(c)) return injected();
    *x.first = p + x.second;
  }
  GD_CUDA(cudaMemcpyAsync(p, U.host.data(), U.host.size(), cudaMemcpyHostToDevice, c->stream));
  return GD_OK;
}

extern "C" gd_status gd_complex_free(gd_dcomplex *d) {
  dcx_release(d);
  return GD_OK;
}

extern "C" size_t gd_complex_device_bytes(const gd_dcomplex *d) { return d ? d->bytes : 0; }

// Packs the protein conformations into {x, y, z, ele} and {hpp, meta}.
// The device order of the points: those whose type forms an H-bond with
// some ligand type (hdb0 > 0.1) first, each kind in the caller's order.  The
// energy is a sum over points, so the order changes nothing but the FP32
// rounding inside a 32-point chunk.
static gd_status upload_protein(const gd_protein &P, const gd_enepara &F, TableUpload &U) {
  gd_dcomplex *d = U.d;
  KTables &T = d->T;
  const int pnp = P.pnp;
  const int pnp_pad = (pnp + TILE_PTS - 1) / TILE_PTS * TILE_PTS;
  bool hb_type[GD_NPT];
  for (int j = 0; j < GD_NPT; ++j) {
    hb_type[j] = false;
    for (int i = 0; i < GD_NLT; ++i) hb_type[j] = hb_type[j] || F.hdb0[i][j] > 0.1f;
  }
  std::vector<int> &order = d->point_order;
  order.clear();
  order.reserve(pnp);
  for (int pass = 0; pass < 2; ++pass)
    for (int p = 0; p < pnp; ++p)
      if (hb_type[P.t[p]] == (pass == 0)) order.push_back(p);
  std::vector<float4> pa((size_t)P.n_conf * pnp_pad,
                         make_float4(PAD_POINT_COORD, PAD_POINT_COORD, PAD_POINT_COORD, 0.f));
  for (int c = 0; c < P.n_conf; ++c)
    for (int s = 0; s < pnp; ++s) {
      const int p = order[s];
      const size_t i = (size_t)c * pnp + p;
      pa[(size_t)c * pnp_pad + s] = make_float4(P.x[i], P.y[i], P.z[i], P.ele[p]);
    }
  float pad_meta;
  {
    const uint32_t m = (uint32_t)PAD_POINT_TYPE;
    std::memcpy(&pad_meta, &m, 4);
  }
  std::vector<float2> pb((size_t)pnp_pad, make_float2(0.f, pad_meta));
  for (int s = 0; s < pnp; ++s) {
    const int p = order[s];
    uint32_t meta = (uint32_t)P.t[p] | ((uint32_t)P.c[p] << META_CLASS_SHIFT) |
                    ((uint32_t)P.seq3r[p] << META_SEQ_SHIFT);
    if (P.c0_and_d12_or_c2[p] == 1) meta |= META_HPC_BIT;
    float mf;
    std::memcpy(&mf, &meta, 4);
    pb[s] = make_float2(P.hpp[p], mf);
  }
  GD_TRY(upload(U, pa, &T.pt_a));
  GD_TRY(upload(U, pb, &T.pt_b));
  T.pnp = pnp;
  T.pnp_pad = pnp_pad;
  T.n_prt = P.n_conf;
  return GD_OK;
}

// The distance from which the kernel's far form holds for a ligand type i and
// a point type j (infinity: never), each bound solved from the term itself:
// - contact PMF pmf1 / (1 + e), e = exp((6 - d/2)(d - pmf0)): from where
//   e <= exp(-18) < 2^-25, 1 + e rounds to 1 in FP32 and the term is pmf1;
// - H-bond hdb1 exp(-h^2/2), h = (d - hdb0) hdb1: exactly zero in FP32 from
//   h = 13.3 on (the argument of 2^x is below -127, and the kernel's 2^x gives 0
//   below -126).  A bound at a small value would not do: a chunk whose other
//   points have no H-bond term starts its sum at 0, and sees any value;
// - near-field electrostatics (el1 d < 1), hydrophobic contact (9 A) and the
//   contact tests (d <= pmf0) are over.
static float far_distance(const gd_enepara &F, int i, int j, float max_pmf0) {
  const double inf = std::numeric_limits<double>::infinity();
  const double p0 = F.pmf0[i][j];
  double D = std::max(9.0, (double)max_pmf0);
  D = std::max(D, F.el1 > 0.f ? 1.0 / (double)F.el1 : inf);
  D = std::max(D, 0.5 * (12.0 + p0 + std::sqrt((12.0 - p0) * (12.0 - p0) + 144.0)));
  if (F.hdb0[i][j] > 0.1f)
    D = std::max(D, F.hdb1[i][j] > 0.f ? (double)F.hdb0[i][j] + 13.3 / (double)F.hdb1[i][j] : inf);
  D = D * 1.0005 + 0.01;  // rounding of the distances compared with it
  return std::isfinite(p0) && D < 1e6 ? (float)D : std::numeric_limits<float>::infinity();
}

// gd_dcomplex.far_share, of protein conformation pc.
static double far_share_of(const gd_complex *cx, int pc) {
  const gd_ligand &L = cx->lig;
  const gd_protein &P = cx->prt;
  const gd_enepara &F = *cx->ff;
  float max_pmf0 = 0.f, reach2 = 0.f;
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) max_pmf0 = std::max(max_pmf0, F.pmf0[i][j]);
  bool present[GD_NLT] = {};
  for (int a = 0; a < L.lna; ++a) {
    present[L.t[a]] = true;
    reach2 = std::max(reach2, L.x[a] * L.x[a] + L.y[a] * L.y[a] + L.z[a] * L.z[a]);
  }
  float far2[GD_NPT];
  for (int j = 0; j < GD_NPT; ++j) {
    float d = 0.f;
    for (int i = 0; i < GD_NLT; ++i)
      if (present[i]) d = std::max(d, far_distance(F, i, j, max_pmf0));
    d += std::sqrt(reach2);
    far2[j] = d * d;
  }
  int n = 0;
  for (int p = 0; p < P.pnp; ++p) {
    const size_t i = (size_t)pc * P.pnp + p;
    const float dx = P.x[i] - L.center[0], dy = P.y[i] - L.center[1], dz = P.z[i] - L.center[2];
    n += dx * dx + dy * dy + dz * dz > far2[P.t[p]];
  }
  return (double)n / P.pnp;
}

// Ligand, pocket template and force-field tables of a complex.
static gd_status upload_ligand(const gd_complex *cx, TableUpload &U) {
  gd_dcomplex *d = U.d;
  const gd_ligand &L = cx->lig;
  const gd_enepara &F = *cx->ff;
  KTables &T = d->T;
  const int lna = L.lna;
  // type-pair table [lig type][point type], plus an all-zero row for the
  // padding atoms of the last atom group
  std::vector<float4> ta(TAB_ROWS * GD_NPT, make_float4(0.f, 0.f, 0.f, 0.f));
  std::vector<float2> tb(TAB_ROWS * GD_NPT, make_float2(0.f, 0.f));
  float max_pmf0 = 0.f;
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) {
      ta[i * GD_NPT + j] = make_float4(F.p1a[i][j], F.p2a[i][j], F.pmf0[i][j], F.pmf1[i][j]);
      tb[i * GD_NPT + j] = make_float2(F.hdb0[i][j], F.hdb1[i][j]);
      max_pmf0 = std::max(max_pmf0, F.pmf0[i][j]);
    }
  // padding atoms (the last row) bound nothing
  std::vector<float> tf(TAB_ROWS * GD_NPT, 0.f);
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) tf[i * GD_NPT + j] = far_distance(F, i, j, max_pmf0);
  std::vector<float4> lg((size_t)L.n_conf * lna);
  for (size_t i = 0; i < lg.size(); ++i) lg[i] = make_float4(L.x[i], L.y[i], L.z[i], 0.f);
  std::vector<int> lt(L.t, L.t + lna);
  std::vector<float> lq(L.c, L.c + lna);
  std::vector<float> psp(cx->psp.psp, cx->psp.psp + (size_t)GD_NLT * cx->psp.n_col);
  // KDE points bucketed by ligand type
  std::vector<int> koff(GD_NLT + 1, 0);
  for (int k = 0; k < cx->kde.pnk; ++k) koff[cx->kde.t[k] + 1] += 1;
  for (int i = 0; i < GD_NLT; ++i) koff[i + 1] += koff[i];
  std::vector<KdeRange> kof(GD_NLT);
  for (int i = 0; i < GD_NLT; ++i)
    kof[i] = {koff[i], koff[i + 1], 1.0 / (double)std::max(1, koff[i + 1] - koff[i])};
  std::vector<float4> kd((size_t)cx->kde.pnk);
  {
    std::vector<int> fill(koff.begin(), koff.end() - 1);
    for (int k = 0; k < cx->kde.pnk; ++k)
      kd[fill[cx->kde.t[k]]++] = make_float4(cx->kde.x[k], cx->kde.y[k], cx->kde.z[k], 0.f);
  }
  // MCS gathered per ligand atom: field n + 1 (calcenergy_d.cu:240-241)
  const int pos = cx->mcs.pos;
  std::vector<float4> mc((size_t)pos * lna);
  std::vector<double2> mw(pos);
  for (int m = 0; m < pos; ++m) {
    int c = 0;
    for (int a = 0; a < lna; ++a) {
      const size_t f = (size_t)m * cx->mcs.n_field + L.n[a] + 1;
      const bool valid = cx->mcs.x[f] != GD_MCS_INVALID_COORD;
      mc[(size_t)m * lna + a] =
          make_float4(cx->mcs.x[f], cx->mcs.y[f], cx->mcs.z[f], valid ? 1.f : 0.f);
      c += valid;
    }
    // no valid atom: 0 x inf = NaN, as the reference's 0 / 0
    mw[m] = make_double2((double)cx->mcs.tcc[m], 1.0 / (double)c);
  }
  GD_TRY(upload(U, ta, &T.tab_a));
  GD_TRY(upload(U, tb, &T.tab_b));
  GD_TRY(upload(U, tf, &T.tab_far));
  GD_TRY(upload(U, lg, &T.lig));
  GD_TRY(upload(U, lt, &T.lig_t));
  GD_TRY(upload(U, lq, &T.lig_q));
  GD_TRY(upload(U, psp, &T.psp));
  {
    // residues where some atom type of this ligand has a nonzero psp entry:
    // the kernel reads the table only there (elsewhere it adds zero)
    const int n_col = cx->psp.n_col;
    bool present[GD_NLT] = {};
    for (int a = 0; a < lna; ++a) present[L.t[a]] = true;
    std::vector<uint32_t> mask((size_t)(n_col + 31) / 32, 0u);
    for (int t = 0; t < GD_NLT; ++t)
      if (present[t])
        for (int r = 0; r < n_col; ++r)
          if (psp[(size_t)t * n_col + r] != 0.0f) mask[r >> 5] |= 1u << (r & 31);
    GD_TRY(upload(U, mask, &T.psp_mask));
  }
  GD_TRY(upload(U, kd, &T.kde));
  GD_TRY(upload(U, kof, &T.kde_of));
  GD_TRY(upload(U, mc, &T.mcs));
  GD_TRY(upload(U, mw, &T.mcs_w));

  T.lna = lna;
  T.n_lig = L.n_conf;
  T.pos = pos;
  T.psp_ncol = cx->psp.n_col;
  T.lj0 = F.lj0;
  T.lj0lj1 = F.lj0 * F.lj1;
  T.el0 = F.el0;
  T.el1 = F.el1;
  T.inv_el1 = 1.0f / F.el1;
  T.a1 = F.a1;
  T.b1 = F.b1;
  T.kde2 = F.kde2;
  T.kde3 = F.kde3;
  T.inv_lna = 1.0 / (double)lna;
  T.inv_pos = 1.0 / (double)pos;  // no records: 0 x inf = NaN, as 0 / 0
  T.inv_kde3 = 1.0 / (double)F.kde3;
  T.inv_s2pi = 1.0 / (double)sqrtf(2.0f * kPI);
  // the close-range terms fire inside these distances: near-field
  // electrostatics el1 d < 1 (every point), hydrophobic d <= 9 (points with
  // the hpc flag), psp d <= pmf0 (class-2 points); thresholds by point kind
  // (hpc flag | class 2 << 1), squared with a margin for rounding
  const float r_ele = F.el1 > 0.f ? 1.0f / F.el1 : 1e30f;
  for (int kind = 0; kind < 4; ++kind) {
    float r = r_ele;
    if (kind & 1) r = std::max(r, 9.0f);
    if (kind & 2) r = std::max(r, max_pmf0);
    T.near4[kind] = r * r * 1.0001f + 1e-3f;
  }
  T.near_ele2 = F.el1 > 0.f ? r_ele * r_ele * 1.0001f + 1e-3f : 1e30f;
  // kernel slot order: atoms with an H-bond term (some point type with
  // hdb0 > 0.1) first, so that they share atom pairs and warps
  std::vector<int> order;
  T.n_hb = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int a = 0; a < lna; ++a) {
      bool hb = false;
      for (int j = 0; j < GD_NPT; ++j) hb = hb || F.hdb0[L.t[a]][j] > 0.1f;
      if (hb == (pass == 0)) order.push_back(a);
      if (hb && pass == 0) ++T.n_hb;
    }
  GD_TRY(upload(U, order, &T.lig_order));
  for (int i = 0; i < GD_NLT; ++i) {
    T.hpl0[i] = F.hpl0[i];
    T.hpl1[i] = F.hpl1[i];
    T.hpl2[i] = F.hpl2[i];
  }
  for (int i = 0; i < GD_NTERM; ++i) {
    T.a_para[i] = F.a_para[i];
    T.b_para[i] = F.b_para[i];
    T.w[i] = F.w[i];
  }
  for (int i = 0; i < 3; ++i) {
    T.lig_center[i] = L.center[i];
    T.pocket[i] = cx->prt.pocket_center[i];
  }
  return GD_OK;
}

// Reference contact map of the MCC score (InitRefMatrix_d,
// calcmcc_d.cu:57-83): pairs with dst <= pmf0 for ligand conformation 0 in
// its start pose (relative coordinates + centre, util.C:230-247) against the
// complex's first protein conformation, in the reference's single-precision
// order; one bit per (atom, point), rows of pnp_pad / 32 words.
static gd_status upload_mcc_ref(const gd_complex *cx, int prt_conf, TableUpload &U) {
  gd_dcomplex *d = U.d;
  const gd_ligand &L = cx->lig;
  const gd_protein &P = cx->prt;
  const gd_enepara &F = *cx->ff;
  KTables &T = d->T;
  const int words = T.pnp_pad / 32;
  const int pc = prt_conf < P.n_conf ? prt_conf : 0;
  // bits are indexed by the device position of a point
  const std::vector<int> &order =
      d->protein_owner ? d->protein_owner->point_order : d->point_order;
  if ((int)order.size() != P.pnp) return fail(GD_EINVAL, "protein point order missing");
  std::vector<uint32_t> bits((size_t)L.lna * words, 0u);
  int nref = 0;
  float max_pmf0 = 0.f;
  for (int i = 0; i < GD_NLT; ++i)
    for (int j = 0; j < GD_NPT; ++j) max_pmf0 = std::max(max_pmf0, F.pmf0[i][j]);
  T.near_mcc2 = max_pmf0 * max_pmf0 * 1.0001f + 1e-3f;
  // points within reach of the ligand's box (the others have no contact)
  float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
  std::vector<float> at((size_t)L.lna * 3);
  for (int a = 0; a < L.lna; ++a) {
    const float v[3] = {L.x[a] + L.center[0], L.y[a] + L.center[1], L.z[a] + L.center[2]};
    for (int k = 0; k < 3; ++k) {
      at[(size_t)a * 3 + k] = v[k];
      lo[k] = std::min(lo[k], v[k]);
      hi[k] = std::max(hi[k], v[k]);
    }
  }
  for (int s = 0; s < P.pnp; ++s) {
    const int p = order[s];
    const size_t i = (size_t)pc * P.pnp + p;
    const float px = P.x[i], py = P.y[i], pz = P.z[i];
    const float bx = std::max(0.f, std::max(lo[0] - px, px - hi[0]));
    const float by = std::max(0.f, std::max(lo[1] - py, py - hi[1]));
    const float bz = std::max(0.f, std::max(lo[2] - pz, pz - hi[2]));
    if (bx * bx + by * by + bz * bz > T.near_mcc2) continue;
    for (int a = 0; a < L.lna; ++a) {
      const float dx = at[(size_t)a * 3] - px;
      const float dy = at[(size_t)a * 3 + 1] - py;
      const float dz = at[(size_t)a * 3 + 2] - pz;
      const float dst = sqrtf(dx * dx + dy * dy + dz * dz);
      if (dst <= F.pmf0[L.t[a]][P.t[p]]) {
        bits[(size_t)a * words + (s >> 5)] |= 1u << (s & 31);
        ++nref;
      }
    }
  }
  GD_TRY(upload(U, bits, &T.mcc_ref));
  T.mcc_words = words;
  T.mcc_nref = (float)nref;
  return GD_OK;
}

static gd_status complex_upload_common(gd_ctx *ctx, const gd_complex *cx,
                                       const gd_dcomplex *share, int prt_conf0, int n_prt,
                                       gd_dcomplex **out) {
  if (!ctx || !out) return fail(GD_EINVAL, "gd_complex_upload: NULL argument");
  *out = nullptr;
  GD_TRY(gd_complex_validate(cx));
  if (share) {
    if (share->ctx != ctx) return fail(GD_EINVAL, "shared protein belongs to another context");
    if (share->T.pnp != cx->prt.pnp)
      return fail(GD_EINVAL, "shared protein has %d points, complex %d", share->T.pnp,
                  cx->prt.pnp);
    if (prt_conf0 < 0 || n_prt < 1 || prt_conf0 + n_prt > share->T.n_prt)
      return fail(GD_EINVAL, "conformations [%d, %d) outside the shared protein's %d", prt_conf0,
                  prt_conf0 + n_prt, share->T.n_prt);
  }
  GD_CUDA(cudaSetDevice(ctx->device));
  gd_dcomplex *d = new (std::nothrow) gd_dcomplex;
  if (!d) return fail(GD_ENOMEM, "host allocation");
  d->ctx = ctx;
  ctx_retain(ctx);
  gd_status st = GD_OK;
  try {
    TableUpload U{d, {}, {}};
    if (share) {
      d->protein_owner = const_cast<gd_dcomplex *>(share);
      dcx_retain(d->protein_owner);
      d->T.pt_a = share->T.pt_a + (size_t)prt_conf0 * share->T.pnp_pad;
      d->T.pt_b = share->T.pt_b;
      d->T.pnp = share->T.pnp;
      d->T.pnp_pad = share->T.pnp_pad;
      d->T.n_prt = n_prt;
    } else {
      st = upload_protein(cx->prt, *cx->ff, U);
    }
    if (st == GD_OK) st = upload_ligand(cx, U);
    if (st == GD_OK) st = upload_mcc_ref(cx, share ? prt_conf0 : 0, U);
    d->far_share = far_share_of(cx, share ? prt_conf0 : 0);
    if (st == GD_OK) st = upload_finish(U);
    if (st == GD_OK) {
      cudaError_t e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) st = fail(GD_ECUDA, "upload: %s", cudaGetErrorString(e));
    }
  } catch (const std::bad_alloc &) {
    st = fail(GD_ENOMEM, "host allocation while packing the complex");
  }
  if (st != GD_OK) {
    dcx_release(d);
    return st;
  }
  *out = d;
  return GD_OK;
}

extern "C" gd_status gd_complex_upload(gd_ctx *ctx, const gd_complex *cx, gd_dcomplex **out) {
  NvtxRange nvtx("gd_complex_upload");
  return complex_upload_common(ctx, cx, nullptr, 0, 0, out);
}

extern "C" gd_status gd_complex_upload_shared(gd_ctx *ctx, const gd_complex *cx,
                                              const gd_dcomplex *protein, int prt_conf0,
                                              int n_prt, gd_dcomplex **out) {
  if (!protein) return fail(GD_EINVAL, "gd_complex_upload_shared: protein is NULL");
  return complex_upload_common(ctx, cx, protein, prt_conf0, n_prt, out);
}

// ---------------------------------------------------------------------------
// Pose energies
// ---------------------------------------------------------------------------
// The unit of a small call: with few poses the launch would leave most SMs
// idle, so a unit's points are split over a cluster (as MC units, split_rule),
// and then the poses over more units of 16 or 8 poses (lane packing).
static void pose_units(gd_ctx *ctx, const KTables &T, int n_pose, int *split, int *packed) {
  int per = 32;
  auto units = [&](int p) { return (n_pose + p - 1) / p; };
  *split = split_rule(ctx, T, units(32), kRunSplitCost);
  while (per > 8 && units(per / 2) > units(per) && units(per / 2) * *split <= ctx->n_sm) per /= 2;
  *packed = per < 32 ? per : 0;
}

gd_status gd::poses_launch(gd_ctx *ctx, const gd_dcomplex *d, int prt_conf, int lig_conf,
                           int n_pose, const float *poses, float *terms, double *raw,
                           void *work) {
  const Tile tile = tile_for(ctx, d->T);
  KRun R{};
  R.mode = KMODE_POSES;
  R.A = tile.A;
  R.P = tile.P;
  R.prt_conf = prt_conf;
  R.lig_conf = lig_conf;
  R.n_pose = n_pose;
  R.poses = poses;
  R.terms = terms;
  R.raw = raw;
  R.err = ctx->h_err;
  R.hb_pairs = hb_pairs_of(d->T, tile.A);
  R.pose_item.T = d->T;
  R.pose_item.n_tmp = 1;
  R.pose_item.n_lig_conf = d->T.n_lig;
  R.pose_item.n_prt = d->T.n_prt;
  int grid = 0;
  if (work) {
    int launches = 0;
    GD_CUDA(pose_cells(&R, work, &grid, &launches, ctx->stream));
    ctx->launches += launches;
  } else {
    pose_units(ctx, d->T, n_pose, &R.split, &R.packed);
    const int per = R.packed ? R.packed : 32;
    grid = (n_pose + per - 1) / per * R.split;
  }
  pick_stages(d->T, tile, &R.n_stages, &R.resident, std::max(1, R.split),
              R.packed != 0 || R.pose_grid != nullptr);
  GD_CUDA(launch_dock(R, tile.NA, grid, ctx->stream));
  ctx->launches += 1;
  return GD_OK;
}

static gd_status check_confs(const gd_dcomplex *d, int prt_conf, int lig_conf) {
  if (prt_conf < 0 || prt_conf >= d->T.n_prt)
    return fail(GD_EINVAL, "prt_conf %d outside [0, %d)", prt_conf, d->T.n_prt);
  if (lig_conf < 0 || lig_conf >= d->T.n_lig)
    return fail(GD_EINVAL, "lig_conf %d outside [0, %d)", lig_conf, d->T.n_lig);
  return GD_OK;
}

static size_t cell_bytes(const gd_ctx *ctx, const gd_dcomplex *d, int n_pose) {
  return pose_work_bytes(d->T, d->far_share, ctx->n_sm, n_pose);
}

// A checked pose call on device pointers, with the call's workspace.
static gd_status poses_dev(gd_ctx *ctx, const gd_dcomplex *d, int prt_conf, int lig_conf,
                           int n_pose, const float *poses, float *terms, double *raw,
                           Workspace &W) {
  void *work = nullptr;
  const size_t bytes = cell_bytes(ctx, d, n_pose);
  // without room for the cells' workspace the call runs without them
  if (bytes && W.get(&work, bytes) != cudaSuccess) cudaGetLastError();
  return poses_launch(ctx, d, prt_conf, lig_conf, n_pose, poses, terms, raw, work);
}

extern "C" gd_status gd_energy_poses_dev(gd_ctx *ctx, const gd_dcomplex *d, int prt_conf,
                                         int lig_conf, int n_pose, const float *poses,
                                         float *terms, double *raw) {
  NvtxRange nvtx("gd_energy_poses_dev");
  if (!ctx || !d) return fail(GD_EINVAL, "gd_energy_poses_dev: NULL handle");
  if (n_pose < 0) return fail(GD_EINVAL, "n_pose=%d", n_pose);
  GD_TRY(check_confs(d, prt_conf, lig_conf));
  if (n_pose == 0) return GD_OK;
  if (!poses || !terms) return fail(GD_EINVAL, "poses/terms NULL");
  GD_CUDA(cudaSetDevice(ctx->device));
  Workspace W(ctx, cell_bytes(ctx, d, n_pose));
  return poses_dev(ctx, d, prt_conf, lig_conf, n_pose, poses, terms, raw, W);
}

extern "C" gd_status gd_energy_poses(gd_ctx *ctx, const gd_dcomplex *d, int prt_conf,
                                     int lig_conf, int n_pose, const float *poses, float *terms,
                                     double *raw) {
  if (!ctx || !d) return fail(GD_EINVAL, "gd_energy_poses: NULL handle");
  if (n_pose < 0) return fail(GD_EINVAL, "n_pose=%d", n_pose);
  if (n_pose == 0) return GD_OK;
  if (!poses || !terms) return fail(GD_EINVAL, "poses/terms NULL");
  GD_CUDA(cudaSetDevice(ctx->device));
  const size_t pose_b = sizeof(float) * 6 * (size_t)n_pose;
  const size_t term_b = sizeof(float) * GD_NTERM * (size_t)n_pose;
  const size_t raw_b = raw ? sizeof(double) * GD_NRAW * (size_t)n_pose : 0;
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t total = up(pose_b) + up(term_b) + raw_b;
  // a small call passes through the context's pinned memory, which the kernel
  // reads and writes directly: no allocation and no copy in the stream
  if (total <= kStageBytes && cell_bytes(ctx, d, n_pose) == 0) {
    std::unique_lock<std::mutex> lk(ctx->stage_mu, std::try_to_lock);
    if (lk.owns_lock()) {
      unsigned char *p = ctx->stage;
      std::memcpy(p, poses, pose_b);
      const gd_status st = gd_energy_poses_dev(
          ctx, d, prt_conf, lig_conf, n_pose, reinterpret_cast<float *>(p),
          reinterpret_cast<float *>(p + up(pose_b)),
          raw ? reinterpret_cast<double *>(p + up(pose_b) + up(term_b)) : nullptr);
      if (st != GD_OK) return st;
      GD_TRY(ctx_check(ctx));
      std::memcpy(terms, p + up(pose_b), term_b);
      if (raw) std::memcpy(raw, p + up(pose_b) + up(term_b), raw_b);
      return GD_OK;
    }
  }
  GD_TRY(check_confs(d, prt_conf, lig_conf));
  gd_status st = GD_OK;
  {
    // (a workspace that is not kept is given back before the call's last wait)
    Workspace W(ctx, Workspace::padded(total) + cell_bytes(ctx, d, n_pose));
    unsigned char *p = nullptr;
    cudaError_t e = W.get((void **)&p, total);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(p, poses, pose_b, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) {
      st = fail(GD_ENOMEM, "pose buffers: %s", cudaGetErrorString(e));
    } else {
      float *dt = reinterpret_cast<float *>(p + up(pose_b));
      double *dr = raw ? reinterpret_cast<double *>(p + up(pose_b) + up(term_b)) : nullptr;
      st = poses_dev(ctx, d, prt_conf, lig_conf, n_pose, reinterpret_cast<float *>(p), dt, dr, W);
      if (st == GD_OK) {
        e = cudaMemcpyAsync(terms, dt, term_b, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess && raw)
          e = cudaMemcpyAsync(raw, dr, raw_b, cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess) st = fail(GD_ECUDA, "copy back: %s", cudaGetErrorString(e));
      }
    }
  }
  if (st != GD_OK) {
    cudaStreamSynchronize(ctx->stream);
    return st;
  }
  return ctx_check(ctx);
}

extern "C" gd_status gd_ctx_set_tile(gd_ctx *ctx, int lna, int pnp, const gd_tile *tile) {
  if (!ctx || !tile) return fail(GD_EINVAL, "gd_ctx_set_tile: NULL argument");
  Tile t;
  t.A = tile->atom_groups;
  t.P = tile->tile_groups;
  t.NA = tile->atoms_per_warp;
  if (!t.valid() || t.A * t.P > MAX_WARPS || round_na(t.NA) != t.NA ||
      t.A * t.NA < lna_bucket(lna))
    return fail(GD_EINVAL, "tile %dx%d with %d atoms per warp does not cover %d atoms", t.A, t.P,
                t.NA, lna);
  std::lock_guard<std::mutex> g(ctx->tile_mu);
  ctx->tiles[{lna_bucket(lna), (pnp + TILE_PTS - 1) / TILE_PTS}] = t;
  return GD_OK;
}

extern "C" gd_status gd_ctx_set_schedule(gd_ctx *ctx, int mode, int machines) {
  if (!ctx) return fail(GD_EINVAL, "gd_ctx_set_schedule: NULL context");
  if (mode < GD_SCHED_AUTO || mode > GD_SCHED_PERSISTENT)
    return fail(GD_EINVAL, "gd_ctx_set_schedule: unknown mode %d", mode);
  if (machines < 0) return fail(GD_EINVAL, "gd_ctx_set_schedule: machines=%d", machines);
  ctx->sched_mode = mode;
  ctx->sched_machines = machines;
  return GD_OK;
}

extern "C" gd_status gd_ctx_set_schedule_tail(gd_ctx *ctx, int tail) {
  if (!ctx) return fail(GD_EINVAL, "gd_ctx_set_schedule_tail: NULL context");
  if (tail < 0 || tail > 64) return fail(GD_EINVAL, "gd_ctx_set_schedule_tail: tail=%d", tail);
  ctx->sched_tail = tail;
  return GD_OK;
}

extern "C" gd_status gd_ctx_set_split(gd_ctx *ctx, int split) {
  if (!ctx) return fail(GD_EINVAL, "gd_ctx_set_split: NULL context");
  if (split < 0 || split > 8 || (split & (split - 1)))
    return fail(GD_EINVAL, "gd_ctx_set_split: %d is not 0, 1, 2, 4 or 8", split);
  ctx->split_mode = split;
  return GD_OK;
}

extern "C" gd_status gd_ctx_set_wait_test(gd_ctx *c, unsigned wait_limit, int never_release) {
  if (!c) return fail(GD_EINVAL, "ctx is NULL");
  if (never_release && wait_limit == 0)
    return fail(GD_EINVAL, "gd_ctx_set_wait_test: never_release needs a wait limit");
  c->wait_limit = wait_limit;
  // no run reaches this many MC steps, so a wait for it can only run out
  c->wait_bias = never_release ? (1 << 30) : 0;
  return GD_OK;
}

extern "C" gd_status gd_ctx_set_alloc_fail(gd_ctx *c, int nth) {
  if (!c) return fail(GD_EINVAL, "ctx is NULL");
  if (nth < 0) return fail(GD_EINVAL, "gd_ctx_set_alloc_fail: nth=%d", nth);
  c->alloc_fail_in.store(nth);
  return GD_OK;
}

extern "C" gd_status gd_schedule_queue(const double *cost, const int *steps, int n_units,
                                       int machines, int tail, int *pieces, int cap,
                                       int *piece_off, int *n_queue) {
  if (n_units < 0 || machines < 1 || tail < 0 || cap < 0 || !piece_off || !n_queue ||
      (n_units > 0 && (!cost || !steps || !pieces)))
    return fail(GD_EINVAL, "gd_schedule_queue: bad arguments");
  std::vector<double> c(cost, cost + n_units);
  std::vector<int> s(steps, steps + n_units);
  for (int u = 0; u < n_units; ++u)
    if (!(c[u] > 0.0) || s[u] < 0)
      return fail(GD_EINVAL, "gd_schedule_queue: unit %d has cost %g, %d steps", u, c[u], s[u]);
  std::vector<int4> pc;
  std::vector<int> off;
  int nq = 0;
  schedule_queue(c, s, machines, tail, &pc, &off, &nq);
  if ((int)pc.size() > cap)
    return fail(GD_EINVAL, "gd_schedule_queue: %zu pieces exceed cap %d", pc.size(), cap);
  for (size_t k = 0; k < pc.size(); ++k) {
    pieces[4 * k] = pc[k].x;
    pieces[4 * k + 1] = pc[k].y;
    pieces[4 * k + 2] = pc[k].z;
    pieces[4 * k + 3] = pc[k].w;
  }
  for (int k = 0; k <= machines; ++k) piece_off[k] = off[k];
  *n_queue = nq;
  return GD_OK;
}

extern "C" gd_status gd_schedule_pieces(const double *cost, const int *steps, int n_units,
                                        int machines, int *pieces, int cap, int *piece_off,
                                        int *n_used) {
  if (n_units < 0 || machines < 1 || cap < 0 || !piece_off || !n_used ||
      (n_units > 0 && (!cost || !steps || !pieces)))
    return fail(GD_EINVAL, "gd_schedule_pieces: bad arguments");
  std::vector<double> c(cost, cost + n_units);
  std::vector<int> s(steps, steps + n_units);
  for (int u = 0; u < n_units; ++u)
    if (!(c[u] > 0.0) || s[u] < 0)
      return fail(GD_EINVAL, "gd_schedule_pieces: unit %d has cost %g, %d steps", u, c[u], s[u]);
  std::vector<int4> pc;
  std::vector<int> off;
  const int used = schedule_pieces(c, s, machines, &pc, &off);
  if ((int)pc.size() > cap)
    return fail(GD_EINVAL, "gd_schedule_pieces: %zu pieces exceed cap %d", pc.size(), cap);
  for (size_t k = 0; k < pc.size(); ++k) {
    pieces[4 * k] = pc[k].x;
    pieces[4 * k + 1] = pc[k].y;
    pieces[4 * k + 2] = pc[k].z;
    pieces[4 * k + 3] = pc[k].w;
  }
  for (int m = 0; m <= used; ++m) piece_off[m] = off[m];
  *n_used = used;
  return GD_OK;
}

namespace gd {

int schedule_pieces(const std::vector<double> &cost, const std::vector<int> &steps, int m,
                    std::vector<int4> *pieces, std::vector<int> *piece_off) {
  pieces->clear();
  piece_off->assign(1, 0);
  double total = 0.0, longest = 0.0;
  for (size_t u = 0; u < cost.size(); ++u) {
    const double p = cost[u] * std::max(steps[u], 0);
    total += p;
    longest = std::max(longest, p);
  }
  if (total <= 0.0 || m < 1) return 0;
  const double C = std::max(longest, total / m);
  // line order: machine k holds [k C, (k+1) C) of the units laid end to end
  std::vector<std::vector<int4>> mach(1);
  double pos = 0.0;  // line length placed so far (cuts are rounded against
                     // the ideal boundaries, so rounding does not accumulate)
  for (size_t u = 0; u < cost.size(); ++u) {
    const int n = steps[u];
    const double c = cost[u];
    int lo = 0;
    while (lo < n) {
      const double end = C * (double)mach.size();  // this machine's boundary
      int s = (int)std::floor((end - pos) / c + 0.5);  // steps that fit, rounded
      if (s >= n - lo || (int)mach.size() == m) s = n - lo;
      if (s <= 0) {  // the machine is full: the unit starts the next one
        mach.emplace_back();
        continue;
      }
      mach.back().push_back(make_int4((int)u, lo, lo + s, lo > 0 ? 1 : 0));
      lo += s;
      pos += s * c;
      if (lo < n) mach.emplace_back();  // cut: the rest opens the next machine
    }
  }
  while (!mach.empty() && mach.back().empty()) mach.pop_back();
  // run order is the reverse of line order: a cut unit's first steps open
  // the lower machine, its last steps close the next one
  for (auto &v : mach) {
    for (auto p = v.rbegin(); p != v.rend(); ++p) pieces->push_back(*p);
    piece_off->push_back((int)pieces->size());
  }
  return (int)mach.size();
}

int schedule_queue(const std::vector<double> &cost, const std::vector<int> &steps, int m, int tail,
                   std::vector<int4> *pieces, std::vector<int> *piece_off, int *n_queue) {
  const size_t n = cost.size();
  std::vector<int> head(n);
  for (size_t u = 0; u < n; ++u) head[u] = std::max(0, steps[u] - std::max(tail, 0));
  const int used = schedule_pieces(cost, head, m, pieces, piece_off);
  // when each unit's first part ends, along its machine's list (cost units)
  std::vector<double> ready(n, 0.0);
  for (int k = 0; k < used; ++k) {
    double t = 0.0;
    for (int q = (*piece_off)[k]; q < (*piece_off)[k + 1]; ++q) {
      const int4 &pz = (*pieces)[q];
      t += cost[pz.x] * (pz.z - pz.y);
      if (pz.z == head[pz.x]) ready[pz.x] = t;
    }
  }
  while ((int)piece_off->size() < m + 1) piece_off->push_back(piece_off->back());
  std::vector<int> order(n);
  for (size_t u = 0; u < n; ++u) order[u] = (int)u;
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return ready[a] < ready[b]; });
  *n_queue = 0;
  for (int j = 0; j < tail; ++j)
    for (int u : order)
      if (head[u] + j < steps[u]) {
        const int lo = head[u] + j;
        pieces->push_back(make_int4(u, lo, lo + 1, lo > 0 ? 1 : 0));
        *n_queue += 1;
      }
  return m;
}

}  // namespace gd

// ---------------------------------------------------------------------------
// Building blocks for tests
// ---------------------------------------------------------------------------
extern "C" gd_status gd_metropolis_dev(gd_ctx *ctx, int n, const float *e_new, const float *e_old,
                                       const float *mbeta, const int *rep, const int *step,
                                       uint64_t seed, uint32_t stream_id, int *accept) {
  if (!ctx || n < 0) return fail(GD_EINVAL, "gd_metropolis_dev: bad arguments");
  if (n == 0) return GD_OK;
  GD_CUDA(cudaSetDevice(ctx->device));
  GD_CUDA(launch_metropolis(n, e_new, e_old, mbeta, rep, step, seed, stream_id, accept,
                            ctx->stream));
  ctx->launches += 1;
  return GD_OK;
}

extern "C" gd_status gd_philox_dev(gd_ctx *ctx, int n, const uint32_t *ctr4, const uint32_t *key2,
                                   uint32_t *out4) {
  if (!ctx || n < 0) return fail(GD_EINVAL, "gd_philox_dev: bad arguments");
  if (n == 0) return GD_OK;
  GD_CUDA(cudaSetDevice(ctx->device));
  GD_CUDA(launch_philox(n, ctr4, key2, out4, ctx->stream));
  ctx->launches += 1;
  return GD_OK;
}

extern "C" gd_status gd_expf_dev(gd_ctx *ctx, int n, const float *x, float *y) {
  if (!ctx || n < 0) return fail(GD_EINVAL, "gd_expf_dev: bad arguments");
  if (n == 0) return GD_OK;
  GD_CUDA(cudaSetDevice(ctx->device));
  GD_CUDA(launch_expf(n, x, y, ctx->stream));
  ctx->launches += 1;
  return GD_OK;
}

extern "C" gd_status gd_fma_peak(gd_ctx *ctx, int n_blocks, int iters, float *ms_out,
                                 double *flops_out) {
  if (!ctx || n_blocks < 1 || iters < 1 || !ms_out || !flops_out)
    return fail(GD_EINVAL, "gd_fma_peak: bad arguments");
  GD_CUDA(cudaSetDevice(ctx->device));
  float *dout = nullptr;
  GD_CUDA(cudaMalloc(&dout, sizeof(float) * n_blocks));
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  launch_fma_peak(dout, n_blocks, iters, ctx->stream);  // warm-up
  cudaEventRecord(a, ctx->stream);
  cudaError_t e = launch_fma_peak(dout, n_blocks, iters, ctx->stream);
  cudaEventRecord(b, ctx->stream);
  cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(dout);
  ctx->launches += 2;
  if (e != cudaSuccess) return fail(GD_ECUDA, "fma probe: %s", cudaGetErrorString(e));
  *ms_out = ms;
  *flops_out = 2.0 * 8.0 * 16.0 * (double)iters * 256.0 * (double)n_blocks;
  return GD_OK;
}
