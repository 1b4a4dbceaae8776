// gd_poses.cu -- the poses of a large energy call dealt into cells of their
// translation, so that a CTA's 32 poses lie close together and most protein
// points are far of all of them (the far form of the pair terms,
// gd_kernels.cu).
//
// Which points take the far form follows from the cell alone, never from the
// other poses of the CTA, and the cells from the box of the call's
// translations: a pose's energy does not depend on the order of the poses.
// Poses without a usable place (a value that is not finite, or a translation
// beyond kFarOut) get a cell of their own, for which no point is far.
//
// Four short launches (33 us together for 65,536 poses, caches cold): the box of
// the translations; every pose's cell and its rank in it; the cells' first
// 32-pose blocks; the poses in block order.  Up to kSmallPoses poses, one launch
// of one CTA does all of it (11 us for 4,096 poses, 27 us for 16,384).
#include <algorithm>
#include <climits>
#include <cmath>

#include "gd_common.h"

namespace gd {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxCells = 4096;
constexpr float kFarOut = 4.0e3f;
// Poses per cell: a cell's last block is half empty on average, so about 5% of
// the blocks' lanes are idle.
constexpr int kPosesPerCell = 320;
constexpr int kSmallPoses = 16384;
// The most poses that are dealt: below it every index here is an int (a pose's
// place in block order, and a grid-stride loop's step past the last pose).
constexpr int kMostPoses = 1 << 30;
static_assert((long long)kMostPoses + 32LL * (kMaxCells + 1) + 148LL * 4 * kThreads < INT_MAX,
              "pose indexes");
constexpr float kMinEdge = 0.75f;  // smaller cells gain little (the ligand is larger)

int max_cells(int n_pose) { return std::max(1, std::min(kMaxCells, n_pose / kPosesPerCell)); }
int max_blocks(int n_pose) { return (n_pose + 31) / 32 + max_cells(n_pose) + 1; }

// Workspace of a call (see pose_work_bytes).
struct Work {
  unsigned *box;    // [6] largest ordered(-t), ordered(t) per axis, 0: none
  PoseGrid *grid;
  int *count;       // [max_cells + 1] poses of each cell
  int *first;       // [max_cells + 1] its first block
  int2 *at;         // [n] {cell, rank}
  int *order;       // [max_blocks * 32]
  int *block_cell;  // [max_blocks]
  size_t zero, total;
};

Work layout(unsigned char *p, int n) {
  Work w{};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    unsigned char *q = p + o;
    o += (bytes + 255) & ~size_t(255);
    return q;
  };
  w.box = (unsigned *)take(6 * sizeof(unsigned));
  w.count = (int *)take((max_cells(n) + 1) * sizeof(int));
  w.zero = o;  // up to here the call starts from zeros
  w.grid = (PoseGrid *)take(sizeof(PoseGrid));
  w.first = (int *)take((max_cells(n) + 1) * sizeof(int));
  w.at = (int2 *)take((size_t)n * sizeof(int2));
  w.order = (int *)take((size_t)max_blocks(n) * 32 * sizeof(int));
  w.block_cell = (int *)take((size_t)max_blocks(n) * sizeof(int));
  w.total = o;
  return w;
}

// Unsigned integers in the order of the floats; 0 is below every one.
__device__ __forceinline__ unsigned ordered(float x) {
  const unsigned u = __float_as_uint(x);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float unordered(unsigned u) {
  return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

__device__ __forceinline__ bool usable(const float t[3]) {
  return fabsf(t[0]) < kFarOut && fabsf(t[1]) < kFarOut && fabsf(t[2]) < kFarOut;
}

// The translation of a pose; not usable when an angle is not finite: its atoms
// have no positions then.
__device__ __forceinline__ void load_translation(const float *poses, int i, float t[3]) {
  const float *m = poses + (size_t)i * 6;
  t[0] = m[0], t[1] = m[1], t[2] = m[2];
  if (!(isfinite(m[3]) && isfinite(m[4]) && isfinite(m[5]))) t[0] = INFINITY;
}

__global__ void __launch_bounds__(kThreads) box_kernel(const float *poses, int n, unsigned *box) {
  unsigned m[6] = {0, 0, 0, 0, 0, 0};
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    float t[3];
    load_translation(poses, i, t);
    if (!usable(t)) continue;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      m[k] = max(m[k], ordered(-t[k]));
      m[3 + k] = max(m[3 + k], ordered(t[k]));
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    m[k] = __reduce_max_sync(0xffffffffu, m[k]);
    if ((threadIdx.x & 31) == 0 && m[k] != 0u) atomicMax(&box[k], m[k]);
  }
}

// The grid over the box: the smallest edge (from kMinEdge on, in steps of
// 10%) that needs at most max_cells cells.
__device__ PoseGrid make_grid(const unsigned *box, int max_cells) {
  PoseGrid g;
  float range[3] = {0.f, 0.f, 0.f};
  float most = 0.f;
  for (int k = 0; k < 3; ++k) {
    g.lo[k] = box[k] ? -unordered(box[k]) : 0.f;
    range[k] = box[3 + k] ? unordered(box[3 + k]) - g.lo[k] : 0.f;
    most = fmaxf(most, range[k]);
  }
  g.edge = kMinEdge;
  for (;;) {
    double cells = 1.0;
    for (int k = 0; k < 3; ++k) {
      g.n[k] = max(1, (int)ceilf(range[k] / g.edge));
      cells *= g.n[k];
    }
    if (cells <= (double)max_cells) break;
    g.edge *= 1.1f;
  }
  g.inv_edge = 1.0f / g.edge;
  g.n_cells = g.n[0] * g.n[1] * g.n[2];
  // how far past its cell's walls rounding can leave a pose
  g.margin = 1e-3f + 1e-5f * most;
  g.n_blocks = 0;
  return g;
}

__device__ __forceinline__ int cell_of(const PoseGrid &g, const float t[3]) {
  if (!usable(t)) return g.n_cells;
  int c[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    c[k] = min(g.n[k] - 1, max(0, (int)((t[k] - g.lo[k]) * g.inv_edge)));
  return (c[2] * g.n[1] + c[1]) * g.n[0] + c[0];
}

__global__ void __launch_bounds__(kThreads)
    cell_kernel(const float *poses, int n, int max_cells, const unsigned *box, PoseGrid *grid,
                int *count, int2 *at) {
  __shared__ PoseGrid g;
  if (threadIdx.x == 0) {
    g = make_grid(box, max_cells);
    if (blockIdx.x == 0) *grid = g;
  }
  __syncthreads();
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  float t[3];
  load_translation(poses, i, t);
  const int cell = cell_of(g, t);
  at[i] = make_int2(cell, atomicAdd(&count[cell], 1));
}

// Exclusive scan of the cells' block counts (one block).
__global__ void __launch_bounds__(1024) scan_kernel(PoseGrid *grid, const int *count, int *first) {
  __shared__ int warp_sum[32];
  const int n = grid->n_cells + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int c0 = 0; c0 < n; c0 += 1024) {
    const int c = c0 + threadIdx.x;
    const int b = c < n ? (count[c] + 31) / 32 : 0;
    int s = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += x;
    }
    if (lane == 31) warp_sum[warp] = s;
    __syncthreads();
    if (warp == 0) {
      int v = warp_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
      }
      warp_sum[lane] = v;
    }
    __syncthreads();
    if (c < n) first[c] = base + (warp ? warp_sum[warp - 1] : 0) + s - b;
    base += warp_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) grid->n_blocks = base;
}

__global__ void __launch_bounds__(kThreads)
    order_kernel(int n, const int2 *at, const int *first, int *order, int *block_cell) {
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int2 a = at[i];
  const int b = first[a.x] + a.y / 32;
  order[b * 32 + a.y % 32] = i;
  if (a.y % 32 == 0) block_cell[b] = a.x;
}

// All of the above for up to kSmallPoses poses: 16 poses a thread, the cells'
// counts in shared memory.
__global__ void __launch_bounds__(1024)
    small_kernel(const float *poses, int n, int max_cells, PoseGrid *grid, int *count, int *first,
                 int *order, int *block_cell) {
  constexpr int kCells = kSmallPoses / kPosesPerCell + 1;
  constexpr int kEach = kSmallPoses / 1024;
  __shared__ unsigned s_box[6];
  __shared__ PoseGrid g;
  __shared__ int s_count[kCells], s_first[kCells];
  if (threadIdx.x < 6) s_box[threadIdx.x] = 0u;
  for (int c = threadIdx.x; c < kCells; c += 1024) s_count[c] = 0;
  __syncthreads();
  float t[kEach][3];
  unsigned m[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int i = j * 1024 + threadIdx.x;
    if (i < n) load_translation(poses, i, t[j]);
    if (i < n && usable(t[j])) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        m[k] = max(m[k], ordered(-t[j][k]));
        m[3 + k] = max(m[3 + k], ordered(t[j][k]));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    m[k] = __reduce_max_sync(0xffffffffu, m[k]);
    if ((threadIdx.x & 31) == 0 && m[k] != 0u) atomicMax(&s_box[k], m[k]);
  }
  __syncthreads();
  if (threadIdx.x == 0) g = make_grid(s_box, max_cells);
  __syncthreads();
  int cell[kEach], rank[kEach];
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    cell[j] = rank[j] = 0;
    if (j * 1024 + (int)threadIdx.x >= n) continue;
    cell[j] = cell_of(g, t[j]);
    rank[j] = atomicAdd(&s_count[cell[j]], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int b = 0;
    for (int c = 0; c <= g.n_cells; ++c) {
      s_first[c] = b;
      b += (s_count[c] + 31) / 32;
    }
    g.n_blocks = b;
    *grid = g;
  }
  __syncthreads();
  for (int c = threadIdx.x; c <= g.n_cells; c += 1024) {
    count[c] = s_count[c];
    first[c] = s_first[c];
  }
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int i = j * 1024 + threadIdx.x;
    if (i >= n) continue;
    const int b = s_first[cell[j]] + rank[j] / 32;
    order[b * 32 + rank[j] % 32] = i;
    if (rank[j] % 32 == 0) block_cell[b] = cell[j];
  }
}

}  // namespace

bool pose_cells_pay(const KTables &T, double far_share, int n_sm, int n_pose) {
  if (n_pose > kMostPoses) return false;
  // While the poses leave half of the SMs idle they are spread over them in
  // other ways (pose_units): 2,048 poses x 48 x 1,100 in 338 us with cells, 181
  // on clusters of two.
  const int units = (n_pose + 31) / 32;
  if (2 * units <= n_sm) return false;
  // Else the waves of blocks (from four on the SMs take them as they come), times
  // a block's time (6 pairs per ns and SM), with the cells' half-filled last blocks
  // and the deal on one side.  A block's time was fitted to calls whose poses lie
  // 1 to 4 A about the start place, where most have more far points than the share
  // there says; in few waves, which last as long as their slowest blocks, less is
  // gained.  Measured, cells against without (box in A, share): 4,700 x 96 x 700 (a
  // second wave) 856 and 442 us; 2,900 x 48 x 1,000 (4, 0.06) 327 and 310; 4,096 x
  // 24 x 1,500 (4, 0.34) 165 and 178 among other calls, whose blocks start as the
  // shorter ones end, 215 and 212 one after another; 60,000 x 48 x 900 (6, 0.02)
  // 3.83 and 3.68 ms; 40,000 x 40 x 700 (2, 0.08) 1.56 and 1.51; 50,000 x 60 x 1,300
  // (6, 0.07) 5.67 and 6.01; 100,000 x 20 x 800 (8, 0.12) 2.86 and 3.16; 131,072 x 48
  // x 2,000 (8, 0.21) 13.8 and 14.9, (8, 0.36) 12.6 and 14.2; 30,011 x 48 x 8,000 (8,
  // 0.79) 9.0 and 12.2.
  const double cells = max_cells(n_pose), f = far_share;
  const double units_with = units + 0.5 * cells;
  const double block_us = 32.0 * T.lna * T.pnp / 6000.0;
  const double deal_us = n_pose <= kSmallPoses ? 6.0 + n_pose / 800.0 : 20.0 + n_pose / 4000.0;
  double w0 = (double)units / n_sm, w1 = units_with / n_sm;
  double block = 1.02 - 0.95 * f + 0.65 * f * f;
  if (w0 < 4.0) {
    w0 = std::ceil(w0);
    w1 = std::ceil((units_with + std::sqrt(cells)) / n_sm);
    block = 1.05 - 0.45 * f;
  }
  return w1 * block_us * block + deal_us < w0 * block_us;
}

size_t pose_work_bytes(const KTables &T, double far_share, int n_sm, int n_pose) {
  return pose_cells_pay(T, far_share, n_sm, n_pose) ? layout(nullptr, n_pose).total : 0;
}

cudaError_t pose_cells(KRun *R, void *work, int *grid, int *launches, cudaStream_t s) {
  const int n = R->n_pose, cells = max_cells(n);
  const Work w = layout(static_cast<unsigned char *>(work), n);
  R->pose_grid = w.grid;
  R->pose_order = w.order;
  R->pose_cell = w.block_cell;
  R->cell_first = w.first;
  R->cell_count = w.count;
  *grid = max_blocks(n);
  if (n <= kSmallPoses) {
    *launches = 1;
    small_kernel<<<1, 1024, 0, s>>>(R->poses, n, cells, w.grid, w.count, w.first, w.order,
                                    w.block_cell);
    return cudaGetLastError();
  }
  *launches = 4;
  cudaError_t e = cudaMemsetAsync(work, 0, w.zero, s);
  if (e != cudaSuccess) return e;
  const int blocks = (n + kThreads - 1) / kThreads;
  box_kernel<<<std::min(blocks, 148 * 4), kThreads, 0, s>>>(R->poses, n, w.box);
  cell_kernel<<<blocks, kThreads, 0, s>>>(R->poses, n, cells, w.box, w.grid, w.count, w.at);
  scan_kernel<<<1, 1024, 0, s>>>(w.grid, w.count, w.first);
  order_kernel<<<blocks, kThreads, 0, s>>>(n, w.at, w.first, w.order, w.block_cell);
  return cudaGetLastError();
}

}  // namespace gd
