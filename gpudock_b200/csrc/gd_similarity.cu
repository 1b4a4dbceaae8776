// gd_similarity.cu -- contact-mode similarity of trajectory conformations:
// the similarity matrix of SimilarityMatirxGen (src/util.C:37-87
// CalculateSimilarityMatrix, :90-110 InitConfMatrix, :146-193
// CalculateContactModeScore).
//
// Entry (i, j) is the Matthews correlation of conformation j's contacts
// against conformation i's contact map, where a contact is a ligand-atom /
// protein-point pair with dst <= pmf0[ligand type][point type].  With A and
// B the two maps: tp = |A & B|, fn = |A| - tp, fp = |B| - tp and tn = the
// remaining pairs, so the matrix is a popcount "product" of bit maps.  The
// maps of a trajectory near one pocket are sparse and overlap: a few percent
// of the pairs are a contact of some conformation, and only those get a bit:
//   contacts  one CTA per conformation places its ligand and tests its atoms
//             against the points near the ligand's box; the contacts go into
//             the union of all maps, their number is kept;
//   rank      the number of union bits below each word of the union;
//   maps      the contacts as bits numbered by their rank;
//   pairs     64 x 64 tiles of (i, j), i <= j: popc(A & B) over the maps'
//             words through shared memory, then both entries' MCC.
// Placement and distances follow the reference's float operations in its
// order (no contraction): the rotation comes from the host (PlaceLigand runs
// on the host in the reference, with sinf / cosf), x = r0 x + r1 y + r2 z +
// m + centre and dst = sqrtf(dx dx + dy dy + dz dz), so every contact and
// every entry is the reference's bit for bit.  The test itself is on the
// squared distance: the correctly rounded root never falls as its argument
// grows, so dst <= pmf0 holds exactly up to the largest float whose root is at
// most pmf0 (contact_bound).
#include <cmath>
#include <cstring>
#include <vector>

#include "gd_common.h"

namespace gd {
namespace {

// One conformation: rotation (row major) and translation as PlaceLigand
// uses them, and its protein and ligand conformations.
struct SimConf {
  float r[9];
  float m[3];
  int prt, lig;
  int pad[2];
};

constexpr int kSimThreads = 256;
constexpr int kPairTile = 64;   // conformations per tile side
constexpr int kPairChunk = 32;  // words per shared-memory chunk

constexpr int kCandidates = 2048;  // points looked at per round
constexpr int kRowWords = 8192;    // largest map kept in shared memory
// Contacts of a conformation kept from the first pass for the second (a
// conformation with more is tested again), while the lists of all take at most
// kListBytes: up to 4,096 conformations; a call with more tests every contact
// twice (3,001 conformations: the second pass 10 us with lists, 143 us as the
// first).
constexpr int kListed = 2048;
constexpr size_t kListBytes = 32 << 20;

// The largest float whose correctly rounded square root is at most p (-1:
// none).
__device__ __forceinline__ float contact_bound(float p) {
  if (!(p >= 0.f)) return -1.f;
  if (__float_as_uint(p) >= 0x7f800000u) return p;  // infinity
  // p^2 is within a few units in the last place of it
  uint32_t b = __float_as_uint(__fmul_rn(p, p));
  while (b < 0x7f800000u && __fsqrt_rn(__uint_as_float(b)) <= p) ++b;
  while (b > 0u && !(__fsqrt_rn(__uint_as_float(b)) <= p)) --b;
  return __uint_as_float(b);
}

__global__ void bound_kernel(const float4 *tab, float *bound) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // [GD_NLT][32]
  if (i >= GD_NLT * 32) return;
  const int lt = i / 32, pt = i % 32;
  bound[i] = pt < GD_NPT ? contact_bound(tab[lt * GD_NPT + pt].z) : -1.f;
}

// Contacts of conformation blockIdx.x.  MAPS = false: into the union's bits
// (contact l * pnp + s of atom l and point s), and their number.  MAPS = true:
// as the conformation's map of Kp words, bits numbered by the contact's rank
// in the union, from the list that the first pass kept, or tested again.  Bound
// by latency and L2 reads of the points: the atoms are tested against the few
// points within reach of the ligand's box (600 conformations x 40 x 4,000, caches
// cold: 42 us; testing every pair took 230 us).
template <bool MAPS>
__global__ void __launch_bounds__(kSimThreads)
    contacts_kernel(KTables T, const SimConf *confs, const float *bound, uint32_t *uni, int *pop,
                    const int *base, uint32_t *maps, int Kp, uint32_t *listed) {
  extern __shared__ float4 s_lig[];  // placed atoms, ligand type in .w; the map's words
  uint32_t *s_row = reinterpret_cast<uint32_t *>(s_lig + T.lna);
  __shared__ float s_bound[GD_NLT * 32];
  __shared__ uint16_t s_cand[kCandidates];
  __shared__ int s_n, s_pop;
  __shared__ unsigned s_box[6];  // largest ordered(-x), ordered(x) per axis
  const SimConf c = confs[blockIdx.x];
  const int lna = T.lna, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool row = MAPS && Kp <= kRowWords;
  uint32_t *out = MAPS ? maps + (size_t)blockIdx.x * Kp : nullptr;
  uint32_t *ids = listed ? listed + (size_t)blockIdx.x * kListed : nullptr;
  auto set_bit = [&](uint32_t id) {
    const uint32_t bit = 1u << (id & 31u);
    const int r = base[id >> 5] + __popc(uni[id >> 5] & (bit - 1u));
    if (row)
      atomicOr(&s_row[r >> 5], 1u << (r & 31));
    else
      atomicOr(&out[r >> 5], 1u << (r & 31));
  };
  if (MAPS && ids && pop[blockIdx.x] <= kListed) {
    const int n = pop[blockIdx.x];
    if (row) {
      for (int i = threadIdx.x; i < Kp; i += kSimThreads) s_row[i] = 0u;
      __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += kSimThreads) set_bit(ids[i]);
    if (row) {
      __syncthreads();
      for (int i = threadIdx.x; i < Kp; i += kSimThreads) out[i] = s_row[i];
    }
    return;
  }
  for (int i = threadIdx.x; i < GD_NLT * 32; i += kSimThreads) s_bound[i] = bound[i];
  if (row)
    for (int i = threadIdx.x; i < Kp; i += kSimThreads) s_row[i] = 0u;
  if (threadIdx.x < 6) s_box[threadIdx.x] = 0u;
  if (threadIdx.x == 0) s_n = s_pop = 0;
  __syncthreads();
  for (int l = threadIdx.x; l < lna; l += kSimThreads) {
    const float4 o = T.lig[(size_t)c.lig * lna + l];
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float a = __fmul_rn(c.r[3 * k], o.x);
      a = __fadd_rn(a, __fmul_rn(c.r[3 * k + 1], o.y));
      a = __fadd_rn(a, __fmul_rn(c.r[3 * k + 2], o.z));
      a = __fadd_rn(a, c.m[k]);
      v[k] = __fadd_rn(a, T.lig_center[k]);
      if (v[k] == v[k]) {  // an atom without a position has no contact
        const unsigned u = __float_as_uint(v[k]), w = __float_as_uint(-v[k]);
        atomicMax(&s_box[k], w & 0x80000000u ? ~w : w | 0x80000000u);
        atomicMax(&s_box[3 + k], u & 0x80000000u ? ~u : u | 0x80000000u);
      }
    }
    s_lig[l] = make_float4(v[0], v[1], v[2], __int_as_float(T.lig_t[l]));
  }
  __syncthreads();
  float lo[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned a = s_box[k], b = s_box[3 + k];
    lo[k] = -__uint_as_float(a & 0x80000000u ? a & 0x7fffffffu : ~a);
    hi[k] = __uint_as_float(b & 0x80000000u ? b & 0x7fffffffu : ~b);
  }
  const float4 *P = T.pt_a + (size_t)c.prt * T.pnp_pad;
  for (int s0 = 0; s0 < T.pnp; s0 += kCandidates) {
    const int s1 = min(T.pnp, s0 + kCandidates);
    // points within reach (near_mcc2: the largest pmf0 squared, with margin)
    for (int i = s0 + warp * 32; i < s1; i += kSimThreads) {
      const int s = i + lane;
      bool near = false;
      if (s < s1) {
        const float4 p = P[s];
        const float bx = fmaxf(fmaxf(lo[0] - p.x, p.x - hi[0]), 0.f);
        const float by = fmaxf(fmaxf(lo[1] - p.y, p.y - hi[1]), 0.f);
        const float bz = fmaxf(fmaxf(lo[2] - p.z, p.z - hi[2]), 0.f);
        near = fmaf(bz, bz, fmaf(by, by, bx * bx)) <= T.near_mcc2;
      }
      const uint32_t m = __ballot_sync(0xffffffffu, near);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(&s_n, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (near) s_cand[at + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(s - s0);
    }
    __syncthreads();
    // a warp takes a point against 32 atoms at a time
    const int n = s_n;
    for (int q = warp; q < n; q += kSimThreads / 32) {
      const int s = s0 + s_cand[q];
      const float4 p = P[s];
      const int pt = (int)(__float_as_uint(T.pt_b[s].y) & META_TYPE_MASK);
      for (int l0 = 0; l0 < lna; l0 += 32) {
        const int l = l0 + lane;
        bool hit = false;
        if (l < lna) {
          const float4 a = s_lig[l];
          const float dx = __fsub_rn(a.x, p.x);
          const float dy = __fsub_rn(a.y, p.y);
          const float dz = __fsub_rn(a.z, p.z);
          const float d2 =
              __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
          hit = d2 <= s_bound[__float_as_int(a.w) * 32 + pt];
        }
        const uint32_t id = (uint32_t)l * (uint32_t)T.pnp + (uint32_t)s;
        if (MAPS) {
          if (hit) set_bit(id);
          continue;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (m == 0u) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_pop, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (hit) {
          const uint32_t bit = 1u << (id & 31u);
          // most contacts are in the union already
          if (!(__ldcg(&uni[id >> 5]) & bit)) atomicOr(&uni[id >> 5], bit);
          if (ids && at < kListed) ids[at] = id;
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
  }
  if (!MAPS) {
    if (threadIdx.x == 0) pop[blockIdx.x] = s_pop;
  } else if (row) {
    for (int i = threadIdx.x; i < Kp; i += kSimThreads) out[i] = s_row[i];
  }
}

// base[w] = number of union bits below word w, base[K] = all (one block).
__global__ void __launch_bounds__(1024) rank_kernel(const uint32_t *uni, int K, int *base) {
  __shared__ int s_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int before = 0;
  for (int k0 = 0; k0 < K; k0 += 1024) {
    const int k = k0 + threadIdx.x;
    const int b = k < K ? __popc(uni[k]) : 0;
    int v = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += x;
    }
    if (lane == 31) s_sum[warp] = v;
    __syncthreads();
    if (warp == 0) {
      int t = s_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += x;
      }
      s_sum[lane] = t;
    }
    __syncthreads();
    if (k < K) base[k] = before + (warp ? s_sum[warp - 1] : 0) + v - b;
    before += s_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) base[K] = before;
}

// CalculateContactModeScore's arithmetic: the four sums as floats multiplied
// left to right, sqrtf, and the integer numerator tp tn - fp fn (wrapping
// like the reference's int) over it; 10000 where the denominator is 0.
__device__ __forceinline__ float contact_mcc(int tp, int fn, int fp, int tn) {
  float q = __fmul_rn(__int2float_rn(tp + fp), __int2float_rn(tp + fn));
  q = __fmul_rn(q, __int2float_rn(tn + fp));
  q = __fmul_rn(q, __int2float_rn(tn + fn));
  const float dividend = __fsqrt_rn(q);
  const int num = (int)((unsigned)tp * (unsigned)tn - (unsigned)fp * (unsigned)fn);
  return dividend != 0.0f ? __fdiv_rn(__int2float_rn(num), dividend) : GD_CMCC_INVALID;
}

// Tile pair t of the upper triangle of tiles x tiles: its row and column.
__device__ __forceinline__ void tile_of(int t, int tiles, int *row, int *col) {
  // row r starts at r tiles - r (r - 1) / 2
  int r = (int)((2.0f * tiles + 1.0f -
                 sqrtf(fmaxf(0.f, (2.0f * tiles + 1.0f) * (2.0f * tiles + 1.0f) - 8.0f * t))) *
                0.5f);
  auto start = [&](int x) { return (long long)x * tiles - (long long)x * (x - 1) / 2; };
  while (r > 0 && start(r) > t) --r;
  while (start(r + 1) <= t) ++r;
  *row = r;
  *col = r + (int)(t - start(r));
}

// Entries of the matrix.  With a bit per contact of the union, in place of the
// 32-bit words that hold one, the maps are several times shorter, and only the
// upper triangle's tiles are counted: 600 conformations 261 -> 24 us, 3,001 3,890
// -> 156 us.  Bound by the ALU pipe (carry-save counting).
__global__ void __launch_bounds__(kSimThreads)
    pairs_kernel(const uint32_t *comp, const int *pop, int n, int Kp, int total, int tiles,
                 float *S) {
  __shared__ uint32_t s_mem[2 * kPairTile * (kPairChunk + 1)];
  uint32_t(*sa)[kPairChunk + 1] = reinterpret_cast<uint32_t(*)[kPairChunk + 1]>(s_mem);
  uint32_t(*sb)[kPairChunk + 1] = sa + kPairTile;
  int ti, tj;
  tile_of(blockIdx.x, tiles, &ti, &tj);
  const int i0 = ti * kPairTile, j0 = tj * kPairTile;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  // Carry-save counting (Harley and Seal; Mula, Kurz and Lemire, "Faster
  // population counts using AVX2 instructions", 2018): the AND words of an
  // entry are added bitwise into `ones` and `twos`; every 4 words the carry
  // out, `fours`, goes through one POPC (which issues on the XU pipe, 16 per
  // clock per SM) and the rest stays in bitwise operations.  The count is
  // 4 sum popc(fours) + 2 popc(twos) + popc(ones).
  uint32_t ones[4][4] = {}, twos[4][4] = {};
  int acc[4][4] = {};
  for (int k0 = 0; k0 < Kp; k0 += kPairChunk) {
    for (int q = tid; q < kPairTile * kPairChunk; q += kSimThreads) {
      const int row = q / kPairChunk, col = q % kPairChunk;
      const int i = i0 + row, j = j0 + row;
      sa[row][col] = i < n ? comp[(size_t)i * Kp + k0 + col] : 0u;
      sb[row][col] = j < n ? comp[(size_t)j * Kp + k0 + col] : 0u;
    }
    __syncthreads();
    for (int kk = 0; kk < kPairChunk; kk += 4) {
      uint32_t a[4][4], b[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) a[r][q] = sa[ty + 16 * r][kk + q];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q) b[c][q] = sb[tx + 16 * c][kk + q];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t x0 = a[r][0] & b[c][0], x1 = a[r][1] & b[c][1];
          const uint32_t x2 = a[r][2] & b[c][2], x3 = a[r][3] & b[c][3];
          uint32_t &o = ones[r][c], &t = twos[r][c];
          // (twos_a, ones) = ones + x0 + x1; (twos_b, ones) = ones + x2 + x3
          uint32_t u = o ^ x0;
          const uint32_t ta = (o & x0) | (u & x1);
          o = u ^ x1;
          u = o ^ x2;
          const uint32_t tb = (o & x2) | (u & x3);
          o = u ^ x3;
          // (fours, twos) = twos + twos_a + twos_b
          u = t ^ ta;
          const uint32_t fours = (t & ta) | (u & tb);
          t = u ^ tb;
          acc[r][c] += __popc(fours);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      acc[r][c] = 4 * acc[r][c] + 2 * __popc(twos[r][c]) + __popc(ones[r][c]);
  // the tile's counts through shared memory (its words have been read), so
  // that both (i, j) and (j, i) are written along rows
  int *s_tp = reinterpret_cast<int *>(s_mem);  // [kPairTile][kPairTile + 1]
  static_assert(kPairTile * (kPairTile + 1) <= 2 * kPairTile * (kPairChunk + 1), "count tile");
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      s_tp[(ty + 16 * r) * (kPairTile + 1) + tx + 16 * c] = acc[r][c];
  __syncthreads();
  for (int q = tid; q < kPairTile * kPairTile; q += kSimThreads) {
    const int r = q / kPairTile, c = q % kPairTile;
    if (i0 + r < n && j0 + c < n) {
      const int tp = s_tp[r * (kPairTile + 1) + c];
      const int fn = pop[i0 + r] - tp, fp = pop[j0 + c] - tp;
      S[(size_t)(i0 + r) * n + j0 + c] = contact_mcc(tp, fn, fp, total - tp - fn - fp);
    }
    if (ti != tj && j0 + r < n && i0 + c < n) {
      const int tp = s_tp[c * (kPairTile + 1) + r];
      const int fn = pop[j0 + r] - tp, fp = pop[i0 + c] - tp;
      S[(size_t)(j0 + r) * n + i0 + c] = contact_mcc(tp, fn, fp, total - tp - fn - fp);
    }
  }
}

template <typename T>
cudaError_t get(Workspace &W, T **p, size_t count) {
  return W.get((void **)p, count * sizeof(T));
}

}  // namespace
}  // namespace gd

using namespace gd;

// The matrix into S_dev (the caller's device memory) or, with S_dev null,
// into S_host through a buffer of its own.
static gd_status similarity_run(gd_ctx *ctx, const gd_dcomplex *d, int n_conf,
                                const float *confs, float *S_dev, float *S_host) {
  if (!ctx || !d) return fail(GD_EINVAL, "gd_similarity_matrix: NULL handle");
  if (n_conf < 0) return fail(GD_EINVAL, "n_conf=%d", n_conf);
  if (n_conf == 0) return GD_OK;
  if (!confs || (!S_dev && !S_host)) return fail(GD_EINVAL, "confs/similarity NULL");
  const KTables &T = d->T;
  if ((size_t)n_conf * (size_t)n_conf > ((size_t)1 << 40))
    return fail(GD_EINVAL, "n_conf=%d: the matrix is too large", n_conf);
  // PlaceLigand's rotation (util.C:496-535) on the host, as the reference
  std::vector<SimConf> hc((size_t)n_conf);
  for (int i = 0; i < n_conf; ++i) {
    const float *t = confs + (size_t)i * 8;
    for (int k = 0; k < 8; ++k)
      if (!std::isfinite(t[k])) return fail(GD_EINVAL, "conformation %d: non-finite value", i);
    const int prt = (int)t[0], lig = (int)t[1];
    if (prt < 0 || prt >= T.n_prt || lig < 0 || lig >= T.n_lig)
      return fail(GD_EINVAL, "conformation %d: protein %d / ligand %d out of range", i, prt,
                  lig);
    const float *m = t + 2;
    const float s1 = sinf(m[3]), c1 = cosf(m[3]);
    const float s2 = sinf(m[4]), c2 = cosf(m[4]);
    const float s3 = sinf(m[5]), c3 = cosf(m[5]);
    SimConf &c = hc[i];
    std::memset(&c, 0, sizeof(c));
    c.r[0] = c1 * c2;
    c.r[1] = c1 * s2 * s3 - c3 * s1;
    c.r[2] = s1 * s3 + c1 * c3 * s2;
    c.r[3] = c2 * s1;
    c.r[4] = c1 * c3 + s1 * s2 * s3;
    c.r[5] = c3 * s1 * s2 - c1 * s3;
    c.r[6] = -1 * s2;
    c.r[7] = c2 * s3;
    c.r[8] = c2 * c3;
    for (int k = 0; k < 3; ++k) c.m[k] = m[k];
    c.prt = prt;
    c.lig = lig;
  }
  GD_CUDA(cudaSetDevice(ctx->device));
  cudaStream_t s = ctx->stream;
  const size_t K = ((size_t)T.lna * T.pnp + 31) / 32;  // words of the union
  const int total = T.lna * T.pnp;
  const size_t n = (size_t)n_conf;
  gd_status st = GD_OK;
  {
    const size_t listed = n * kListed * sizeof(uint32_t) <= kListBytes ? n * kListed : 0;
    // (the maps' words follow from the contacts: 1 in 16 pairs of the union at most
    // is what a trajectory near one pocket has)
    Workspace W(ctx, 4096 + sizeof(SimConf) * n + 8 * K + 4 * (n + listed + n * (K / 16)) +
                         (S_dev ? 0 : sizeof(float) * n * n));
    SimConf *d_conf = nullptr;
    uint32_t *d_uni = nullptr, *d_maps = nullptr;
    float *d_bound = nullptr, *d_S = nullptr;
    int *d_pop = nullptr, *d_base = nullptr;
    uint32_t *d_listed = nullptr;
    cudaError_t e = get(W, &d_conf, n);
    if (e == cudaSuccess) e = get(W, &d_uni, K);
    if (e == cudaSuccess) e = get(W, &d_bound, (size_t)GD_NLT * 32);
    if (e == cudaSuccess) e = get(W, &d_pop, n);
    if (e == cudaSuccess) e = get(W, &d_base, K + 1);
    if (e == cudaSuccess && listed && get(W, &d_listed, listed) != cudaSuccess) {
      cudaGetLastError();  // without room for the lists the contacts are tested twice
      d_listed = nullptr;
    }
    if (e == cudaSuccess && !S_dev) e = get(W, &d_S, n * n);
    if (S_dev) d_S = S_dev;
    if (e != cudaSuccess) return fail(GD_ENOMEM, "similarity buffers: %s", cudaGetErrorString(e));
    GD_CUDA(cudaMemcpyAsync(d_conf, hc.data(), sizeof(SimConf) * n, cudaMemcpyHostToDevice, s));
    GD_CUDA(cudaMemsetAsync(d_uni, 0, sizeof(uint32_t) * K, s));
    bound_kernel<<<(GD_NLT * 32 + 255) / 256, 256, 0, s>>>(T.tab_a, d_bound);
    GD_CUDA(cudaGetLastError());
    contacts_kernel<false><<<n_conf, kSimThreads, sizeof(float4) * T.lna, s>>>(
        T, d_conf, d_bound, d_uni, d_pop, nullptr, nullptr, 0, d_listed);
    GD_CUDA(cudaGetLastError());
    rank_kernel<<<1, 1024, 0, s>>>(d_uni, (int)K, d_base);
    GD_CUDA(cudaGetLastError());
    int n_bits = 0;
    GD_CUDA(cudaMemcpyAsync(&n_bits, d_base + K, sizeof(int), cudaMemcpyDeviceToHost, s));
    GD_CUDA(cudaStreamSynchronize(s));
    const int Kp = (n_bits + 32 * kPairChunk - 1) / (32 * kPairChunk) * kPairChunk;
    if (Kp) {
      e = get(W, &d_maps, n * (size_t)Kp);
      if (e != cudaSuccess)
        return fail(GD_ENOMEM, "similarity buffers: %s", cudaGetErrorString(e));
      const bool row = Kp <= kRowWords;
      if (!row) GD_CUDA(cudaMemsetAsync(d_maps, 0, sizeof(uint32_t) * n * Kp, s));
      contacts_kernel<true><<<n_conf, kSimThreads,
                              sizeof(float4) * T.lna + (row ? sizeof(uint32_t) * Kp : 0), s>>>(
          T, d_conf, d_bound, d_uni, d_pop, d_base, d_maps, Kp, d_listed);
      GD_CUDA(cudaGetLastError());
    }
    const int tiles = (n_conf + kPairTile - 1) / kPairTile;
    pairs_kernel<<<(unsigned)((long long)tiles * (tiles + 1) / 2), kSimThreads, 0, s>>>(
        d_maps, d_pop, n_conf, Kp, total, tiles, d_S);
    GD_CUDA(cudaGetLastError());
    ctx->launches += Kp ? 5 : 4;
    if (!S_dev)
      GD_CUDA(cudaMemcpyAsync(S_host, d_S, sizeof(float) * n * n, cudaMemcpyDeviceToHost, s));
    st = ctx_check(ctx);
  }
  if (st == GD_OK) GD_CUDA(cudaStreamSynchronize(s));
  return st;
}

extern "C" gd_status gd_similarity_matrix(gd_ctx *ctx, const gd_dcomplex *d, int n_conf,
                                          const float *confs, float *similarity) {
  NvtxRange nvtx("gd_similarity_matrix");
  if (n_conf > 0 && !similarity) return fail(GD_EINVAL, "similarity NULL");
  return similarity_run(ctx, d, n_conf, confs, nullptr, similarity);
}

extern "C" gd_status gd_similarity_matrix_dev(gd_ctx *ctx, const gd_dcomplex *d, int n_conf,
                                              const float *confs, float *similarity_dev) {
  if (n_conf > 0 && !similarity_dev) return fail(GD_EINVAL, "similarity_dev NULL");
  return similarity_run(ctx, d, n_conf, confs, similarity_dev, nullptr);
}
