// Batched ensembles: many independent systems ("clusters") of uneven size
// advanced together, one persistent pair launch per Hermite step.
//
// Layout: cluster c owns padded rows [row0_c, row0_c + ld_c) of every
// ensemble array (ld_c = n_c rounded up to 256), so j-tiles never straddle
// clusters and padding rows are zero-mass bodies that add nothing.  A row's
// cluster comes from cid[row] (-1 on padding rows).
//
// Work list: item = (cluster, 256-row block, range of at most `tiles_per_item`
// j-tiles; in the symmetric schedule, sympair.cuh, of the block's run).  Items
// are sorted by cost (longest first) and a fixed grid of SMs x resident CTAs
// takes them from an atomic counter, so a 256-body cluster and an 8192-body
// cluster share one launch without the small one idling the GPU.  The partial-sum slots of cluster c live at P + p_off_c ([slot][6][ld_c])
// and are added in a fixed order by the corrector, so results are bitwise
// reproducible.
//
// A step is memset(counter) -> predict -> persistent pair -> correct, captured
// into a CUDA graph; only the last step of a call carries the event records of
// last_step_ms (about 3.6 us each).  FP64 ensembles and pair_variant 4 run the
// symmetric kernels, mixed ones by default (and pair_variant 3) the one-sided
// packed hi/lo kernel, pair_variant 5 the one-sided near/far kernel with every
// tile taken as far.  pair_variant 4 and 5 use tile-relative records: each
// cluster then keeps its bodies in Hilbert order within its own padded segment (every
// sort_every steps a second captured graph sorts (cluster, Hilbert code) keys
// over all rows and gathers the state into that order; perm maps positions
// back to the caller's rows).
// Each cluster has its own softening and fixed shared step (the adaptive
// criterion is per system in the reference, src/nbody.cpp:198-222; ensembles
// here run fixed steps).
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <numeric>
#include <vector>

#include "../../include/nbody_cuda.h"
#include "errors.h"
#include "hermite.cuh"
#include "pair.cuh"
#include "reltiles.cuh"
#include "sympair.cuh"
#include "trace.h"

using namespace nbody;

namespace {

constexpr int kPadRows = kEnsRows;  // cluster padding = rows per work item
constexpr int kBlock = 256;
// Bodies of an item's tile range by default: the most of these that leaves
// several items per resident CTA, so that the last ones are short.  Steps by
// bodies per item, packed hi/lo: 256 clusters of 256-8192 bodies 2.87 ms (1024),
// 2.89 (512); 256 of 256-1024 302 us (1024), 193 (512); 16 of 256-2048 284 us
// (1024), 152 (512), 56 (128).
constexpr int kItemBodies[] = {1024, 512, 256, 128, 64};
// A j-tile of the interface (tiles_per_item, info's j_tile) in tiles of the
// kernel: FP64 items are given in tiles of 128 bodies, whatever the kernel streams.
constexpr int kFp64ItemTile = 128;
constexpr double kItemsPerCta = 2.5;
constexpr int kWideCtasPerSm = 6;  // resident CTAs of the four-row near/far shape

struct ClusterDev {
  int row0, n, ld;
  int S, block_rows, nb;  // slots of a row: RowSlots(S, block_rows, nb)
  long long p_off;
  double eps2, dt;
};

#define EN_CUDA(call)                                                                      \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess) {                                                               \
      cudaGetLastError(); /* returned here, not by the next call's check of its launches */ \
      return nbody_set_error(e_ == cudaErrorMemoryAllocation ? NBODY_ERR_OOM : NBODY_ERR_CUDA, \
                             "%s failed: %s", #call, cudaGetErrorString(e_));              \
    }                                                                                      \
  } while (0)
#define EN_TRY(expr)               \
  do {                             \
    nbody_status s_ = (expr);      \
    if (s_ != NBODY_OK) return s_; \
  } while (0)

// ---- kernels ----------------------------------------------------------------

__global__ void ens_pack_kernel(int L, const int* __restrict__ cid, const double* __restrict__ X,
                                const double* __restrict__ V, const double* __restrict__ M,
                                JBody64* __restrict__ jb64, JBodyX2* __restrict__ jbx = nullptr) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L) return;
  const bool real = cid[r] >= 0;
  const double x = real ? X[r] : 0, y = real ? X[L + r] : 0, z = real ? X[2 * L + r] : 0;
  const double m = real ? M[r] : 0;
  const double u = real ? V[r] : 0, v = real ? V[L + r] : 0, w = real ? V[2 * L + r] : 0;
  if (jb64) store_jb64(jb64, r, x, y, z, m, u, v, w);
  if (jbx) jbx[r] = make_jbx2(x, y, z, m, u, v, w);
}

// Near/far subtile blockIdx.x of the state; PREDICT: of the predicted state,
// which is written back to X, V.
template <bool PREDICT>
__global__ void __launch_bounds__(64)
    ens_tile_kernel(int L, const int* __restrict__ cid, const ClusterDev* __restrict__ cl,
                    double* __restrict__ X, double* __restrict__ V, const double* __restrict__ M,
                    const double* __restrict__ D, SymSub* __restrict__ out) {
  const int r = blockIdx.x * 64 + threadIdx.x;
  const int c = cid[r];  // L is a multiple of 256
  double p[3] = {0.0, 0.0, 0.0}, u[3] = {0.0, 0.0, 0.0}, m = 0.0;
  if (c >= 0) {
    m = M[r];
    if (PREDICT) {
      predict_body(cl[c].dt, L, r, X, V, D, p, u);
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[k] = X[k * L + r];
        u[k] = V[k * L + r];
      }
    }
  }
  write_subtile<true>(out + blockIdx.x, c >= 0, p, u, m);
}

// Predictor of the FP64 ensemble and of the one-sided kernels, with the records
// that are not null.
__global__ void ens_predict_kernel(int L, const int* __restrict__ cid,
                                   const ClusterDev* __restrict__ cl, double* __restrict__ X,
                                   double* __restrict__ V, const double* __restrict__ M,
                                   const double* __restrict__ D, JBody64* __restrict__ jb64,
                                   JBodyX2* __restrict__ jbx) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L) return;
  const int c = cid[r];
  if (c < 0) return;
  double p[3], u[3];
  predict_body(cl[c].dt, L, r, X, V, D, p, u);
  if (jb64) store_jb64(jb64, r, p[0], p[1], p[2], M[r], u[0], u[1], u[2]);
  if (jbx) jbx[r] = make_jbx2(p[0], p[1], p[2], M[r], u[0], u[1], u[2]);
}

// Between the caller's concatenated arrays ([count][total]) and the padded
// ones ([count][L]): idx[row] is a padded row's index in the caller's order, -1
// on padding.  One launch instead of a copy per cluster and array.
__global__ void ens_expand_kernel(int L, int total, int count, const int* __restrict__ idx,
                                  const double* __restrict__ src, double* __restrict__ dst) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L) return;
  const int o = idx[r];
  for (int k = 0; k < count; ++k)
    dst[static_cast<size_t>(k) * L + r] = o >= 0 ? src[static_cast<size_t>(k) * total + o] : 0.0;
}
// perm (nullable): row r holds the body of padded row perm[r].
__global__ void ens_compact_kernel(int L, int total, int count, const int* __restrict__ idx,
                                   const int* __restrict__ perm, const double* __restrict__ src,
                                   double* __restrict__ dst) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L) return;
  const int o = idx[perm ? perm[r] : r];
  if (o < 0) return;
  for (int k = 0; k < count; ++k)
    dst[static_cast<size_t>(k) * total + o] = src[static_cast<size_t>(k) * L + r];
}

// bbox[c*6 + k]: min (k < 3) / max of cluster c's positions (one CTA each).
__global__ void __launch_bounds__(kBlock) ens_bbox_kernel(const ClusterDev* __restrict__ cl,
                                                         const double* __restrict__ X, int L,
                                                         double* __restrict__ bbox) {
  __shared__ double sh[6 * 32];
  const ClusterDev k = cl[blockIdx.x];
  double v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int i = threadIdx.x; i < k.n; i += blockDim.x) {
    const int r = k.row0 + i;
    const double x = X[r], y = X[L + r], z = X[2 * L + r];
    v[0] = fmin(v[0], x); v[1] = fmin(v[1], y); v[2] = fmin(v[2], z);
    v[3] = fmax(v[3], x); v[4] = fmax(v[4], y); v[5] = fmax(v[5], z);
  }
  block_minmax6(v, sh);
#pragma unroll
  for (int q = 0; q < 6; ++q)
    if (threadIdx.x == q) bbox[blockIdx.x * 6 + q] = v[q];
}

// keys[r] = (segment cluster << 48) | 48-bit Hilbert index (16 bits per axis)
// in the cluster's box; padding rows take the segment's largest key, so the
// sorted rows of cluster c fill exactly its padded segment, bodies first.
__global__ void ens_key_kernel(int L, const int* __restrict__ cid, const int* __restrict__ seg,
                               const double* __restrict__ X, const double* __restrict__ bbox,
                               uint64_t* __restrict__ keys, int* __restrict__ vals) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= L) return;
  const int c = seg[r];
  uint64_t key = static_cast<uint64_t>(c) << 48;
  if (cid[r] < 0) {
    key |= 0xffffffffffffull;
  } else {
    constexpr double kCells = 65535.0;
    uint32_t cell[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double lo = bbox[c * 6 + k], w = bbox[c * 6 + 3 + k] - lo;
      double q = w > 0.0 ? (X[k * L + r] - lo) * (kCells / w) : 0.0;
      q = fmin(fmax(q, 0.0), kCells);  // NaN -> 0
      cell[k] = static_cast<uint32_t>(q);
    }
    key |= hilbert_key48(cell[0], cell[1], cell[2]);
  }
  keys[r] = key;
  vals[r] = r;
}

// The slot sums of row r (CTAs of kSumThreads: kSumRows<GR> rows of one cluster,
// GR groups), valid in group 0 of real rows; returns the row's cluster or -1.
template <int GR>
__device__ __forceinline__ int ens_slot_sums(int r, const int* __restrict__ cid,
                                             const ClusterDev* __restrict__ cl,
                                             const double* __restrict__ P, double sum[6], double* sh) {
  const int c = cid[r];
  const ClusterDev k = cl[max(c, 0)];
  const int i = c >= 0 ? r - k.row0 : 0;
  slot_sums<GR>(P + k.p_off, k.ld, c >= 0 ? RowSlots(k.S, k.block_rows, k.nb).count(i) : 0, i, sum, sh);
  return threadIdx.x < kSumRows<GR> ? c : -1;
}

template <int GR>
__global__ void __launch_bounds__(kSumThreads)
    ens_correct_kernel(int L, const int* __restrict__ cid, const ClusterDev* __restrict__ cl,
                       const double* __restrict__ P, double* __restrict__ X, double* __restrict__ V,
                       double* __restrict__ D) {
  __shared__ double sh[GR > 1 ? 6 * kSumThreads : 1];
  const int r = blockIdx.x * kSumRows<GR> + threadIdx.x % kSumRows<GR>;
  double sum[6];
  const int c = ens_slot_sums<GR>(r, cid, cl, P, sum, sh);
  if (c < 0) return;
  const double dt = cl[c].dt;
  const double idt2 = 1.0 / (dt * dt), idt3 = idt2 / dt;
  const double dt3 = dt * dt * dt, dt4 = dt3 * dt, dt5 = dt4 * dt;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double a1 = sum[q], j1 = sum[3 + q];
    const double a = D[q * L + r], j = D[(3 + q) * L + r];
    const double da = a - a1;
    const double a2 = 2.0 * idt2 * (-3.0 * da - (2.0 * j + j1) * dt);
    const double a3 = 6.0 * idt3 * (2.0 * da + (j + j1) * dt);
    X[q * L + r] += a2 * dt4 * (1.0 / 24.0) + a3 * dt5 * (1.0 / 120.0);
    V[q * L + r] += a2 * dt3 * (1.0 / 6.0) + a3 * dt4 * (1.0 / 24.0);
    D[q * L + r] = a1;
    D[(3 + q) * L + r] = j1;
  }
}

template <int GR>
__global__ void __launch_bounds__(kSumThreads)
    ens_reduce_kernel(int L, const int* __restrict__ cid, const ClusterDev* __restrict__ cl,
                      const double* __restrict__ P, double* __restrict__ D) {
  __shared__ double sh[GR > 1 ? 6 * kSumThreads : 1];
  const int r = blockIdx.x * kSumRows<GR> + threadIdx.x % kSumRows<GR>;
  double sum[6];
  if (ens_slot_sums<GR>(r, cid, cl, P, sum, sh) < 0) return;
#pragma unroll
  for (int f = 0; f < 6; ++f) D[f * L + r] = sum[f];
}

// phi[r] = sum over the same cluster's j != r of m_j / sqrt(r^2 + eps2_c);
// one CTA per 256-row block, blocks listed in `blk` as cluster ids.
__global__ void __launch_bounds__(kBlock) ens_phi_kernel(const int* __restrict__ blk_cluster,
                                                         const int* __restrict__ blk_row,
                                                         const ClusterDev* __restrict__ cl,
                                                         const JBody64* __restrict__ jb,
                                                         double* __restrict__ phi) {
  __shared__ double4 tile[kBlock];
  const ClusterDev k = cl[blk_cluster[blockIdx.x]];
  const int i = blk_row[blockIdx.x] + threadIdx.x;  // cluster-relative row
  const double2* pi = jb64_at(jb, k.row0 + i);
  const double2 pi0 = pi[0], pi1 = pi[32];
  const double4 bi = make_double4(pi0.x, pi0.y, pi1.x, pi1.y);
  double acc = 0.0;
  for (int j0 = 0; j0 < k.ld; j0 += kBlock) {
    const double2* pj = jb64_at(jb, k.row0 + j0 + threadIdx.x);
    const double2 pj0 = pj[0], pj1 = pj[32];
    tile[threadIdx.x] = make_double4(pj0.x, pj0.y, pj1.x, pj1.y);
    __syncthreads();
#pragma unroll 4
    for (int t = 0; t < kBlock; ++t) {
      const double4 p = tile[t];
      const double dx = p.x - bi.x, dy = p.y - bi.y, dz = p.z - bi.z;
      const double y = rsqrt_f64(fma(dx, dx, fma(dy, dy, fma(dz, dz, k.eps2))));
      acc += (j0 + t != i) ? p.w * y : 0.0;
    }
    __syncthreads();
  }
  phi[k.row0 + i] = acc;
}

// Per cluster (one CTA each): T = sum 0.5 m v^2, U = -0.5 sum m phi.
__global__ void ens_energy_sum_kernel(const ClusterDev* __restrict__ cl, const double* __restrict__ V,
                                      const double* __restrict__ M, const double* __restrict__ phi,
                                      int L, double* __restrict__ T, double* __restrict__ U) {
  __shared__ double sh[32];
  const ClusterDev k = cl[blockIdx.x];
  double t = 0.0, u = 0.0;
  for (int i = threadIdx.x; i < k.n; i += blockDim.x) {
    const int r = k.row0 + i;
    const double a = V[r], b = V[L + r], c = V[2 * L + r];
    t += 0.5 * M[r] * (a * a + b * b + c * c);
    u += M[r] * phi[r];
  }
  const double bt = block_sum(t, sh);
  const double bu = block_sum(u, sh);
  if (threadIdx.x == 0) {
    T[blockIdx.x] = bt;
    U[blockIdx.x] = -0.5 * bu;
  }
}

// Persistent-kernel shapes (all with 256-row items = one padding unit); the
// default is the first of a (precision, record format) or, for large near/far
// ensembles, the second; the autotuner times all of them.  The packed hi/lo
// default is one-sided with tiles of 128 by contract: its float sums, tile by
// tile, are those of the single-system hi/lo kernel (pair_variant 3), and its
// results stay what they are.  A symmetric hi/lo form sums in another order: it
// moved the worst body of 256 clusters (softening 4/N) by 8.5e-8 in 8 steps, a
// distance between the two forms and not an error.  Against FP64 sums the default
// has acc errors of 5.0e-8 / 2.7e-7 / 1.9e-6 (median / p99 / max, 32 clusters of
// 256-8192 bodies), the symmetric near/far kernel 4.3e-8 / 2.3e-7 / 1.7e-6; who
// wants its speed asks for pair_variant 4 (pair launch of 256 clusters of
// 256-8192 bodies 1.92 ms; hi/lo with two rows per thread and the j-loop
// unrolled four times 2.64, with four rows 2.74).
struct EnsKernel {
  int precision, nt, tile;
  int fmt;  // RecordFormat of its j-records
  const void* fn;
  size_t smem;
  bool sym = true;
};

template <int IPT, int W, int UNR, int MINB>
EnsKernel ens_sym_fp64() {
  return {NBODY_FP64, 32 * W, kSymTile64, kRecF64,
          reinterpret_cast<const void*>(&ensemble_sym_fp64_kernel<IPT, W, UNR, MINB>),
          sym_fp64_smem<IPT, W, UNR>()};
}
template <int IPT, int W, int SUB, int UNR, int NUNR, int MINB>
EnsKernel ens_sym_nf() {
  return {NBODY_MIXED, 32 * W, 64 * SUB, kRecSym,
          reinterpret_cast<const void*>(&ensemble_sym_nf_kernel<IPT, W, SUB, UNR, NUNR, MINB>),
          sym_nf_smem<IPT, W, SUB>()};
}
template <class R>
EnsKernel ens_hilo() {
  static_assert(R::ROWS == kPadRows, "an item's row block is one padding unit");
  return {NBODY_MIXED, R::NT, R::TJ, kRecX2, reinterpret_cast<const void*>(&ensemble_pair_kernel<R>),
          pair_smem_bytes<R>(), false};
}
template <class R>
EnsKernel ens_all_far() {
  static_assert(R::ROWS == kPadRows, "an item's row block is one padding unit");
  return {NBODY_MIXED, R::NT, R::TJ, kRecRel, reinterpret_cast<const void*>(&ensemble_pair_nf_kernel<R, 1>),
          2 * (R::TJ + 1) * sizeof(JBodyNF) + R::kExtraSmem, false};
}

const std::vector<EnsKernel>& ens_registry() {
  static const std::vector<EnsKernel> r = {
      ens_sym_fp64<2, 4, 4, 4>(),
      ens_sym_nf<2, 4, 1, 4, 8, 4>(),
      ens_sym_nf<4, 2, 1, 4, 2, 6>(),
      ens_hilo<RowsMixedX2<128, 2, 128, 1, 4>>(),
      ens_hilo<RowsMixedX2<64, 4, 128, 1, 1>>(),
      ens_hilo<RowsMixedX2<128, 2, 64, 1, 2>>(),
      ens_all_far<RowsMixedNF<64, 4, 64, 1, 1, 0>>(),
      ens_all_far<RowsMixedNF<128, 2, 128, 1, 1, 0>>(),
  };
  return r;
}

}  // namespace

struct nbody_ensemble {
  int C = 0, L = 0, dev = 0, sms = 0, precision = 0;
  int fmt = kRecF64;      // record format of the pair kernels in use
  bool ordered = false;   // clusters kept in Hilbert order (pair_variant 4, 5)
  int tiles_per_item = 8;
  const EnsKernel* kern = nullptr;  // persistent pair kernel in use
  int grid = 0;
  long long interactions = 0;  // sum of n_c^2 per step
  cudaStream_t stream = nullptr;
  std::vector<int> n, row0, ld;
  std::vector<double> eps2, dt;
  double* state = nullptr;  // [13][L]
  double *X = nullptr, *V = nullptr, *M = nullptr, *D = nullptr;
  double* P = nullptr;
  size_t p_doubles = 0;
  JBody64* jb64 = nullptr;
  void* jmix = nullptr;  // mixed records: SymSub, JBodyX2 or tiles of JBodyNF
  int* cid = nullptr;
  int* idx = nullptr;    // [L] padded row -> index in the caller's arrays, -1 on padding
  double* io = nullptr;  // [7][total] the caller's arrays on their way in or out
  int total = 0;         // bodies
  ClusterDev* cl = nullptr;
  EnsItem* items = nullptr;
  int n_items = 0;
  unsigned int* counter = nullptr;
  int* status = nullptr;
  int *blk_cluster = nullptr, *blk_row = nullptr;
  int n_blk = 0;
  double *phi = nullptr, *Tc = nullptr, *Uc = nullptr;
  cudaGraphExec_t graph = nullptr;  // one step with the event records of last_step_ms
  cudaGraphExec_t plain = nullptr;  // one step
  int step_kernels = 0;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  bool have_derivs = false;
  long long steps = 0;
  // Hilbert ordering (mixed, tile-relative variants): each cluster keeps its
  // bodies in Hilbert order within its segment; position r holds the body of
  // padded row perm[r] (the caller's order).
  int* perm = nullptr;            // [2][L]
  double* scratch = nullptr;      // [13][L]
  bool sorted = false, permuted = false;
  int* seg = nullptr;             // [L] cluster owning each padded row
  double* bbox = nullptr;         // [C][6]
  uint64_t* sort_keys = nullptr;  // [2][L]
  int* sort_idx = nullptr;        // [2][L]; second half = order
  void* sort_tmp = nullptr;
  size_t sort_tmp_bytes = 0;
  int sort_bits = 49, sort_every = 16, since_sort = 0;
  cudaGraphExec_t order_graph = nullptr;
  int order_kernels = 0;
  long long reorders = 0;
  int tile_unit() const { return precision == NBODY_FP64 ? kFp64ItemTile / kSymTile64 : 1; }
};

namespace {

nbody_status ens_status(nbody_ensemble* e) {
  int h = 0;
  EN_CUDA(cudaMemcpyAsync(&h, e->status, sizeof h, cudaMemcpyDeviceToHost, e->stream));
  EN_CUDA(cudaStreamSynchronize(e->stream));
  if (h) {
    cudaMemsetAsync(e->status, 0, sizeof(int), e->stream);
    return nbody_set_error(NBODY_ERR_TIMEOUT, "an ensemble pair-kernel wait exceeded its limit");
  }
  return NBODY_OK;
}

void drop_graphs(nbody_ensemble* e) {
  for (cudaGraphExec_t* g : {&e->graph, &e->plain}) {
    if (*g) cudaGraphExecDestroy(*g);
    *g = nullptr;
  }
}

// How cluster c is cut for kernel k: tiles that hold bodies (the padding rows of
// a segment come last, in the tile-relative order too, so whole padding tiles
// are skipped), blocks of 256 rows or, in clusters of more than kMaxSymBlocks
// of those, of several times that, and the splits of a block's run.
struct ClusterCut {
  int tiles, subs, block, nb, S;
  ClusterCut(const EnsKernel& k, int n, int tpi) {
    tiles = (n + k.tile - 1) / k.tile;
    subs = k.sym ? (n + kMaxSymBlocks * kPadRows - 1) / (kMaxSymBlocks * kPadRows) : 1;
    block = kPadRows * subs;
    nb = (n + block - 1) / block;
    S = (run(k, 0) + tpi - 1) / tpi;
  }
  int run(const EnsKernel& k, int I) const {  // tiles of block I's run
    return k.sym ? sym_q_count(nb, I, block / k.tile, tiles) : tiles;
  }
};

long count_items(const nbody_ensemble* e, int tpi) {
  long items = 0;
  for (int c = 0; c < e->C; ++c) {
    const ClusterCut k(*e->kern, e->n[c], tpi);
    items += static_cast<long>(k.nb) * k.S;
  }
  return items;
}

int default_tiles_per_item(const nbody_ensemble* e) {
  int tpi = 1;
  for (int bodies : kItemBodies) {
    tpi = std::max(1, bodies / e->kern->tile);
    if (count_items(e, tpi) >= kItemsPerCta * e->grid) break;
  }
  return tpi;
}

// (Re)builds the work list and partial-sum layout for `tpi` tiles per item.
nbody_status build_items(nbody_ensemble* e, int tpi) {
  std::vector<ClusterDev> cl(e->C);
  std::vector<EnsItem> items;
  long long p_off = 0;
  for (int c = 0; c < e->C; ++c) {
    const EnsKernel& kern = *e->kern;
    const ClusterCut k(kern, e->n[c], tpi);
    cl[c] = ClusterDev{e->row0[c], e->n[c], e->ld[c], k.S, k.block, kern.sym ? k.nb : 0, p_off, e->eps2[c], e->dt[c]};
    for (int rb = 0; rb < k.nb; ++rb)
      for (int s = 0; s < k.S; ++s) {
        EnsItem it;
        it.jrow0 = e->row0[c];
        it.row0 = rb * k.block;
        it.rows_end = e->n[c];
        it.ld = e->ld[c];
        it.S = k.S;
        it.nb = k.nb;
        it.subs = k.subs;
        it.split = s;
        it.p_off = kern.sym ? p_off : p_off + static_cast<long long>(s) * 6 * e->ld[c];
        it.eps2 = e->eps2[c];
        const int q0 = s * tpi;
        it.t_begin = kern.sym ? rb * (k.block / kern.tile) + q0 : q0;
        it.nt = std::max(0, std::min(tpi, k.run(kern, rb) - q0));  // 0: the item writes zeros to its slot
        items.push_back(it);
      }
    p_off += static_cast<long long>(k.S + (kern.sym ? k.nb / 2 : 0)) * 6 * e->ld[c];
  }
  // longest items first, then by cluster so neighbours share L2 lines
  std::stable_sort(items.begin(), items.end(),
                   [](const EnsItem& a, const EnsItem& b) { return a.nt * a.subs > b.nt * b.subs; });
  drop_graphs(e);
  EN_CUDA(cudaStreamSynchronize(e->stream));
  cudaFree(e->P);
  cudaFree(e->items);
  e->P = nullptr;
  e->items = nullptr;
  e->p_doubles = static_cast<size_t>(p_off);
  EN_CUDA(cudaMalloc(&e->P, sizeof(double) * e->p_doubles));
  EN_CUDA(cudaMalloc(&e->items, sizeof(EnsItem) * items.size()));
  EN_CUDA(cudaMemcpy(e->items, items.data(), sizeof(EnsItem) * items.size(), cudaMemcpyHostToDevice));
  EN_CUDA(cudaMemcpy(e->cl, cl.data(), sizeof(ClusterDev) * e->C, cudaMemcpyHostToDevice));
  e->n_items = static_cast<int>(items.size());
  e->tiles_per_item = tpi;
  return NBODY_OK;
}

SoA7 ens_state(nbody_ensemble* e) {
  const size_t L = e->L;
  return SoA7{e->X, e->X + L, e->X + 2 * L, e->M, e->V, e->V + L, e->V + 2 * L};
}

nbody_status launch_ens_pair(nbody_ensemble* e) {
  EN_CUDA(cudaMemsetAsync(e->counter, 0, sizeof(unsigned int), e->stream));
  const void* jb = e->fmt == kRecF64 ? static_cast<const void*>(e->jb64) : e->jmix;
  SoA7 rows = ens_state(e);
  RowSrc src{rows.x, rows.y, rows.z, rows.vx, rows.vy, rows.vz};
  void* args[] = {const_cast<void*>(static_cast<const void*>(&jb)), &e->items, &e->n_items,
                  &e->counter, &e->P, &e->status,
                  e->kern->sym ? static_cast<void*>(&rows) : static_cast<void*>(&src)};
  EN_CUDA(cudaLaunchKernel(e->kern->fn, dim3(e->grid), dim3(e->kern->nt), args, e->kern->smem,
                           e->stream));
  return NBODY_OK;
}

// Hilbert order of every cluster's bodies within its padded segment.
nbody_status ens_order(nbody_ensemble* e, cudaStream_t st) {
  ens_bbox_kernel<<<e->C, kBlock, 0, st>>>(e->cl, e->X, e->L, e->bbox);
  ens_key_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, st>>>(e->L, e->cid, e->seg, e->X,
                                                                  e->bbox, e->sort_keys, e->sort_idx);
  EN_CUDA(cudaGetLastError());
  const size_t L = e->L;
  size_t bytes = e->sort_tmp_bytes;
  EN_CUDA(cub::DeviceRadixSort::SortPairs(e->sort_tmp, bytes, e->sort_keys, e->sort_keys + L,
                                          e->sort_idx, e->sort_idx + L, e->L, 0, e->sort_bits, st));
  return NBODY_OK;
}

// Puts every cluster's bodies into Hilbert order within its segment: the
// order of ens_order, a gather of all 13 state arrays (and of perm) into
// scratch, and a copy back.  Capturable (the re-ordering graph).
nbody_status ens_reorder_state(nbody_ensemble* e, cudaStream_t st) {
  const size_t L = e->L;
  EN_TRY(ens_order(e, st));
  GatherArgs g;
  g.arrays = 13;
  for (int a = 0; a < 13; ++a) {
    g.src[a] = e->state + a * L;
    g.dst[a] = e->scratch + a * L;
  }
  gather_rows_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, st>>>(e->L, e->sort_idx + L, g,
                                                                     e->perm, e->perm + L);
  EN_CUDA(cudaGetLastError());
  EN_CUDA(cudaMemcpyAsync(e->state, e->scratch, sizeof(double) * 13 * L, cudaMemcpyDeviceToDevice, st));
  EN_CUDA(cudaMemcpyAsync(e->perm, e->perm + L, sizeof(int) * L, cudaMemcpyDeviceToDevice, st));
  e->sorted = e->permuted = true;
  e->since_sort = 0;
  return NBODY_OK;
}

// Records of the pair kernel in use from the state (tile-relative ones: in
// Hilbert order within each cluster segment); predict: of the predicted state.
nbody_status ens_records(nbody_ensemble* e, cudaStream_t st, bool predict) {
  const int blocks = (e->L + kBlock - 1) / kBlock;
  JBodyX2* jbx = e->fmt == kRecX2 ? static_cast<JBodyX2*>(e->jmix) : nullptr;
  if (e->fmt == kRecSym) {
    SymSub* out = static_cast<SymSub*>(e->jmix);
    if (predict)
      ens_tile_kernel<true><<<e->L / 64, 64, 0, st>>>(e->L, e->cid, e->cl, e->X, e->V, e->M, e->D, out);
    else
      ens_tile_kernel<false><<<e->L / 64, 64, 0, st>>>(e->L, e->cid, e->cl, e->X, e->V, e->M, e->D, out);
    EN_CUDA(cudaGetLastError());
    return NBODY_OK;
  }
  if (predict)
    ens_predict_kernel<<<blocks, kBlock, 0, st>>>(e->L, e->cid, e->cl, e->X, e->V, e->M, e->D,
                                                  e->fmt == kRecF64 ? e->jb64 : nullptr, jbx);
  else if (e->fmt != kRecRel)
    ens_pack_kernel<<<blocks, kBlock, 0, st>>>(e->L, e->cid, e->X, e->V, e->M,
                                               e->fmt == kRecF64 ? e->jb64 : nullptr, jbx);
  EN_CUDA(cudaGetLastError());
  if (e->fmt == kRecRel) {
    JBodyNF* out = static_cast<JBodyNF*>(e->jmix);
    const int tiles = e->L / e->kern->tile;
    switch (e->kern->tile) {
      case 64: rel_tile_nf_kernel<64><<<tiles, 64, 0, st>>>(e->L, ens_state(e), out, e->cid); break;
      case 128: rel_tile_nf_kernel<128><<<tiles, 128, 0, st>>>(e->L, ens_state(e), out, e->cid); break;
      default: return nbody_set_error(NBODY_ERR_INVALID_ARG, "no record builder for tile %d", e->kern->tile);
    }
    EN_CUDA(cudaGetLastError());
  }
  return NBODY_OK;
}

// Copies `count` [L] arrays starting at src to the caller's concatenated
// arrays (cluster c's n_c bodies in turn).
nbody_status ens_download(nbody_ensemble* e, const double* src, double* const* dst, int count) {
  ens_compact_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, e->stream>>>(
      e->L, e->total, count, e->idx, e->permuted ? e->perm : nullptr, src, e->io);
  EN_CUDA(cudaGetLastError());
  const size_t n = e->total;
  for (int k = 0; k < count; ++k)
    if (dst[k])
      EN_CUDA(cudaMemcpyAsync(dst[k], e->io + k * n, sizeof(double) * n, cudaMemcpyDeviceToHost, e->stream));
  EN_CUDA(cudaStreamSynchronize(e->stream));
  return NBODY_OK;
}

// Selects a persistent kernel: opts in to its shared memory and sizes the
// grid to the SMs x resident CTAs it reaches.
nbody_status use_kernel(nbody_ensemble* e, const EnsKernel* k) {
  EN_CUDA(cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(k->smem)));
  int occ = 0;
  EN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k->fn, k->nt, k->smem));
  e->kern = k;
  e->grid = e->sms * std::max(occ, 1);
  return NBODY_OK;
}

nbody_status launch_ens_pack(nbody_ensemble* e) {
  if (e->ordered && !e->sorted)  // tile-relative: bodies into Hilbert order first
    EN_TRY(ens_reorder_state(e, e->stream));
  return ens_records(e, e->stream, false);
}

// Whether the rows' slots are summed by eight groups of threads or by one thread:
// as sum_in_groups (hermite.cuh), by the mean over the rows.  512 clusters of 256
// to 8192 bodies, 1.2e6 rows of 3 slots on average: corrector 173 us in groups,
// 57 by one thread.
bool sum_by_groups(const nbody_ensemble* e) {
  return e->p_doubles >= static_cast<size_t>(kSumGroupSlots) * 6 * e->L;
}
// L is a multiple of 256
int sum_blocks(const nbody_ensemble* e, bool groups) { return e->L / (groups ? kSumRows<8> : kSumRows<1>); }

int count_graph_kernels(cudaGraph_t g) {
  size_t nodes = 0;
  int kernels = 0;
  if (cudaGraphGetNodes(g, nullptr, &nodes) == cudaSuccess && nodes > 0) {
    std::vector<cudaGraphNode_t> v(nodes);
    if (cudaGraphGetNodes(g, v.data(), &nodes) == cudaSuccess)
      for (size_t k = 0; k < nodes; ++k) {
        cudaGraphNodeType ty;
        if (cudaGraphNodeGetType(v[k], &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel)
          ++kernels;
      }
  }
  return kernels;
}

nbody_status ens_eval_current(nbody_ensemble* e) {
  EN_TRY(launch_ens_pack(e));
  EN_TRY(launch_ens_pair(e));
  const bool groups = sum_by_groups(e);
  (groups ? ens_reduce_kernel<8> : ens_reduce_kernel<1>)<<<sum_blocks(e, groups), kSumThreads, 0, e->stream>>>(
      e->L, e->cid, e->cl, e->P, e->D);
  EN_CUDA(cudaGetLastError());
  e->have_derivs = true;
  return NBODY_OK;
}

// Captures one step (timed: with its event records) into *out.
nbody_status ens_capture(nbody_ensemble* e, bool timed, cudaGraphExec_t* out) {
  if (*out) return NBODY_OK;
  cudaGraph_t g = nullptr;
  EN_CUDA(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
  nbody_status s = NBODY_OK;
  if (timed && cudaEventRecordWithFlags(e->ev[0], e->stream, cudaEventRecordExternal) != cudaSuccess)
    s = nbody_set_error(NBODY_ERR_CUDA, "event record during capture failed");
  if (s == NBODY_OK) s = ens_records(e, e->stream, true);
  if (s == NBODY_OK) s = launch_ens_pair(e);
  const bool groups = sum_by_groups(e);
  (groups ? ens_correct_kernel<8> : ens_correct_kernel<1>)<<<sum_blocks(e, groups), kSumThreads, 0, e->stream>>>(
      e->L, e->cid, e->cl, e->P, e->X, e->V, e->D);
  if (timed && s == NBODY_OK &&
      cudaEventRecordWithFlags(e->ev[1], e->stream, cudaEventRecordExternal) != cudaSuccess)
    s = nbody_set_error(NBODY_ERR_CUDA, "event record during capture failed");
  cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
  if (s != NBODY_OK) {
    if (g) cudaGraphDestroy(g);
    return s;
  }
  if (ce != cudaSuccess) return nbody_set_error(NBODY_ERR_CUDA, "capture: %s", cudaGetErrorString(ce));
  if (timed) e->step_kernels = count_graph_kernels(g);
  ce = cudaGraphInstantiate(out, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) {
    *out = nullptr;
    return nbody_set_error(NBODY_ERR_CUDA, "instantiate: %s", cudaGetErrorString(ce));
  }
  return NBODY_OK;
}

nbody_status ens_build_graph(nbody_ensemble* e) {
  if (e->graph) return NBODY_OK;
  EN_TRY(ens_capture(e, true, &e->graph));
  cudaGraph_t g = nullptr;
  nbody_status s = NBODY_OK;
  cudaError_t ce = cudaSuccess;
  if (e->ordered && !e->order_graph) {
    const bool sorted = e->sorted, permuted = e->permuted;
    const int since = e->since_sort;
    EN_CUDA(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
    s = ens_reorder_state(e, e->stream);
    ce = cudaStreamEndCapture(e->stream, &g);
    e->sorted = sorted;  // capturing ran nothing
    e->permuted = permuted;
    e->since_sort = since;
    if (s != NBODY_OK) {
      if (g) cudaGraphDestroy(g);
      return s;
    }
    if (ce != cudaSuccess) return nbody_set_error(NBODY_ERR_CUDA, "capture: %s", cudaGetErrorString(ce));
    e->order_kernels = count_graph_kernels(g);
    ce = cudaGraphInstantiate(&e->order_graph, g, 0);
    cudaGraphDestroy(g);
    if (ce != cudaSuccess) {
      e->order_graph = nullptr;
      return nbody_set_error(NBODY_ERR_CUDA, "instantiate: %s", cudaGetErrorString(ce));
    }
  }
  return NBODY_OK;
}

// Times the pair launch for every (kernel shape, item size) pair, the default's
// sizes among them, and keeps the pair with the least time of launch and slot
// sums (short items leave many slots).  Items count j-tiles, so tiles_per_item
// x tile = j per item.
nbody_status ens_autotune(nbody_ensemble* e) {
  EN_TRY(launch_ens_pack(e));
  cudaEvent_t a, b;
  EN_CUDA(cudaEventCreate(&a));
  EN_CUDA(cudaEventCreate(&b));
  float best = 1e30f;
  const EnsKernel* best_k = e->kern;
  int best_tpi = 8;
  for (const EnsKernel& k : ens_registry()) {
    if (k.precision != e->precision || k.fmt != e->fmt) continue;
    EN_TRY(use_kernel(e, &k));
    if (e->fmt == kRecRel) EN_TRY(ens_records(e, e->stream, false));  // this kernel's tile size
    // shorter items than 256 bodies only where the default takes them: they
    // leave the most slots
    const int least = std::min(std::max(1, 256 / k.tile), default_tiles_per_item(e));
    int last_tpi = 0;
    for (int j_per_item : {64, 128, 256, 512, 1024, 2048, 4096, 8192}) {
      const int tpi = std::max(1, j_per_item / k.tile);
      if (tpi == last_tpi || tpi < least) continue;
      last_tpi = tpi;
      EN_TRY(build_items(e, tpi));
      EN_TRY(launch_ens_pair(e));
      EN_CUDA(cudaEventRecord(a, e->stream));
      for (int r = 0; r < 2; ++r) EN_TRY(launch_ens_pair(e));
      EN_CUDA(cudaEventRecord(b, e->stream));
      EN_CUDA(cudaEventSynchronize(b));
      float ms = 0;
      EN_CUDA(cudaEventElapsedTime(&ms, a, b));
      const float pair_ms = ms / 2;
      ms = pair_ms + static_cast<float>(8.0 * e->p_doubles / kSplitSumBytesPerMs);
      if (getenv("NBODY_TUNE_VERBOSE"))
        fprintf(stderr, "[nbody ens tune] nt=%d tile=%d tiles_per_item=%d  %.4f ms (pair %.4f)\n", k.nt,
                k.tile, tpi, ms, pair_ms);
      if (ms < best) {
        best = ms;
        best_k = &k;
        best_tpi = tpi;
      }
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  EN_TRY(ens_status(e));
  EN_TRY(use_kernel(e, best_k));
  if (e->fmt == kRecRel) EN_TRY(ens_records(e, e->stream, false));
  return build_items(e, best_tpi);
}

nbody_status ens_check(nbody_ensemble* e) {
  if (!e) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null ensemble");
  if (cudaSetDevice(e->dev) != cudaSuccess) return nbody_set_error(NBODY_ERR_CUDA, "cudaSetDevice failed");
  return NBODY_OK;
}

}  // namespace

extern "C" {

nbody_status nbody_ensemble_destroy(nbody_ensemble* e) {
  if (!e) return NBODY_OK;
  cudaSetDevice(e->dev);
  if (e->stream) cudaStreamSynchronize(e->stream);
  drop_graphs(e);
  if (e->order_graph) cudaGraphExecDestroy(e->order_graph);
  for (auto ev : e->ev)
    if (ev) cudaEventDestroy(ev);
  void* bufs[] = {e->state, e->P, e->jb64, e->jmix, e->cid, e->cl, e->items, e->counter,
                  e->status, e->blk_cluster, e->blk_row, e->phi, e->Tc, e->Uc,
                  e->idx, e->io, e->seg, e->bbox, e->sort_keys, e->sort_idx, e->sort_tmp, e->perm, e->scratch};
  for (void* p : bufs) cudaFree(p);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
  return NBODY_OK;
}

nbody_status nbody_ensemble_create(nbody_ensemble** out, const nbody_ensemble_config* cfg) {
  if (!out || !cfg || !cfg->n || !cfg->eps2 || !cfg->dt)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "null ensemble argument");
  *out = nullptr;
  const int C = cfg->nclusters;
  if (C < 1) return nbody_set_error(NBODY_ERR_INVALID_ARG, "nclusters = %d", C);
  if (cfg->precision != NBODY_FP64 && cfg->precision != NBODY_MIXED)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "precision = %d", cfg->precision);
  if (cfg->tiles_per_item < 0) return nbody_set_error(NBODY_ERR_INVALID_ARG, "tiles_per_item < 0");
  if (cfg->precision == NBODY_MIXED && cfg->pair_variant != 0 && cfg->pair_variant != 3 &&
      cfg->pair_variant != 4 && cfg->pair_variant != 5)
    return nbody_set_error(NBODY_ERR_INVALID_ARG,
                           "ensemble pair_variant = %d (0 automatic = packed hi/lo, 3 packed hi/lo, "
                           "4 near/far tile-relative, 5 plain tile-relative)", cfg->pair_variant);
  if (cfg->sort_every < 0) return nbody_set_error(NBODY_ERR_INVALID_ARG, "sort_every < 0");
  const bool rel = cfg->precision == NBODY_MIXED && (cfg->pair_variant == 4 || cfg->pair_variant == 5);
  if (rel && C > 65536)
    return nbody_set_error(NBODY_ERR_INVALID_ARG,
                           "tile-relative ensembles hold at most 65536 clusters (use pair_variant 3)");
  long long L = 0;
  for (int c = 0; c < C; ++c) {
    if (cfg->n[c] < 1) return nbody_set_error(NBODY_ERR_INVALID_ARG, "cluster %d has n = %d", c, cfg->n[c]);
    if (!(cfg->eps2[c] >= 1e-30 && cfg->eps2[c] <= 1e30))
      return nbody_set_error(NBODY_ERR_INVALID_ARG, "cluster %d eps2 = %g", c, cfg->eps2[c]);
    if (cfg->precision == NBODY_MIXED && cfg->eps2[c] < kMinEps2Mixed)
      return nbody_set_error(NBODY_ERR_INVALID_ARG, "cluster %d eps2 = %g below %g (mixed precision)",
                             c, cfg->eps2[c], kMinEps2Mixed);
    if (!(cfg->dt[c] > 0)) return nbody_set_error(NBODY_ERR_INVALID_ARG, "cluster %d dt = %g (ensembles use fixed steps)", c, cfg->dt[c]);
    L += (cfg->n[c] + kPadRows - 1) / kPadRows * kPadRows;
  }
  if (L > (1LL << 28)) return nbody_set_error(NBODY_ERR_INVALID_ARG, "ensemble too large");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return nbody_set_error(NBODY_ERR_NO_DEVICE, "no CUDA device visible");
  if (cfg->device < 0 || cfg->device >= ndev)
    return nbody_set_error(NBODY_ERR_INVALID_ARG, "device %d of %d", cfg->device, ndev);
  int major = 0;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, cfg->device);
  if (major != 10) return nbody_set_error(NBODY_ERR_NO_DEVICE, "device %d is not sm_100", cfg->device);
  EN_CUDA(cudaSetDevice(cfg->device));

  std::unique_ptr<nbody_ensemble> e(new nbody_ensemble);
  e->C = C;
  e->L = static_cast<int>(L);
  e->dev = cfg->device;
  e->precision = cfg->precision;
  e->fmt = cfg->precision == NBODY_FP64 ? kRecF64
           : cfg->pair_variant == 4     ? kRecSym
           : cfg->pair_variant == 5     ? kRecRel
                                        : kRecX2;
  e->ordered = rel;
  e->sort_every = cfg->sort_every > 0 ? cfg->sort_every : 16;
  while ((1LL << (e->sort_bits - 48)) < C) ++e->sort_bits;  // cluster id above the 48-bit code
  cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->dev);
  e->n.assign(cfg->n, cfg->n + C);
  e->eps2.assign(cfg->eps2, cfg->eps2 + C);
  e->dt.assign(cfg->dt, cfg->dt + C);
  std::vector<int> cid(e->L, -1), idx(e->L, -1), seg(e->L, 0), blk_cluster, blk_row;
  int r0 = 0;
  for (int c = 0; c < C; ++c) {
    const int ld = (e->n[c] + kPadRows - 1) / kPadRows * kPadRows;
    e->row0.push_back(r0);
    e->ld.push_back(ld);
    for (int i = 0; i < e->n[c]; ++i) {
      cid[r0 + i] = c;
      idx[r0 + i] = e->total++;
    }
    for (int i = 0; i < ld; ++i) seg[r0 + i] = c;
    for (int b = 0; b < ld; b += kPadRows) {
      blk_cluster.push_back(c);
      blk_row.push_back(b);
    }
    e->interactions += static_cast<long long>(e->n[c]) * e->n[c];
    r0 += ld;
  }
  e->n_blk = static_cast<int>(blk_cluster.size());
  nbody_ensemble* raw = e.get();
  auto body = [&]() -> nbody_status {
    EN_CUDA(cudaStreamCreateWithFlags(&raw->stream, cudaStreamNonBlocking));
    const size_t Ls = raw->L;
    EN_CUDA(cudaMalloc(&raw->state, sizeof(double) * 13 * Ls));
    EN_CUDA(cudaMemset(raw->state, 0, sizeof(double) * 13 * Ls));
    raw->X = raw->state;
    raw->V = raw->state + 3 * Ls;
    raw->M = raw->state + 6 * Ls;
    raw->D = raw->state + 7 * Ls;
    EN_CUDA(cudaMalloc(&raw->jb64, sizeof(JBody64) * Ls));
    // subtiles of 64 bodies, packed hi/lo records, or tiles of TJ + 1 JBodyNF (TJ >= 64)
    static_assert(sizeof(JBodyNF) >= sizeof(JBodyX2), "jmix sized by the larger record");
    if (raw->precision == NBODY_MIXED)
      EN_CUDA(cudaMalloc(&raw->jmix, (Ls / 64) * (raw->fmt == kRecSym ? sizeof(SymSub) : 65 * sizeof(JBodyNF))));
    EN_CUDA(cudaMalloc(&raw->cid, sizeof(int) * Ls));
    EN_CUDA(cudaMemcpy(raw->cid, cid.data(), sizeof(int) * Ls, cudaMemcpyHostToDevice));
    EN_CUDA(cudaMalloc(&raw->idx, sizeof(int) * Ls));
    EN_CUDA(cudaMemcpy(raw->idx, idx.data(), sizeof(int) * Ls, cudaMemcpyHostToDevice));
    EN_CUDA(cudaMalloc(&raw->io, sizeof(double) * 7 * raw->total));
    EN_CUDA(cudaMalloc(&raw->cl, sizeof(ClusterDev) * raw->C));
    EN_CUDA(cudaMalloc(&raw->counter, sizeof(unsigned int)));
    EN_CUDA(cudaMalloc(&raw->status, sizeof(int)));
    EN_CUDA(cudaMemset(raw->status, 0, sizeof(int)));
    EN_CUDA(cudaMalloc(&raw->blk_cluster, sizeof(int) * raw->n_blk));
    EN_CUDA(cudaMalloc(&raw->blk_row, sizeof(int) * raw->n_blk));
    EN_CUDA(cudaMemcpy(raw->blk_cluster, blk_cluster.data(), sizeof(int) * raw->n_blk, cudaMemcpyHostToDevice));
    EN_CUDA(cudaMemcpy(raw->blk_row, blk_row.data(), sizeof(int) * raw->n_blk, cudaMemcpyHostToDevice));
    EN_CUDA(cudaMalloc(&raw->phi, sizeof(double) * Ls));
    EN_CUDA(cudaMalloc(&raw->Tc, sizeof(double) * raw->C));
    EN_CUDA(cudaMalloc(&raw->Uc, sizeof(double) * raw->C));
    if (raw->ordered) {
      EN_CUDA(cudaMalloc(&raw->seg, sizeof(int) * Ls));
      EN_CUDA(cudaMemcpy(raw->seg, seg.data(), sizeof(int) * Ls, cudaMemcpyHostToDevice));
      EN_CUDA(cudaMalloc(&raw->bbox, sizeof(double) * 6 * raw->C));
      EN_CUDA(cudaMalloc(&raw->sort_keys, sizeof(uint64_t) * 2 * Ls));
      EN_CUDA(cudaMalloc(&raw->sort_idx, sizeof(int) * 2 * Ls));
      EN_CUDA(cudaMalloc(&raw->perm, sizeof(int) * 2 * Ls));
      iota_kernel<<<(raw->L + kBlock - 1) / kBlock, kBlock, 0, raw->stream>>>(raw->L, raw->perm);
      EN_CUDA(cudaGetLastError());
      EN_CUDA(cudaMalloc(&raw->scratch, sizeof(double) * 13 * Ls));
      EN_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, raw->sort_tmp_bytes, raw->sort_keys,
                                              raw->sort_keys + Ls, raw->sort_idx,
                                              raw->sort_idx + Ls, raw->L, 0, raw->sort_bits,
                                              raw->stream));
      EN_CUDA(cudaMalloc(&raw->sort_tmp, std::max<size_t>(raw->sort_tmp_bytes, 16)));
    }
    for (auto& ev : raw->ev) EN_CUDA(cudaEventCreate(&ev));
    // the first shape, or the second where there are several long items for
    // each of its CTAs (pair launch of 256 clusters of 256-8192 bodies 2.04 vs
    // 1.96 ms, of 64 0.543 vs 0.539, of 256 of 256-2048 0.27 vs 0.28)
    const EnsKernel* first = nullptr;
    for (const EnsKernel& k : ens_registry()) {
      if (k.precision != raw->precision || k.fmt != raw->fmt) continue;
      if (first && (!k.sym || count_items(raw, kItemBodies[0] / k.tile) < 4L * raw->sms * kWideCtasPerSm)) break;
      EN_TRY(use_kernel(raw, &k));
      if (first) break;
      first = &k;
    }
    if (cfg->tiles_per_item == 0) return build_items(raw, default_tiles_per_item(raw));
    return build_items(raw, std::min(cfg->tiles_per_item, 1 << 28) * raw->tile_unit());
  };
  nbody_status s = body();
  if (s != NBODY_OK) {
    nbody_ensemble_destroy(e.release());
    return s;
  }
  if (cfg->tune && cfg->tiles_per_item == 0) e->tiles_per_item = -1;  // tune at first state
  *out = e.release();
  return NBODY_OK;
}

nbody_status nbody_ensemble_set_state(nbody_ensemble* e, const double* x, const double* y,
                                      const double* z, const double* m, const double* vx,
                                      const double* vy, const double* vz) {
  EN_TRY(ens_check(e));
  const double* src[7] = {x, y, z, vx, vy, vz, m};
  for (auto p : src)
    if (!p) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null state array");
  const size_t L = e->L;
  const size_t n = e->total;
  for (int k = 0; k < 7; ++k)  // state order: x, y, z, vx, vy, vz, m
    EN_CUDA(cudaMemcpyAsync(e->io + k * n, src[k], sizeof(double) * n, cudaMemcpyHostToDevice, e->stream));
  ens_expand_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, e->stream>>>(e->L, e->total, 7, e->idx,
                                                                          e->io, e->state);
  EN_CUDA(cudaGetLastError());
  EN_CUDA(cudaMemsetAsync(e->D, 0, sizeof(double) * 6 * L, e->stream));
  if (e->perm) {  // the caller's order again; re-ordered before the next evaluation
    iota_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, e->stream>>>(e->L, e->perm);
    EN_CUDA(cudaGetLastError());
  }
  e->sorted = e->permuted = false;
  EN_TRY(launch_ens_pack(e));
  EN_CUDA(cudaStreamSynchronize(e->stream));
  e->have_derivs = false;
  e->steps = 0;
  if (e->tiles_per_item < 0) EN_TRY(ens_autotune(e));
  return NBODY_OK;
}

nbody_status nbody_ensemble_get_state(nbody_ensemble* e, double* x, double* y, double* z,
                                      double* vx, double* vy, double* vz) {
  EN_TRY(ens_check(e));
  double* dst[6] = {x, y, z, vx, vy, vz};
  EN_TRY(ens_download(e, e->X, dst, 6));  // X(3) and V(3) are consecutive state arrays
  return ens_status(e);
}

nbody_status nbody_ensemble_get_derivs(nbody_ensemble* e, double* ax, double* ay, double* az,
                                       double* jx, double* jy, double* jz) {
  EN_TRY(ens_check(e));
  if (!e->have_derivs) return nbody_set_error(NBODY_ERR_STATE, "no derivatives yet");
  double* dst[6] = {ax, ay, az, jx, jy, jz};
  EN_TRY(ens_download(e, e->D, dst, 6));
  return ens_status(e);
}

nbody_status nbody_ensemble_acc_jerk(nbody_ensemble* e) {
  EN_TRY(ens_check(e));
  return ens_eval_current(e);
}

nbody_status nbody_ensemble_step(nbody_ensemble* e, int nsteps) {
  TraceRange trace_("nbody_ensemble_step");
  EN_TRY(ens_check(e));
  if (nsteps < 0) return nbody_set_error(NBODY_ERR_INVALID_ARG, "nsteps < 0");
  if (!e->have_derivs) EN_TRY(ens_eval_current(e));
  EN_TRY(ens_build_graph(e));
  for (int k = 0; k < nsteps; ++k) {
    if (e->ordered && e->since_sort >= e->sort_every) {
      EN_CUDA(cudaGraphLaunch(e->order_graph, e->stream));
      e->since_sort = 0;
      ++e->reorders;
    }
    if (k + 1 < nsteps) EN_TRY(ens_capture(e, false, &e->plain));
    EN_CUDA(cudaGraphLaunch(k + 1 < nsteps ? e->plain : e->graph, e->stream));
    ++e->since_sort;
  }
  e->steps += nsteps;
  return NBODY_OK;
}

nbody_status nbody_ensemble_synchronize(nbody_ensemble* e) {
  EN_TRY(ens_check(e));
  EN_CUDA(cudaStreamSynchronize(e->stream));
  return ens_status(e);
}

nbody_status nbody_ensemble_energy(nbody_ensemble* e, double* T, double* U) {
  EN_TRY(ens_check(e));
  if (!T || !U) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null energy arrays");
  ens_pack_kernel<<<(e->L + kBlock - 1) / kBlock, kBlock, 0, e->stream>>>(e->L, e->cid, e->X, e->V,
                                                                        e->M, e->jb64);
  ens_phi_kernel<<<e->n_blk, kBlock, 0, e->stream>>>(e->blk_cluster, e->blk_row, e->cl, e->jb64, e->phi);
  ens_energy_sum_kernel<<<e->C, kBlock, 0, e->stream>>>(e->cl, e->V, e->M, e->phi, e->L, e->Tc, e->Uc);
  EN_CUDA(cudaGetLastError());
  EN_CUDA(cudaMemcpyAsync(T, e->Tc, sizeof(double) * e->C, cudaMemcpyDeviceToHost, e->stream));
  EN_CUDA(cudaMemcpyAsync(U, e->Uc, sizeof(double) * e->C, cudaMemcpyDeviceToHost, e->stream));
  EN_CUDA(cudaStreamSynchronize(e->stream));
  return NBODY_OK;
}

nbody_status nbody_ensemble_info(nbody_ensemble* e, nbody_ensemble_info_t* out) {
  EN_TRY(ens_check(e));
  if (!out) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null info");
  EN_CUDA(cudaStreamSynchronize(e->stream));
  memset(out, 0, sizeof *out);
  out->nclusters = e->C;
  out->padded_rows = e->L;
  out->items = e->n_items;
  const int unit = e->tile_unit();
  out->tiles_per_item = e->tiles_per_item < 0 ? -1 : (e->tiles_per_item + unit - 1) / unit;
  out->j_tile = e->kern->tile * unit;
  out->threads = e->kern->nt;
  out->grid = e->grid;
  out->interactions_per_step = static_cast<double>(e->interactions);
  out->steps = e->steps;
  float ms = 0;
  if (e->graph && cudaEventElapsedTime(&ms, e->ev[0], e->ev[1]) == cudaSuccess) out->last_step_ms = ms;
  cudaGetLastError();
  out->record_format = e->fmt == kRecSym ? kRecRel : e->fmt;
  out->step_kernels = e->step_kernels;
  out->reorders = e->reorders;
  out->order_kernels = e->order_kernels;
  return NBODY_OK;
}

nbody_status nbody_ensemble_get_stream(nbody_ensemble* e, void** stream) {
  EN_TRY(ens_check(e));
  if (!stream) return nbody_set_error(NBODY_ERR_INVALID_ARG, "null stream out");
  *stream = e->stream;
  return NBODY_OK;
}

}  // extern "C"
