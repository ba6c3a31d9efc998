// Symmetric O(N^2) pair kernels: every unordered pair of bodies once.
//
// The one-sided kernels (pair.cuh) evaluate each pair twice, once for either
// body.  Here the pair's separation, 1/sqrt, and tidal vector are formed once
// and added to both bodies (Newton's third law): 38 FP64 operations per pair
// instead of 2 x 31, 32 FP32 lane operations (38 near) instead of 2 x 25 (31).
// The pair kernels are bound by their arithmetic pipe, so the fewer operations
// are the gain.
//
// Schedule.  Rows are cut into nb blocks of `block_rows` rows.  Block I meets
// the D(I) blocks that follow it cyclically (all blocks at distance 1 ..
// (nb-1)/2; for an even nb the distance nb/2 belongs to the lower half), so
// every pair of different blocks is met exactly once and all blocks have the
// same work; its own block (distance 0) is evaluated one-sided.  In tiles of
// TJ bodies that is one contiguous cyclic run of q_count(I) tiles from the
// block's own first tile, which the S splits (blockIdx.y) share.
//
// Inside a CTA each of W warps holds 32 * IPT rows in registers and all warps
// stream the same j-tiles through shared memory.  For a subtile of 32 bodies
// lane l reads body (l + k) & 31 at step k, adds the pair to its own rows and
// to that body's six sums, and hands the sums to the next lane (shuffles, so
// that they follow their body); after 32 steps they are home.  The W warps'
// sums are added in shared memory, in warp order, and stored.
//
// Partial sums are slots of P, [slot][6][stride]: the rows' own sums of split
// s in slot s, the sums a block at distance d adds to its partners in slot
// S + d - 1.  Every (slot, row) is written by exactly one thread, and slot
// sums run in slot order, so results are bitwise reproducible.  A row's slot
// count is RowSlots::count.  The schedule's arithmetic is in symplan.h.
//
// Large systems: a block is `subs` sub-blocks of 32 * IPT * W rows, which the
// CTA works through one after another over the same tiles, adding to the slots
// it wrote itself; this bounds the slots (nb / 2 + S) whatever N is.
#pragma once
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hermite.cuh"
#include "pair.cuh"
#include "reltiles.cuh"
#include "symplan.h"

namespace nbody {

struct SymArgs {
  int n, ld;       // bodies, padded rows (records exist for rows < ld)
  int nb, subs;    // blocks, sub-blocks per block
  int S;           // splits of a block's tile run
  int tiles;       // tiles that hold bodies: ceil(n / TJ)
  double eps2;
  double* out;     // P
  size_t stride;
  int* status;
  SoA7 rows;       // near/far kernel: the bodies its tiles were built from
  unsigned long long* near_count;  // near/far kernel: += near (warp, subtile) pairs (nullable)
};

// The tile run of one CTA (SymSpan) as the kernels stream it.
struct SymRun : SymSpan {
  __device__ __forceinline__ SymRun(int I_, int nb_, int tb_, int tiles_, int first_, int nq_, int split_)
      : SymSpan(I_, nb_, tb_, tiles_, first_, nq_, split_) {}
  // CTA (blockIdx.x, blockIdx.y) = (block, split) of a grid
  __device__ __forceinline__ SymRun(const SymArgs& a, int tb_)
      : SymSpan(blockIdx.x, a.nb, tb_, a.tiles, a.S, blockIdx.y) {}
  // Streams the run, tiles of TJ records, through `pipe` (it wraps at most once).
  template <class JB, int TJ, class Consume, class Post>
  __device__ __forceinline__ bool stream(TilePipe<JB, TJ>& pipe, const JB* src, int* status,
                                         Consume&& consume, Post&& post) const {
    for (int done = 0; done < nq;) {
      const int t0 = tile(done);
      const int run = min(nq - done, tiles - t0);
      if (!pipe.run(src + static_cast<size_t>(t0) * TJ, run, status, consume, post)) return false;
      done += run;
    }
    return true;
  }
};

// ---------------------------------------------------------------------------
// FP64
// ---------------------------------------------------------------------------
// One pair in double: i-row r against the j-body p0..p3 (jb64 chunks).
// SYM adds the pair to the j-body's sums bj = (acc, jerk), with the sign of
// the i-side (the caller negates).
template <bool SYM>
__device__ __forceinline__ void sym_pair_fp64(const double2& p0, const double2& p1,
                                              const double2& p2, const double2& p3, double xi,
                                              double yi, double zi, double ui, double vi, double wi,
                                              double mi, double eps2, double* ai, double* bj) {
  const double dx = p0.x - xi, dy = p0.y - yi, dz = p1.x - zi;
  const double du = p2.x - ui, dv = p2.y - vi, dw = p3.x - wi;
  const double s = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
  const double rv = fma(dx, du, fma(dy, dv, dz * dw));
  const double y = rsqrt_f64(s);
  const double y2 = y * y;
  const double y3 = y * y2;
  const double q = p1.y * y3, h = SYM ? mi * y3 : 0.0;
  const double c = rv * (-3.0 * y2);
  const double ex = fma(c, dx, du), ey = fma(c, dy, dv), ez = fma(c, dz, dw);
  ai[0] = fma(q, dx, ai[0]); ai[1] = fma(q, dy, ai[1]); ai[2] = fma(q, dz, ai[2]);
  ai[3] = fma(q, ex, ai[3]); ai[4] = fma(q, ey, ai[4]); ai[5] = fma(q, ez, ai[5]);
  if (SYM) {
    bj[0] = fma(h, dx, bj[0]); bj[1] = fma(h, dy, bj[1]); bj[2] = fma(h, dz, bj[2]);
    bj[3] = fma(h, ex, bj[3]); bj[4] = fma(h, ey, bj[4]); bj[5] = fma(h, ez, bj[5]);
  }
}

// A tile is one group of 32 FP64 records (2 KB).  Bound by the FP64 pipe;
// four rows per lane make the 12 shuffles and four 16-byte shared loads of a
// step (28 cycles of the shared pipe) hide under 4 x 38 FP64 instructions (76
// cycles), and the unrolled pair of steps gives the scheduler eight
// independent chains, so two CTAs of four warps per SM are as fast as three
// with spills.  Measured against the one-sided kernel at its best tiling:
// N = 65536 5.67 vs 8.24 ms, 16384 0.380 vs 0.539, 4096 0.034 vs 0.044.
constexpr int kSymTile64 = 32;

template <int IPT, int W, int UNR>
constexpr size_t sym_fp64_smem() {
  return 2 * kSymTile64 * sizeof(JBody64) + 2 * 6 * W * 32 * sizeof(double);
}

// One run of a CTA of W warps: `half` is the half of `red` ([2][6][W][32]) of
// the current tile, alternating over the CTA's life.  False if a wait timed out.
template <int IPT, int W, int UNR>
__device__ __forceinline__ bool sym_fp64_rows(TilePipe<JBody64, kSymTile64>& pipe, double* red, int& half,
                                              const JBody64* __restrict__ jb, const SymRun& run,
                                              const SymArgs& a) {
  constexpr int kRows = 32 * IPT * W;
  static_assert(kRows % kSymTile64 == 0, "blocks are whole tiles");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, next = (lane + 1) & 31;
  const double eps2 = a.eps2;
  for (int g = 0; g < a.subs; ++g) {
    const int row0 = (run.I * a.subs + g) * kRows + warp * 32 * IPT;
    if ((run.I * a.subs + g) * kRows >= a.n) break;  // a short last block
    double xi[IPT], yi[IPT], zi[IPT], ui[IPT], vi[IPT], wi[IPT], mi[IPT], acc[IPT][6];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      double2 p0{0, 0}, p1{0, 0}, p2{0, 0}, p3{0, 0};
      if (r < a.ld) {  // rows in [n, ld) are zero-mass records, rows past ld have none
        const double2* p = jb64_at(jb, r);
        p0 = p[0]; p1 = p[32]; p2 = p[64]; p3 = p[96];
      }
      xi[k] = p0.x; yi[k] = p0.y; zi[k] = p1.x; mi[k] = p1.y;
      ui[k] = p2.x; vi[k] = p2.y; wi[k] = p3.x;
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[k][c] = 0.0;
    }
    int t = 0;
    auto consume = [&](const JBody64* tile) {
      const double2* p = reinterpret_cast<const double2*>(tile);
      if (run.distance(run.tile(t)) == 0) {
#pragma unroll 1
        for (int k = 0; k < 32; ++k) {
          const double2 p0 = p[k], p1 = p[32 + k], p2 = p[64 + k], p3 = p[96 + k];
#pragma unroll
          for (int r = 0; r < IPT; ++r)
            sym_pair_fp64<false>(p0, p1, p2, p3, xi[r], yi[r], zi[r], ui[r], vi[r], wi[r], mi[r],
                                 eps2, acc[r], nullptr);
        }
      } else {
        double b[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll UNR
        for (int k = 0; k < 32; ++k) {
          const int j = (lane + k) & 31;
          const double2 p0 = p[j], p1 = p[32 + j], p2 = p[64 + j], p3 = p[96 + j];
#pragma unroll
          for (int r = 0; r < IPT; ++r)
            sym_pair_fp64<true>(p0, p1, p2, p3, xi[r], yi[r], zi[r], ui[r], vi[r], wi[r], mi[r],
                                eps2, acc[r], b);
#pragma unroll
          for (int c = 0; c < 6; ++c) b[c] = __shfl_sync(0xffffffffu, b[c], next);
        }
        double* o = red + half * 6 * W * 32 + warp * 32 + lane;
#pragma unroll
        for (int c = 0; c < 6; ++c) o[c * W * 32] = b[c];
      }
    };
    // after the tile's barrier: the W warps' sums of the tile's bodies, in warp
    // order, into their slot.  The next tile fills the other half of `red`.
    auto post = [&]() {
      const int tt = run.tile(t), d = run.distance(tt);
      if (d != 0) {
        const double* o = red + half * 6 * W * 32;
        double* out = a.out + static_cast<size_t>(a.S + d - 1) * 6 * a.stride +
                      static_cast<size_t>(tt) * kSymTile64;
        for (int e = threadIdx.x; e < 6 * 32; e += 32 * W) {
          const int l = e & 31, c = e >> 5;
          double v = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) v -= o[(c * W + w) * 32 + l];
          double* dst = out + static_cast<size_t>(c) * a.stride + l;
          *dst = g ? *dst + v : v;  // a later sub-block adds to this thread's own store
        }
      }
      ++t;
      half ^= 1;
    };
    if (!run.stream(pipe, jb, a.status, consume, post)) return false;
    double* out = a.out + static_cast<size_t>(run.split) * 6 * a.stride;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      if (r < a.n)
#pragma unroll
        for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * a.stride + r] = acc[k][c];
    }
  }
  return true;
}

// UNR: unrolled steps; MINB: CTAs per SM asked of the register allocator.
template <int IPT, int W, int UNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
    pair_sym_fp64_kernel(const JBody64* __restrict__ jb, SymArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  TilePipe<JBody64, kSymTile64> pipe;
  pipe.init(reinterpret_cast<JBody64*>(smem_raw), full);
  const SymRun run(a, a.subs * (32 * IPT * W / kSymTile64));
  int half = 0;
  grid_wait();
  if (sym_fp64_rows<IPT, W, UNR>(pipe, reinterpret_cast<double*>(smem_raw + 2 * kSymTile64 * sizeof(JBody64)),
                                 half, jb, run, a))
    grid_release();
}

// ---------------------------------------------------------------------------
// Potential energy (FP64)
// ---------------------------------------------------------------------------
// partial[y * gridDim.x + x]: the CTA's sum over its unordered pairs (i, j) of
// m_i m_j / sqrt(r^2 + eps2) (COMPAT = 0) or, the reference's printed potential,
// m_k^2 / sqrt(.) with k the later of the two (COMPAT = 1).  Only the total is
// wanted, so the pair goes to the row's sum alone and nothing rotates: rows in
// registers, bodies of TJ-body tiles broadcast from shared memory, 12 FP64
// operations per pair (the one-sided form spent them on each ordered pair: N =
// 32768 1.23 ms).  Off its own block a tile lies wholly after or before the
// rows, so COMPAT's later body is the same side for a whole tile.
template <int COMPAT, int IPT, int W, int TJ>
__global__ void __launch_bounds__(32 * W)
    potential_sym_kernel(const JBody64* __restrict__ jb, SymArgs a, double* __restrict__ partial) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  __shared__ double sh[32];
  constexpr int kRows = 32 * IPT * W;
  static_assert(kRows % TJ == 0 && TJ % 32 == 0, "blocks are whole tiles of whole groups");
  TilePipe<JBody64, TJ> pipe;
  pipe.init(reinterpret_cast<JBody64*>(smem_raw), full);
  const SymRun run(a, a.subs * (kRows / TJ));
  const double eps2 = a.eps2;
  double total = 0.0;
  for (int g = 0; g < a.subs; ++g) {
    const int row0 = (run.I * a.subs + g) * kRows + threadIdx.x;  // rows row0 + k * 32 W
    if (row0 - static_cast<int>(threadIdx.x) >= a.n) break;
    double xi[IPT], yi[IPT], zi[IPT], mi[IPT], after[IPT], before[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * W * k;
      double2 p0{0, 0}, p1{0, 0};
      if (r < a.ld) {
        const double2* p = jb64_at(jb, r);
        p0 = p[0];
        p1 = p[32];
      }
      xi[k] = p0.x; yi[k] = p0.y; zi[k] = p1.x; mi[k] = p1.y;
      after[k] = before[k] = 0.0;
    }
    int t = 0;
    auto consume = [&](const JBody64* tile) {
      const int tt = run.tile(t);
      const bool own = run.distance(tt) == 0;
      const int j0 = tt * TJ;
      auto pair = [&](int j, auto&& add) {
        const double2* p = jb64_at(tile, j);
        const double2 p0 = p[0], p1 = p[32];
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
          const double dx = p0.x - xi[k], dy = p0.y - yi[k], dz = p1.x - zi[k];
          add(k, p1.y, rsqrt_f64(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)))));
        }
      };
      if (own) {  // each pair from its later row; padding bodies have no mass
#pragma unroll 2
        for (int j = 0; j < TJ; ++j)
          pair(j, [&](int k, double m, double y) {
            const bool take = j0 + j < row0 + 32 * W * k;
            if (COMPAT) before[k] += take ? y : 0.0;
            else after[k] = fma(take ? m : 0.0, y, after[k]);
          });
      } else if (COMPAT && j0 < run.I * a.subs * kRows) {  // the row is the later body
#pragma unroll 2
        for (int j = 0; j < TJ; ++j)
          pair(j, [&](int k, double, double y) { before[k] += y; });
      } else {
#pragma unroll 2
        for (int j = 0; j < TJ; ++j)
          pair(j, [&](int k, double m, double y) {
            after[k] = fma(COMPAT ? m * m : m, y, after[k]);
          });
      }
    };
    if (!run.stream(pipe, jb, a.status, consume, [&] { ++t; })) return;
#pragma unroll
    for (int k = 0; k < IPT; ++k)
      total += COMPAT ? fma(mi[k] * mi[k], before[k], after[k]) : mi[k] * after[k];
  }
  const double b = block_sum(total, sh);
  if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = b;
}

// ---------------------------------------------------------------------------
// Mixed precision, near/far tile-relative
// ---------------------------------------------------------------------------
// Subtile of 64 bodies.  Header: centre c, radius R >= max |x_j - c|, bounding
// box rounded outward (as JBodyNF's header).  Bodies: lane l holds bodies l and
// l + 32 as packed pairs, so each 64-bit word is an f32x2 operand: chunks
// 0 (-Dx, -Dy), 1 (-Dz, m), 2 (vx, vy), 3 (vz, -), 4 (-Dx_lo, -Dy_lo),
// 5 (-Dz_lo, -), with (D, D_lo) = ds_offset(c, x_hi, x_lo).  50 bytes per body.
// Bodies that are in no order get centre 0 and a box without end: D is then -x
// itself and no subtile is far, so every separation has the accuracy of the
// hi/lo kernels, whatever order the bodies are in and whatever shares a subtile
// (beside an escaper at 1e10, D_lo holds the others' positions as mere floats).
struct __align__(128) SymSub {
  float c[3], R, lo[3], hi[3], pad[22];
  ulonglong2 v[6][32];
};
static_assert(sizeof(SymSub) == 3200, "subtiles start 128-byte aligned");

// Writes one subtile from the values of the calling CTA's first 64 threads' 64
// bodies (invalid ones are zero-mass padding at the centre); called by all.
// ORDERED: neighbours in space share a subtile.
template <bool ORDERED>
__device__ __forceinline__ void write_subtile(SymSub* __restrict__ out, bool valid, const double p[3],
                                              const double u[3], double m) {
  __shared__ SymSub stage;  // written out in one bulk copy
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float c[3] = {0.f, 0.f, 0.f};
  if (ORDERED) {
    __shared__ double box[6][2];
    __shared__ float rmax[2];
#pragma unroll
    for (int k = 0; k < 6; ++k) {  // bounding box in double (empty subtile: +inf/-inf)
      double w = k < 3 ? (valid ? p[k] : INFINITY) : (valid ? p[k - 3] : -INFINITY);
      w = k < 3 ? warp_min(w) : warp_max(w);
      if (lane == 0 && warp < 2) box[k][warp] = w;
    }
    __syncthreads();
    double lo[3], hi[3];
    double r2 = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = fmin(box[k][0], box[k][1]);
      hi[k] = fmax(box[3 + k][0], box[3 + k][1]);
      const double mid = 0.5 * lo[k] + 0.5 * hi[k];
      c[k] = isfinite(mid) ? static_cast<float>(mid) : 0.0f;
      const double d = p[k] - static_cast<double>(c[k]);
      r2 += valid ? d * d : 0.0;
    }
    float R = __double2float_ru(sqrt(r2));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) R = fmaxf(R, __shfl_xor_sync(0xffffffffu, R, o));
    if (lane == 0 && warp < 2) rmax[warp] = R;
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        stage.c[k] = c[k];
        stage.lo[k] = __double2float_rd(lo[k]);
        stage.hi[k] = __double2float_ru(hi[k]);
      }
      stage.R = fmaxf(rmax[0], rmax[1]);
    }
  } else if (tid == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      stage.c[k] = 0.f;
      stage.lo[k] = -INFINITY;
      stage.hi[k] = INFINITY;
    }
    stage.R = 0.f;
  }
  float oh[3], ol[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float h, l, dh = 0.f, dl = 0.f;
    split_hilo(p[k], h, l);
    if (valid) ds_offset(c[k], h, l, dh, dl);
    oh[k] = -dh;
    ol[k] = -dl;
  }
  if (tid < 64) {
    // body tid = half `warp` of lane `lane`'s pairs; word w of chunk q at [128 q + 2 w]
    float* f = reinterpret_cast<float*>(&stage.v[0][lane]) + warp;
    f[0] = oh[0];
    f[2] = oh[1];
    f[128] = oh[2];
    f[130] = __double2float_rn(m);
    f[256] = __double2float_rn(u[0]);
    f[258] = __double2float_rn(u[1]);
    f[384] = __double2float_rn(u[2]);
    f[386] = 0.f;
    f[512] = ol[0];
    f[514] = ol[1];
    f[640] = ol[2];
    f[642] = 0.f;
  }
  if (tid < 22) stage.pad[tid] = 0.f;
  bulk_store_fence();
  __syncthreads();
  if (tid == 0) bulk_store(out, &stage, static_cast<uint32_t>(sizeof stage));
}

// Subtile blockIdx.x of the bodies of `in` (64 threads, one per body).
// PREDICT: `in` is the state X, V (written), with its derivatives D and step
// ctl, and the subtile is that of the predicted state (predict_kernel's
// arithmetic): one pass instead of two.  Bound by its launch below some 10^5
// bodies (104 B read, 48 + 50 written per body): the phase at N = 65536 9.6 us
// instead of 12.6.  Zeroes near_count for the pair pass that follows.
template <bool PREDICT, bool ORDERED>
__global__ void __launch_bounds__(64)
    sym_tile_kernel(int n, SoA7 in, SymSub* __restrict__ out, int ld = 0, double* X = nullptr,
                    double* V = nullptr, const double* __restrict__ D = nullptr,
                    const StepCtl* __restrict__ ctl = nullptr,
                    unsigned long long* near_count = nullptr, double* __restrict__ XP = nullptr) {
  grid_wait();
  grid_release();
  const int slot = blockIdx.x * 64 + threadIdx.x;
  const bool valid = slot < n;
  if (near_count && slot == 0) *near_count = 0;
  double p[3] = {0.0, 0.0, 0.0}, u[3] = {0.0, 0.0, 0.0}, m = 0.0;
  if (valid) {
    m = in.m[slot];
    if (PREDICT) {
      predict_body(ctl->dt, ld, slot, X, V, D, p, u, XP);
    } else {
      p[0] = in.x[slot]; p[1] = in.y[slot]; p[2] = in.z[slot];
      u[0] = in.vx[slot]; u[1] = in.vy[slot]; u[2] = in.vz[slot];
    }
  }
  write_subtile<ORDERED>(out + blockIdx.x, valid, p, u, m);
}

// correct_kernel<8, true> for the near/far records: corrector and the next
// step's predictor on the 64 bodies of subtile blockIdx.x (64 rows times eight
// groups of threads, the sums in correct_kernel<8>'s order), and the subtile.
constexpr int kCorrectTileThreads = 512;
template <bool ORDERED>
static __global__ void __launch_bounds__(kCorrectTileThreads)
    correct_tile_kernel(int n, int ld, RowSlots slots, const double* __restrict__ P,
                        double* __restrict__ X, double* __restrict__ V, double* __restrict__ D,
                        StepCtl* __restrict__ ctl, double eta, const double* __restrict__ M,
                        SymSub* __restrict__ out, unsigned long long* near_count) {
  __shared__ double sh[6 * kCorrectTileThreads];
  const int r = threadIdx.x & 63, g = threadIdx.x >> 6;
  const int i = blockIdx.x * 64 + r;
  const bool mine = i < n && g == 0;
  if (near_count && blockIdx.x == 0 && threadIdx.x == 0) *near_count = 0;
  double crit = __longlong_as_double(static_cast<long long>(kPosInfBits));
  double x[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0}, d[6], m = 0.0;
  if (mine) {
    m = M[i];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      x[c] = X[c * ld + i]; v[c] = V[c * ld + i];
      d[c] = D[c * ld + i]; d[3 + c] = D[(3 + c) * ld + i];
    }
  }
  const int S = i < n ? slots.count(i) : 0;
  double sum[6];
  split_sums(P + static_cast<size_t>(g) * 6 * ld, ld, (S - g + 7) / 8, i, sum, 8);
#pragma unroll
  for (int c = 0; c < 6; ++c) sh[(g * 6 + c) * 64 + r] = sum[c];
  __syncthreads();
  if (mine) {
#pragma unroll
    for (int q = 1; q < 8; ++q)
#pragma unroll
      for (int c = 0; c < 6; ++c) sum[c] += sh[(q * 6 + c) * 64 + r];
    const double dt = ctl->dt;
    crit = correct_body(dt, eta, d, sum, x, v);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      predict_component(dt, x[c], v[c], sum[c], sum[3 + c], x[c], v[c]);
      X[c * ld + i] = x[c];
      V[c * ld + i] = v[c];
      D[c * ld + i] = sum[c];
      D[(3 + c) * ld + i] = sum[3 + c];
    }
  }
  write_subtile<ORDERED>(out + blockIdx.x, mine, x, v, m);
  __syncthreads();  // sh is reused
  finish_criterion(ctl, crit, true, sh);
}

__device__ __forceinline__ uint64_t f2_dup(float v) { return f2_pack(v, v); }

// One i-row (its values in both halves) against two j-bodies, separations
// (dx, dy, dz) given.  MUFU rsqrt and rcp (1/s) as in the one-sided kernels.
template <bool SYM>
__device__ __forceinline__ void sym_pair_x2(uint64_t dx, uint64_t dy, uint64_t dz, uint64_t mj,
                                            uint64_t vxj, uint64_t vyj, uint64_t vzj, uint64_t ui,
                                            uint64_t vi, uint64_t wi, uint64_t mi, uint64_t eps2,
                                            uint64_t m3, uint64_t* ai, uint64_t* bj) {
  const uint64_t du = f2_sub(vxj, ui), dv = f2_sub(vyj, vi), dw = f2_sub(vzj, wi);
  const uint64_t s = f2_fma(dx, dx, f2_fma(dy, dy, f2_fma(dz, dz, eps2)));
  const uint64_t rv = f2_fma(dx, du, f2_fma(dy, dv, f2_mul(dz, dw)));
  float s0, s1;
  f2_unpack(s, s0, s1);
  const uint64_t y = f2_pack(rsqrt_mufu(s0), rsqrt_mufu(s1));
  const uint64_t y2 = f2_pack(rcp_mufu(s0), rcp_mufu(s1));
  const uint64_t y3 = f2_mul(y, y2);
  const uint64_t q = f2_mul(mj, y3), h = SYM ? f2_mul(mi, y3) : 0ull;
  const uint64_t c = f2_mul(rv, f2_mul(y2, m3));
  const uint64_t ex = f2_fma(c, dx, du), ey = f2_fma(c, dy, dv), ez = f2_fma(c, dz, dw);
  ai[0] = f2_fma(q, dx, ai[0]); ai[1] = f2_fma(q, dy, ai[1]); ai[2] = f2_fma(q, dz, ai[2]);
  ai[3] = f2_fma(q, ex, ai[3]); ai[4] = f2_fma(q, ey, ai[4]); ai[5] = f2_fma(q, ez, ai[5]);
  if (SYM) {
    bj[0] = f2_fma(h, dx, bj[0]); bj[1] = f2_fma(h, dy, bj[1]); bj[2] = f2_fma(h, dz, bj[2]);
    bj[3] = f2_fma(h, ex, bj[3]); bj[4] = f2_fma(h, ey, bj[4]); bj[5] = f2_fma(h, ez, bj[5]);
  }
}

// Sums of a lane's j-bodies, handed to the next lane's.
__device__ __forceinline__ void sym_rotate(uint64_t* b, int next) {
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    float l, h;
    f2_unpack(b[c], l, h);
    b[c] = f2_pack(__shfl_sync(0xffffffffu, l, next), __shfl_sync(0xffffffffu, h, next));
  }
}

// Near/far form of a pair (pair.cuh, RowsMixedNF): far subtiles form the
// separation with one add per component, near ones in double-single; a
// (warp, subtile) pair is far when their boxes are apart by at least R / 2.
// Float sums (a row's over one tile of 64 SUB bodies in two halves, a
// j-body's over the warp's 32 IPT rows) are flushed into double: at most 128
// terms per float sum, as in the one-sided kernel, most sums fewer, and smaller
// errors (N = 65536 median / p99 / rms acc error 2.3e-8 / 1.2e-7 / 3.8e-8,
// one-sided 3.0e-8 / 1.6e-7 / 5.0e-8).  Jerk likewise.
//
// Two j-bodies per lane are packed, the i-rows are held in both halves of
// their registers: the packed j-operands and their sums come from shared
// memory and shuffles as they are, and 12 shuffles serve 2 IPT pairs.  At four
// rows per lane a step is 64 cycles of the FP32 pipe against 28 of the shared
// pipe; 168 registers leave three CTAs of four warps per SM (two with more
// registers per thread: 3.0 ms; two rows per lane and four CTAs: 2.9 ms at N
// = 65536).  FP32 pipe 68-72 % active, stalls on the pipe and on fixed
// latencies.  Measured against the one-sided kernel at its tuned tiling: N =
// 65536 2.70 vs 4.00 ms, 262144 41.1 vs 60.8, 16384 0.226 vs 0.300.
// xhl: the rows' (x_hi, x_lo), in shared memory, read once per subtile.
template <int IPT, int W, int SUB>
constexpr size_t sym_nf_smem() {
  return 2 * SUB * sizeof(SymSub) + 6 * IPT * 32 * W * (sizeof(double) + sizeof(float)) +
         2 * SUB * 6 * W * 32 * sizeof(uint64_t);
}

// A CTA's shared memory.
template <int IPT, int W, int SUB>
struct SymNfSmem {
  SymSub* tiles;   // [2][SUB]
  double* acc;     // [6 IPT][NT]
  float* xhl;      // [6 IPT][NT]
  uint64_t* red;   // [2][SUB][6][W][32]
  __device__ __forceinline__ explicit SymNfSmem(unsigned char* raw)
      : tiles(reinterpret_cast<SymSub*>(raw)),
        acc(reinterpret_cast<double*>(raw + 2 * SUB * sizeof(SymSub))),
        xhl(reinterpret_cast<float*>(acc + 6 * IPT * 32 * W)),
        red(reinterpret_cast<uint64_t*>(xhl + 6 * IPT * 32 * W)) {}
};

// One run of a CTA of W warps: SUB subtiles per tile (one barrier each); UNR /
// NUNR: unrolled steps of the far / near loop (two bodies per lane and step).
// `half` is the half of `red` of the current tile, alternating over the CTA's
// life; near_subs counts this warp's near subtiles.  False if a wait timed out.
template <int IPT, int W, int SUB, int UNR, int NUNR>
__device__ __forceinline__ bool sym_nf_rows(TilePipe<SymSub, SUB>& pipe, const SymNfSmem<IPT, W, SUB>& sm,
                                            int& half, int& near_subs, const SymSub* __restrict__ jt,
                                            const SymRun& run, const SymArgs& a) {
  constexpr int NT = 32 * W, kRows = 32 * IPT * W, TJ = 64 * SUB;
  static_assert(kRows % TJ == 0, "blocks are whole tiles");
  double* const acc = sm.acc;
  float* const xhl = sm.xhl;
  uint64_t* const red = sm.red;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, next = (lane + 1) & 31;
  const float e2 = static_cast<float>(a.eps2);
  const uint64_t eps2 = f2_dup(e2), m3 = f2_dup(-3.0f);
  for (int g = 0; g < a.subs; ++g) {
    const int row0 = (run.I * a.subs + g) * kRows + warp * 32 * IPT;
    if ((run.I * a.subs + g) * kRows >= a.n) break;  // a short last block
    uint64_t ui[IPT], vi[IPT], wi[IPT], mi[IPT], fa[IPT][6];
    float blo[3], bhi[3];
    {
      double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int k = 0; k < IPT; ++k) {
        const int r = row0 + 32 * k + lane;
        const bool ok = r < a.n;  // rows >= n: massless copies of the last body, not stored
        const int i = min(r, a.n - 1);
        const double x[3] = {a.rows.x[i], a.rows.y[i], a.rows.z[i]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (ok) { lo[c] = fmin(lo[c], x[c]); hi[c] = fmax(hi[c], x[c]); }
          float h, l;
          split_hilo(x[c], h, l);
          xhl[(k * 6 + c) * NT + tid] = h;
          xhl[(k * 6 + 3 + c) * NT + tid] = l;
        }
        ui[k] = f2_dup(static_cast<float>(a.rows.vx[i]));
        vi[k] = f2_dup(static_cast<float>(a.rows.vy[i]));
        wi[k] = f2_dup(static_cast<float>(a.rows.vz[i]));
        mi[k] = f2_dup(ok ? static_cast<float>(a.rows.m[i]) : 0.f);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          fa[k][c] = 0ull;
          acc[(c * IPT + k) * NT + tid] = 0.0;
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {  // the warp's box, rounded outward
        float l = __double2float_rd(lo[c]), h = __double2float_ru(hi[c]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          l = fminf(l, __shfl_xor_sync(0xffffffffu, l, o));
          h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
        }
        blo[c] = l;
        bhi[c] = h;
      }
    }
    // (D, D_lo)(x_i) relative to the subtile's centre, bit-identical to the records'
    auto offsets = [&](const SymSub* t, int k, uint64_t oh[3], uint64_t ol[3]) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float h, l;
        ds_offset(t->c[c], xhl[(k * 6 + c) * NT + tid], xhl[(k * 6 + 3 + c) * NT + tid], h, l);
        oh[c] = f2_dup(h);
        ol[c] = f2_dup(l);
      }
    };
    auto near_sub = [&](const SymSub* t, auto sym, uint64_t* b) {
      constexpr bool SYM = decltype(sym)::value;
      uint64_t oh[IPT][3], ol[IPT][3];
#pragma unroll
      for (int k = 0; k < IPT; ++k) offsets(t, k, oh[k], ol[k]);
#pragma unroll NUNR
      for (int k = 0; k < 32; ++k) {
        const int j = (lane + k) & 31;
        const ulonglong2 r0 = t->v[0][j], r1 = t->v[1][j], r2 = t->v[2][j], r3 = t->v[3][j];
        const ulonglong2 r4 = t->v[4][j], r5 = t->v[5][j];
#pragma unroll
        for (int r = 0; r < IPT; ++r)
          sym_pair_x2<SYM>(f2_add(f2_add(r0.x, oh[r][0]), f2_add(r4.x, ol[r][0])),
                           f2_add(f2_add(r0.y, oh[r][1]), f2_add(r4.y, ol[r][1])),
                           f2_add(f2_add(r1.x, oh[r][2]), f2_add(r5.x, ol[r][2])), r1.y, r2.x,
                           r2.y, r3.x, ui[r], vi[r], wi[r], mi[r], eps2, m3, fa[r], b);
        if (SYM) sym_rotate(b, next);
      }
    };
    auto far_sub = [&](const SymSub* t, uint64_t* b) {
      uint64_t o[IPT][3];  // D(x_i) to float accuracy: fl(fl(c - x_hi) - x_lo)
#pragma unroll
      for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          o[k][c] = f2_dup(__fsub_rn(__fsub_rn(t->c[c], xhl[(k * 6 + c) * NT + tid]),
                                     xhl[(k * 6 + 3 + c) * NT + tid]));
#pragma unroll UNR
      for (int k = 0; k < 32; ++k) {
        const int j = (lane + k) & 31;
        const ulonglong2 r0 = t->v[0][j], r1 = t->v[1][j], r2 = t->v[2][j], r3 = t->v[3][j];
#pragma unroll
        for (int r = 0; r < IPT; ++r)
          sym_pair_x2<true>(f2_add(r0.x, o[r][0]), f2_add(r0.y, o[r][1]), f2_add(r1.x, o[r][2]),
                            r1.y, r2.x, r2.y, r3.x, ui[r], vi[r], wi[r], mi[r], eps2, m3, fa[r], b);
        sym_rotate(b, next);
      }
    };
    const bool idle = row0 >= a.n;  // a warp of padding rows adds nothing
    int t = 0;
    auto consume = [&](const SymSub* tile) {
      const bool own = run.distance(run.tile(t)) == 0;
      if (idle) {
#pragma unroll
        for (int s = 0; s < SUB; ++s)
#pragma unroll
          for (int c = 0; c < 6; ++c)
            red[(((half * SUB + s) * 6 + c) * W + warp) * 32 + lane] = 0ull;
        return;
      }
#pragma unroll 1
      for (int s = 0; s < SUB; ++s) {
        const SymSub* sub = tile + s;
        // far: boxes apart by d > 0 with d^2 >= R^2 / 4 (gaps rounded down, R up)
        float d2 = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float gap = fmaxf(0.f, fmaxf(__fsub_rd(blo[c], sub->hi[c]), __fsub_rd(sub->lo[c], bhi[c])));
          d2 = __fmaf_rd(gap, gap, d2);
        }
        const bool far = d2 > 0.f && d2 >= __fmul_ru(0.25f, __fmul_ru(sub->R, sub->R));
        uint64_t b[6] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull};
        if (own) {
          ++near_subs;
          near_sub(sub, std::false_type{}, b);
          continue;
        }
        if (far) {
          far_sub(sub, b);
        } else {
          ++near_subs;
          near_sub(sub, std::true_type{}, b);
        }
        uint64_t* o = red + ((half * SUB + s) * 6 * W + warp) * 32 + lane;
#pragma unroll
        for (int c = 0; c < 6; ++c) o[c * W * 32] = b[c];
      }
#pragma unroll
      for (int k = 0; k < IPT; ++k)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          float l, h;
          f2_unpack(fa[k][c], l, h);
          acc[(c * IPT + k) * NT + tid] += static_cast<double>(l + h);
          fa[k][c] = 0ull;
        }
    };
    // after the tile's barrier: the W warps' sums of the tile's bodies, in warp
    // order, into their slot (double from here on)
    auto post = [&]() {
      const int tt = run.tile(t), d = run.distance(tt);
      if (d != 0) {
        double* out = a.out + static_cast<size_t>(a.S + d - 1) * 6 * a.stride +
                      static_cast<size_t>(tt) * TJ;
        for (int e = tid; e < SUB * 6 * 32; e += NT) {
          const int l = e & 31, c = (e >> 5) % 6, s = e / (6 * 32);
          const uint64_t* o = red + ((half * SUB + s) * 6 + c) * W * 32 + l;
          double v0 = 0.0, v1 = 0.0;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            float x, y;
            f2_unpack(o[w * 32], x, y);
            v0 -= static_cast<double>(x);
            v1 -= static_cast<double>(y);
          }
          double* dst = out + static_cast<size_t>(c) * a.stride + s * 64 + l;
          dst[0] = g ? dst[0] + v0 : v0;  // a later sub-block adds to this thread's own store
          dst[32] = g ? dst[32] + v1 : v1;
        }
      }
      ++t;
      half ^= 1;
    };
    if (!run.stream(pipe, jt, a.status, consume, post)) return false;
    double* out = a.out + static_cast<size_t>(run.split) * 6 * a.stride;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      if (r < a.n)
#pragma unroll
        for (int c = 0; c < 6; ++c)
          out[static_cast<size_t>(c) * a.stride + r] = acc[(c * IPT + k) * NT + tid];
    }
  }
  return true;
}

template <int IPT, int W, int SUB, int UNR, int NUNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
    pair_sym_nf_kernel(const SymSub* __restrict__ jt, SymArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  const SymNfSmem<IPT, W, SUB> sm(smem_raw);
  TilePipe<SymSub, SUB> pipe;
  pipe.init(sm.tiles, full);
  const SymRun run(a, a.subs * (32 * IPT * W / (64 * SUB)));
  int half = 0, near_subs = 0;
  grid_wait();
  if (!sym_nf_rows<IPT, W, SUB, UNR, NUNR>(pipe, sm, half, near_subs, jt, run, a)) return;
  grid_release();
  if (a.near_count && (threadIdx.x & 31) == 0 && near_subs)
    atomicAdd(a.near_count, static_cast<unsigned long long>(near_subs));
}

// ---------------------------------------------------------------------------
// Ensembles: one persistent launch over a work list of (cluster, block of 256
// rows, part of its tile run) items; CTAs take items from an atomic counter
// (zeroed before each launch) until the list is exhausted.  Cluster segments
// are padded to whole blocks, so a cluster's records are its own tiles.
// ---------------------------------------------------------------------------
// The item's run; TJ: bodies per tile.
__device__ __forceinline__ SymRun item_run(const EnsItem& it, int TJ) {
  const int block = kEnsRows * it.subs;
  return SymRun(it.row0 / block, it.nb, block / TJ, (it.rows_end + TJ - 1) / TJ, it.t_begin, it.nt, it.split);
}
__device__ __forceinline__ SymArgs item_args(const EnsItem& it, double* P, int* status) {
  SymArgs a{};
  a.n = it.rows_end;
  a.ld = it.ld;
  a.nb = it.nb;
  a.subs = it.subs;
  a.S = it.S;
  a.eps2 = it.eps2;
  a.out = P + it.p_off;
  a.stride = static_cast<size_t>(it.ld);
  a.status = status;
  return a;
}

template <int IPT, int W, int UNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) ensemble_sym_fp64_kernel(
    const JBody64* __restrict__ jb, const EnsItem* __restrict__ items, int n_items, unsigned int* counter,
    double* P, int* status, SoA7) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  __shared__ int s_item;
  static_assert(32 * IPT * W == kEnsRows, "an item's rows are one padding unit");
  TilePipe<JBody64, kSymTile64> pipe;
  pipe.init(reinterpret_cast<JBody64*>(smem_raw), full);
  int half = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = static_cast<int>(atomicAdd(counter, 1u));
    __syncthreads();
    const int k = s_item;
    __syncthreads();
    if (k >= n_items) return;
    const EnsItem it = items[k];
    if (!sym_fp64_rows<IPT, W, UNR>(
            pipe, reinterpret_cast<double*>(smem_raw + 2 * kSymTile64 * sizeof(JBody64)), half,
            jb + it.jrow0, item_run(it, kSymTile64), item_args(it, P, status)))
      return;
  }
}

template <int IPT, int W, int SUB, int UNR, int NUNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB) ensemble_sym_nf_kernel(
    const SymSub* __restrict__ jt, const EnsItem* __restrict__ items, int n_items, unsigned int* counter,
    double* P, int* status, SoA7 rows) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  __shared__ int s_item;
  static_assert(32 * IPT * W == kEnsRows, "an item's rows are one padding unit");
  const SymNfSmem<IPT, W, SUB> sm(smem_raw);
  TilePipe<SymSub, SUB> pipe;
  pipe.init(sm.tiles, full);
  int half = 0, near_subs = 0;
  for (;;) {
    if (threadIdx.x == 0) s_item = static_cast<int>(atomicAdd(counter, 1u));
    __syncthreads();
    const int k = s_item;
    __syncthreads();
    if (k >= n_items) return;
    const EnsItem it = items[k];
    SymArgs a = item_args(it, P, status);
    a.rows = SoA7{rows.x + it.jrow0, rows.y + it.jrow0, rows.z + it.jrow0, rows.m + it.jrow0,
                  rows.vx + it.jrow0, rows.vy + it.jrow0, rows.vz + it.jrow0};
    if (!sym_nf_rows<IPT, W, SUB, UNR, NUNR>(pipe, sm, half, near_subs, jt + it.jrow0 / 64,
                                             item_run(it, 64 * SUB), a))
      return;
  }
}

}  // namespace nbody
