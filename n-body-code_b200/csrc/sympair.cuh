// Symmetric O(N^2) pair kernels: every unordered pair of bodies once.
//
// The one-sided kernels (pair.cuh) evaluate each pair twice, once for either
// body.  Here the pair's separation, 1/sqrt, and tidal vector are formed once
// and added to both bodies (Newton's third law): 38 FP64 operations per pair
// instead of 2 x 31.  The pair kernels are bound by their arithmetic pipe, so
// the fewer operations are the gain.
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
// count is RowSlots::count.
//
// Large systems: a block is `subs` sub-blocks of 32 * IPT * W rows, which the
// CTA works through one after another over the same tiles, adding to the slots
// it wrote itself; this bounds the slots (nb / 2 + S) whatever N is.
#pragma once
#include <cstdint>

#include "hermite.cuh"
#include "pair.cuh"

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
};

__host__ __device__ __forceinline__ int sym_distances(int nb, int I) {
  return (nb & 1) ? (nb - 1) / 2 : (I < nb / 2 ? nb / 2 : nb / 2 - 1);
}

// Tiles of block I's run (its own block first); tb = tiles per whole block,
// only the last block may hold fewer.
__host__ __device__ __forceinline__ int sym_q_count(int nb, int I, int tb, int tiles) {
  const int E = I + sym_distances(nb, I);
  const int whole = (E + 1) * tb;
  return E < nb ? (whole < tiles ? whole : tiles) - I * tb : tiles - I * tb + (E - nb + 1) * tb;
}

// The tile run of one CTA: tiles (first + t) mod tiles, t < nq.
struct SymRun {
  int I, nb, tb, tiles, first, nq;
  __device__ __forceinline__ SymRun(const SymArgs& a, int tb_) : I(blockIdx.x), nb(a.nb), tb(tb_), tiles(a.tiles) {
    const int Q = sym_q_count(nb, I, tb, tiles);
    const int tps = (Q + a.S - 1) / a.S;
    const int q0 = blockIdx.y * tps;
    first = I * tb + q0;
    nq = max(0, min(tps, Q - q0));
  }
  __device__ __forceinline__ int tile(int t) const {  // t-th tile of the run
    const int tt = first + t;
    return tt >= tiles ? tt - tiles : tt;
  }
  __device__ __forceinline__ int distance(int tt) const {
    const int d = tt / tb - I;
    return d < 0 ? d + nb : d;
  }
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
  const double q = p1.y * y3;
  const double c = rv * (-3.0 * y2);
  const double ex = fma(c, dx, du), ey = fma(c, dy, dv), ez = fma(c, dz, dw);
  ai[0] = fma(q, dx, ai[0]); ai[1] = fma(q, dy, ai[1]); ai[2] = fma(q, dz, ai[2]);
  ai[3] = fma(q, ex, ai[3]); ai[4] = fma(q, ey, ai[4]); ai[5] = fma(q, ez, ai[5]);
  if (SYM) {
    const double h = mi * y3;
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

template <int IPT, int W, int UNR, int MINB>
__global__ void __launch_bounds__(32 * W, MINB)
    pair_sym_fp64_kernel(const JBody64* __restrict__ jb, SymArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t full[2];
  constexpr int kRows = 32 * IPT * W;
  TilePipe<JBody64, kSymTile64> pipe;
  pipe.init(reinterpret_cast<JBody64*>(smem_raw), full);
  double* red = reinterpret_cast<double*>(smem_raw + 2 * kSymTile64 * sizeof(JBody64));  // [2][6][W][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, next = (lane + 1) & 31;
  const SymRun run(a, a.subs * (kRows / kSymTile64));
  const double eps2 = a.eps2;
  int half = 0;  // half of `red` of the current tile, alternating over the CTA's life
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
    if (!run.stream(pipe, jb, a.status, consume, post)) return;
    double* out = a.out + static_cast<size_t>(blockIdx.y) * 6 * a.stride;
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const int r = row0 + 32 * k + lane;
      if (r < a.n)
#pragma unroll
        for (int c = 0; c < 6; ++c) out[static_cast<size_t>(c) * a.stride + r] = acc[k][c];
    }
  }
}

}  // namespace nbody
