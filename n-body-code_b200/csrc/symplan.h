// The schedule of the symmetric kernels (sympair.cuh): which tiles a block of rows
// meets, which partial-sum slots a row has, and how many blocks and splits a
// system gets.  Plain C++, shared by the kernels and the host.
#pragma once
#include <algorithm>

#ifdef __CUDACC__
#define NB_HD __host__ __device__ __forceinline__
#else
#define NB_HD inline
#endif

namespace nbody {

// Partial-sum slots of a row: S of every row and, where the symmetric pair
// kernels (sympair.cuh) wrote them, one per block at distance 1, 2, ... ahead
// of which the row's block lies.
struct RowSlots {
  int S;           // splits
  int block_rows;  // rows per block of the symmetric schedule
  int nb;          // its blocks; 0: no such slots
  NB_HD RowSlots(int splits, int rows = 1, int blocks = 0)
      : S(splits), block_rows(rows), nb(blocks) {}
  NB_HD int count(int i) const {
    if (nb == 0) return S;
    const int half = nb / 2;  // an even nb's last distance reaches the upper half only
    return S + ((nb & 1) ? half : half - (i / block_rows < half ? 1 : 0));
  }
};

NB_HD int sym_distances(int nb, int I) {
  return (nb & 1) ? (nb - 1) / 2 : (I < nb / 2 ? nb / 2 : nb / 2 - 1);
}

// Tiles of block I's run (its own block first); tb = tiles per whole block,
// only the last block may hold fewer.
NB_HD int sym_q_count(int nb, int I, int tb, int tiles) {
  const int E = I + sym_distances(nb, I);
  const int whole = (E + 1) * tb;
  return E < nb ? (whole < tiles ? whole : tiles) - I * tb : tiles - I * tb + (E - nb + 1) * tb;
}

// The tile run of one CTA: tiles (first + t) mod tiles, t < nq, for the rows of
// block I; its own sums go to slot `split`.
struct SymSpan {
  int I, nb, tb, tiles, first, nq, split;
  NB_HD SymSpan(int I_, int nb_, int tb_, int tiles_, int first_, int nq_, int split_)
      : I(I_), nb(nb_), tb(tb_), tiles(tiles_), first(first_), nq(nq_), split(split_) {}
  // Part `split` of S of the block's run.
  NB_HD SymSpan(int I_, int nb_, int tb_, int tiles_, int S, int split_)
      : I(I_), nb(nb_), tb(tb_), tiles(tiles_), split(split_) {
    const int Q = sym_q_count(nb, I, tb, tiles);
    const int tps = (Q + S - 1) / S;
    const int q0 = split * tps;
    first = I * tb + q0;
    nq = Q - q0 < tps ? Q - q0 : tps;
    if (nq < 0) nq = 0;
  }
  NB_HD int tile(int t) const {  // t-th tile of the run
    const int tt = first + t;
    return tt >= tiles ? tt - tiles : tt;
  }
  NB_HD int distance(int tt) const {
    const int d = tt / tb - I;
    return d < 0 ? d + nb : d;
  }
};

// ---- host side of the schedule --------------------------------------------

// Blocks of a schedule: nb / 2 partial-sum slots, so at most 64 beside the
// splits.  More blocks would need more slots (48 bytes per row each), fewer
// would evaluate more of the pairs one-sided (1 / nb of them).
constexpr int kMaxSymBlocks = 128;
constexpr int kMaxSymSplits = 64;
// Slots are further bounded by memory (8 GiB of P): from 1.4e6 bodies on systems
// take fewer, larger blocks and fewer splits.  At least 32 slots, 1536 bytes per
// body: 32 blocks of 16 splits still fill the SMs, where the 8 that fit at 2e7
// bodies would be 32 CTAs.  Where the slots find no memory, an engine's pass is
// one-sided and an adjoint's schedule is planned with half of them.
inline int max_sym_slots(int n) {
  const double fit = 8.0 * (1 << 30) / (48.0 * n);
  return fit > 2 * kMaxSymSplits ? 2 * kMaxSymSplits : std::max(32, static_cast<int>(fit));
}

// The blocks of n bodies for a kernel whose CTAs hold `rows` rows.
// most_slots: bound on its partial-sum slots.
struct SymGrid {
  int subs, block_rows, nb;
  SymGrid(int rows, int n) : SymGrid(rows, n, max_sym_slots(n)) {}
  SymGrid(int rows, int n, int most_slots) {
    const long most = static_cast<long>(std::min(kMaxSymBlocks, most_slots)) * rows;
    subs = static_cast<int>((n + most - 1) / most);
    block_rows = subs * rows;
    nb = (n + block_rows - 1) / block_rows;
  }
  RowSlots slots(int S) const { return RowSlots(S, block_rows, nb); }
  int count(int S) const { return S + nb / 2; }
};

// Rate at which the corrector sums slots (116 slots at N = 65536: 380 MB with the
// state in 96 us): the price of each partial a tiling leaves.
constexpr double kSplitSumBytesPerMs = 3.9e9;

// Interactions per ms of a GPU full of a pass's CTAs (fitted, see sym_plan).
inline double sym_rate(bool fp64, bool wide) {
  return fp64 ? (wide ? 7.87e8 : 7.44e8) : (wide ? 1.667e9 : 1.505e9);
}
// Smallest system for a kernel.  With one or two tiles a CTA, latency counts,
// which the prediction leaves out: a four-row CTA's tile takes 11.5 us alone on
// its SM, a two-row one's 6 (FP64 N = 1831, a step: 31.3 us against 27.9).
inline int sym_min_bodies(bool wide) { return wide ? 4096 : 0; }
// Time of the last CTAs that leave SMs idle, in units of one CTA's time: the
// near/far kernel's CTAs differ with their near subtiles.
constexpr double kSymTail64 = 0.12, kSymTailNF = 0.2;
constexpr double kSymCtaTiles = 0.2;  // overhead of a CTA in tiles

// One way of splitting the blocks' runs: S CTAs per block, tps tiles each.
struct SymSplit {
  int S, tps;   // tps: of the longest run
  long ctas;    // with tiles
  double mean;  // tiles of one
};
// Calls f for every split into at most max_s CTAs per block that differs from
// the ones into fewer.
template <class F>
inline void for_sym_splits(const SymGrid& g, int tj, int n, int max_s, F&& f) {
  const int tb = g.block_rows / tj, tiles = (n + tj - 1) / tj;
  int Q = 0;
  long total = 0;
  for (int I = 0; I < g.nb; ++I) {
    const int q = sym_q_count(g.nb, I, tb, tiles);
    Q = std::max(Q, q);
    total += q;
  }
  for (int s = 1; s <= max_s; ++s) {
    const int tps = (Q + s - 1) / s;
    if ((Q + tps - 1) / tps != s) continue;
    long ctas = 0;
    for (int I = 0; I < g.nb; ++I) {  // as SymRun
      const int q = sym_q_count(g.nb, I, tb, tiles), own = (q + s - 1) / s;
      ctas += (q + own - 1) / own;
    }
    f(SymSplit{s, tps, ctas, static_cast<double>(total) / ctas});
  }
}

// Splits of a symmetric kernel over n bodies and the predicted time of the
// pass and of the sum over its slots.  rate: interactions per ms; tail: below.
//
// A CTA's time is its tiles and a small overhead.  C CTAs on `slots` places take
// whole waves and one more that lasts by what its fullest SM holds, a tile's
// time being nearly all throughput; CTAs are not equally long, so past the
// first wave up to a third of the work does not keep to waves.  A wave that
// would fill the last place spills (N = 2721, four rows, 296 CTAs of one tile on
// 296 places: 24 us, two waves' time).  Each slot is 48
// bytes per row to sum.  Fitted to the pass's time over every split of both
// kernels at 19 (mixed, 1500 to 262144 bodies) and 13 sizes (FP64, 1024 to
// 100000): 5 % rms; the kernel and split with the least time are on average
// 0.6 % (4 % at most) slower than the measured best of all, at 12 sizes not
// fitted (FP64, 1500 to 10000) 3 %, at worst 26 % (N = 4679, where a step takes
// 60 us, one-sided 84).  Pass and sums in
// us against a fixed line between the kernels at 16384 bodies and a model that
// counted idle CTAs: FP64 N = 3000 25 / 28, 5003 48 / 51, 8192 107 / 122, 12000
// 219 / 234, 65536 5744 / 5794; mixed 5003 33 / 34, 8192 69 / 73, 18001 267 /
// 294, 32768 768 / 802, 65536 2855 / 2874.
struct SymPlan {
  int S;
  double ms;
};
inline SymPlan sym_plan(int sms, int occ, int rows, int tj, int n, double rate, double tail, int most_slots) {
  const SymGrid g(rows, n, most_slots);
  const long slots = static_cast<long>(sms) * occ;
  const double tile_ms = 2.0 * rows * tj * slots / rate;
  SymPlan best{1, 1e300};
  for_sym_splits(g, tj, n, std::min(kMaxSymSplits, std::max(1, most_slots / 2)), [&](const SymSplit& p) {
    const double one = static_cast<double>(p.tps) * g.subs + kSymCtaTiles;
    const double mean = p.mean * g.subs + kSymCtaTiles;
    const long last = (p.ctas + 1) % slots;
    double work = one * ((p.ctas + 1) / slots);
    if (last) work += one * (0.08 + 0.92 * ((last + sms - 1) / sms) / occ);
    if (p.ctas > slots) {
      const double waves = static_cast<double>(p.ctas) / slots;
      work += (mean * waves - work) * (1.0 - 1.0 / waves) / 3.0;
    }
    const double ms = tile_ms * (work + tail * one) + 48.0 * n * g.count(p.S) / kSplitSumBytesPerMs;
    if (ms < best.ms) best = {p.S, ms};
  });
  return best;
}
inline SymPlan sym_plan(int sms, int occ, int rows, int tj, int n, double rate, double tail) {
  return sym_plan(sms, occ, rows, tj, n, rate, tail, max_sym_slots(n));
}

// Splits of the potential kernel, which leaves no slots and keeps 7 to 10 CTAs
// on an SM: the fewest tiles on the fullest SM and, for the last CTAs, two more
// CTAs' time.  In us against sym_plan, which prices slots and waves: N = 8192
// 77 / 88, 16384 169 / 195, 24000 292 / 305; within 4 % of the best split at 12
// sizes from 4097 to 131072.
inline int potential_splits(int sms, int rows, int tj, int n) {
  const SymGrid g(rows, n);
  long best = -1;
  int best_s = 1;
  for_sym_splits(g, tj, n, kMaxSymSplits, [&](const SymSplit& p) {
    const long cost = p.tps * ((p.ctas + sms - 1) / sms + 2);
    if (best < 0 || cost < best) {
      best = cost;
      best_s = p.S;
    }
  });
  return best_s;
}

}  // namespace nbody
