// The symmetric kernels' schedule (csrc/symplan.h) carried out on paper: called
// by test_sym_schedule.py.
#include <cstdio>
#include <cstring>
#include <vector>

#include "symplan.h"

using namespace nbody;

static char g_msg[256];
#define REQUIRE(cond, ...)                      \
  do {                                          \
    if (!(cond)) {                              \
      snprintf(g_msg, sizeof g_msg, __VA_ARGS__); \
      return g_msg;                             \
    }                                           \
  } while (0)

extern "C" {

// Runs every CTA of n bodies on a kernel of `rows` rows and tiles of tj in S
// splits.  Null if each pair of (block, tile) is met once, each (slot, tile) has
// one writer and a row's slots are 0 .. RowSlots::count - 1; else what is wrong.
const char* check_schedule(int rows, int tj, int n, int S) {
  const SymGrid g(rows, n);
  const int nb = g.nb, tb = g.block_rows / tj, tiles = (n + tj - 1) / tj;
  REQUIRE(nb >= 1 && nb <= kMaxSymBlocks, "nb = %d", nb);
  REQUIRE(static_cast<long>(nb) * g.block_rows >= n && static_cast<long>(nb - 1) * g.block_rows < n, "blocks");
  REQUIRE(g.block_rows % tj == 0, "a block is not whole tiles");
  std::vector<unsigned char> met(static_cast<size_t>(nb) * tiles, 0);  // block I met tile t
  std::vector<int> writers(static_cast<size_t>(nb / 2 + 1) * tiles, 0);  // partner slot d - 1, tile
  for (int I = 0; I < nb; ++I) {
    for (int s = 0; s < S; ++s) {
      const SymSpan run(I, nb, tb, tiles, S, s);
      REQUIRE(run.split == s, "split");
      for (int t = 0; t < run.nq; ++t) {
        const int tt = run.tile(t), d = run.distance(tt);
        REQUIRE(tt >= 0 && tt < tiles, "tile %d of %d (block %d, split %d)", tt, tiles, I, s);
        REQUIRE(d >= 0 && d <= nb / 2, "distance %d (block %d, tile %d)", d, I, tt);
        REQUIRE((I + d) % nb == tt / tb, "distance %d of block %d is not tile %d's", d, I, tt);
        REQUIRE(!met[static_cast<size_t>(I) * tiles + tt], "block %d meets tile %d twice", I, tt);
        met[static_cast<size_t>(I) * tiles + tt] = 1;
        if (d) ++writers[static_cast<size_t>(d - 1) * tiles + tt];
      }
    }
  }
  // a block meets all tiles of another or none
  std::vector<int> count(static_cast<size_t>(nb) * nb, 0);
  for (int I = 0; I < nb; ++I)
    for (int tt = 0; tt < tiles; ++tt) count[static_cast<size_t>(I) * nb + tt / tb] += met[static_cast<size_t>(I) * tiles + tt];
  auto size = [&](int J) { return std::min((J + 1) * tb, tiles) - J * tb; };
  for (int I = 0; I < nb; ++I) {
    REQUIRE(count[static_cast<size_t>(I) * nb + I] == size(I), "block %d misses tiles of its own", I);
    for (int J = 0; J < I; ++J) {
      const int ij = count[static_cast<size_t>(I) * nb + J], ji = count[static_cast<size_t>(J) * nb + I];
      REQUIRE((ij == size(J) && ji == 0) || (ij == 0 && ji == size(I)), "blocks %d and %d: %d and %d tiles", I, J, ij, ji);
    }
  }
  const RowSlots slots = g.slots(S);
  for (int tt = 0; tt < tiles; ++tt) {
    int partners = 0;
    for (int d = 1; d <= nb / 2; ++d) {
      const int w = writers[static_cast<size_t>(d - 1) * tiles + tt];
      REQUIRE(w <= 1, "slot of distance %d has %d writers at tile %d", d, w, tt);
      REQUIRE(w == 0 || partners == d - 1, "a slot before distance %d is empty at tile %d", d, tt);
      partners += w;
    }
    for (const int i : {tt * tj, std::min((tt + 1) * tj, n) - 1})
      REQUIRE(slots.count(i) == S + partners, "row %d has %d slots, %d are written", i, slots.count(i), S + partners);
  }
  REQUIRE(g.count(S) >= S + nb / 2, "slots allocated");
  return nullptr;
}

// The planned splits: within their limits, and the CTAs that hold tiles counted
// as the kernels cut the runs.
const char* check_plan(int rows, int tj, int n, int wide, int fp64) {
  const SymGrid g(rows, n);
  const SymPlan p = sym_plan(148, 2, rows, tj, n, sym_rate(fp64, wide), fp64 ? kSymTail64 : kSymTailNF);
  REQUIRE(p.S >= 1 && p.S <= kMaxSymSplits && p.ms > 0 && p.ms < 1e290, "S = %d, %g ms", p.S, p.ms);
  REQUIRE(g.count(p.S) <= max_sym_slots(n), "%d slots of %d", g.count(p.S), max_sym_slots(n));
  const int ps = potential_splits(148, rows, tj, n);
  REQUIRE(ps >= 1 && ps <= kMaxSymSplits, "potential: S = %d", ps);
  const char* bad = nullptr;
  const int tb = g.block_rows / tj, tiles = (n + tj - 1) / tj;
  for_sym_splits(g, tj, n, kMaxSymSplits, [&](const SymSplit& q) {
    long ctas = 0, total = 0;
    for (int I = 0; I < g.nb; ++I)
      for (int s = 0; s < q.S; ++s) {
        const SymSpan run(I, g.nb, tb, tiles, q.S, s);
        ctas += run.nq > 0;
        total += run.nq;
      }
    if (ctas != q.ctas || total != static_cast<long>(q.mean * ctas + 0.5)) bad = "CTAs of a split";
  });
  return bad;
}

int blocks(int rows, int n) { return SymGrid(rows, n).nb; }
int sub_blocks(int rows, int n) { return SymGrid(rows, n).subs; }
int slot_limit(int n) { return max_sym_slots(n); }

}  // extern "C"
