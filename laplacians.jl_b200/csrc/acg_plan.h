// Sweep plan: how the LDLinv sweeps walk the factor's dependency DAG.
//
// The sweeps are bound by the DAG's depth: a level costs one hand-over of
// values between SMs through L2 (about 1 us) however few vertices it has.  The
// plan merges runs of consecutive levels into blocks.  With C the unit lower
// triangular operator's off-diagonal part, a block B of several levels is
//
//   forward   w_B = r_B + C_{B,before} s_before        s_B = M_B w_B
//   backward  w'_B = g_B s_B + C_{after,B}^T y_after   y_B = M_B^T w'_B
//
// with M_B = (I - C_BB)^{-1}, a sparse matrix formed once in FP64: two
// hand-overs a block instead of one a level.  It is the same linear operator
// (src/approxChol.jl:1347-1408); every coefficient is non-negative, so forming
// M_B cancels nothing.  M_B has more entries than C_BB, so a block grows only
// while the entries (and the longest row) cost less than the levels saved.
//
// w and w' have their own slots behind the n values of the swept vector: a
// vertex v of a block of several levels has slot v + delta (delta one per run
// of consecutive vertices).  Rows come in four kinds, each a sweep task:
//   kRowPlain  out[v] = aux(v) + sum          (a block's first level)
//   kRowWork   out[v + delta] = aux(v) + sum  (the other levels' w or w')
//   kRowFinal  out[v] = sum                   (the same vertices' M_B row)
//   kRowPart   out[v + delta] = sum           (a part of a long row)
// A row's sum runs over entries (slot, coefficient).  A long row would keep one
// warp through many value round trips while its block's other rows are done, so
// the one-vector plan cuts it into parts with slots of their own (behind the
// work slots), whose sums the row adds.
#pragma once
#include <cstdint>
#include <utility>
#include <vector>

namespace acg {

enum SweepRowKind { kRowPlain = 0, kRowWork = 1, kRowFinal = 2, kRowPart = 3 };

// A run of rows of one kind over consecutive vertices [v0, v0 + count).
struct SweepRun {
  int v0, count, kind, delta;
  int row;  // first row in ptr
};

// One direction's rows, in the order the sweep takes them.
struct SweepRows {
  std::vector<SweepRun> runs;
  std::vector<int> ptr, idx;
  std::vector<double> coef;
  std::vector<int> upto;  // per DAG level: runs up to the last one the level needs
};

struct SweepPlan {
  int nslots = 0;  // n + work slots + part slots
  int blocks = 0;
  SweepRows fwd, bwd;
};

// What a level, an entry and a long row cost, in hand-overs.
struct SweepCost {
  double entries_per_hop;  // entries all warps work through in the time of one hand-over
  double row_entries;      // entries of one row walked before it costs another load round trip
  double row_round;        // that round trip
  int split;               // rows longer than this are cut (one more hand-over); 0: none are
  int part;                // entries of a part
  // What the blocks' rows of M_B may hold at most: `fill` times the factor's
  // entries, or fill_min entries where that is more.
  double fill;
  size_t fill_min;
};

// The DAG in internal vertex order (per graph: level by level): in-edges and
// column entries as CSR, and per level the vertex ranges (one per graph).
struct SweepDag {
  int n, nlev;
  const std::vector<std::vector<std::pair<int, int>>>* level_runs;
  const std::vector<int>*fptr, *fidx, *bptr, *bidx;
  const std::vector<double>*fc, *bc;
  int tail_level;  // levels >= tail_level are the dense tail (nlev: none)
};

// Entries that the rows of all M_B together may hold: what `cost` allows, and
// no more than leaves every entry, slot and row number of the plan an int.
size_t sweep_fill_limit(const SweepCost& cost, int n, size_t factor_entries);

// merge = false: every level is a block of its own.
SweepPlan build_sweep_plan(const SweepDag& dag, const SweepCost& cost, bool merge);

}  // namespace acg
