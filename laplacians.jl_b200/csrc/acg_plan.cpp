#include "acg_plan.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <limits>

#include "acg_threads.h"

namespace acg {
namespace {

constexpr int kMaxBlockLevels = 256;
// a row's own cost in entries: its task record, its right-hand side and store
constexpr double kRowCost = 4.0;

// A block of levels [l0, l1); rows of M_B (its vertices in level order) when it
// has several levels.
struct Block {
  int l0, l1;
  std::vector<int> vert;       // vertices, level by level
  std::vector<int> ptr, idx;   // M_B by row, internal vertex ids ascending
  std::vector<double> val;
};

struct Shared {
  const SweepDag& d;
  const SweepCost* cost;
  std::vector<int> lev, mark;
  std::vector<int> where;  // a vertex's row in the block being grown
  std::vector<double> acc;
  std::vector<double> level_cost;  // rows and entries of a level, both directions averaged
  std::atomic<size_t> held{0};     // entries of the blocks made so far, on all threads
};

// Greedy blocks over the levels [la, lb): from each level on, the length with
// the largest saving in hand-overs.  Gives up once all threads' blocks hold more
// than `limit` entries.
void partition(Shared& s, int la, int lb, size_t limit, std::vector<Block>& out) {
  const SweepDag& d = s.d;
  const auto& runs = *d.level_runs;
  const double A = s.cost->entries_per_hop;
  std::vector<int> cols;
  int stamp_at = -1;
  for (int l = la; l < lb;) {
    Block b;
    b.l0 = l;
    b.ptr.push_back(0);
    double inner = 0.0, all = 0.0, best = 0.0;
    size_t best_verts = 0, first = 0;
    int best_len = 1, longest = 0;
    for (int len = 1; l + len <= lb && len <= kMaxBlockLevels; ++len) {
      const int L = l + len - 1;
      size_t last = 0;
      all += s.level_cost[L];
      // more entries than the block's levels are worth: no gain from here on
      const double most = A * len + all;
      bool over = false;
      for (const auto& r : runs[L]) {
        for (int v = r.first; v < r.second && !over; ++v) {
          ++last;
          stamp_at = v;
          cols.clear();
          cols.push_back(v);
          s.mark[v] = stamp_at;
          s.acc[v] = 1.0;
          for (int k = (*d.fptr)[v + 1] - 1; k >= (*d.fptr)[v]; --k) {
            const int u = (*d.fidx)[k];
            if (s.lev[u] < l) break;  // inputs ascend by level
            const double c = (*d.fc)[k];
            inner += 1.0;
            const int ru = s.where[u];
            for (int e = b.ptr[ru]; e < b.ptr[ru + 1]; ++e) {
              const int w = b.idx[e];
              if (s.mark[w] != stamp_at) {
                s.mark[w] = stamp_at;
                s.acc[w] = 0.0;
                cols.push_back(w);
              }
              s.acc[w] += c * b.val[e];
            }
          }
          std::sort(cols.begin(), cols.end());
          s.where[v] = (int)b.vert.size();
          b.vert.push_back(v);
          for (int w : cols) {
            b.idx.push_back(w);
            b.val.push_back(s.acc[w]);
            s.mark[w] = -1;
          }
          b.ptr.push_back((int)b.idx.size());
          longest = std::max(longest, (int)cols.size());
          over = (double)b.idx.size() > most;
        }
        if (over) break;
      }
      if (over) break;
      if (len == 1) first = last;
      if (len >= 2) {
        const double ends = 0.5 * (double)(first + last);
        const double work = all - inner;
        const double fin = (double)b.idx.size() - ends + kRowCost * ((double)b.vert.size() - ends);
        const double rounds = s.cost->split ? (longest > s.cost->split ? 1.0 : 0.0)
                                            : std::floor((double)(longest - 1) / s.cost->row_entries);
        // a level costs a hand-over and its entries; the block two hand-overs
        const double gain = (len - 2) - (work + fin - all) / A - s.cost->row_round * rounds;
        if (gain > best) {
          best = gain;
          best_len = len;
          best_verts = b.vert.size();
        } else if ((best == 0.0 && len >= 4) || gain < best - std::max(2.0, 0.25 * best)) {
          break;
        }
      }
    }
    b.l1 = l + best_len;
    if (best_len == 1) {
      b.vert.clear();
      b.ptr.clear();
      b.idx.clear();
      b.val.clear();
    } else {
      b.vert.resize(best_verts);
      b.idx.resize(b.ptr[best_verts]);
      b.val.resize(b.ptr[best_verts]);
      b.ptr.resize(best_verts + 1);
      b.idx.shrink_to_fit();
      b.val.shrink_to_fit();
    }
    out.push_back(std::move(b));
    l = out.back().l1;
    const size_t size = out.back().idx.size();
    if (s.held.fetch_add(size, std::memory_order_relaxed) + size > limit) return;
  }
}

// The vertex ranges of levels [l0, l1), one per graph (a graph's vertices are
// numbered level by level, so consecutive levels join up; blocks of several
// levels are made for one graph alone).  Ranges of one level are different
// graphs' and stay apart: next to a graph of one level lies the next graph's
// first, and a group's task tables are cut by graph.
std::vector<std::pair<int, int>> ranges(const SweepDag& d, int l0, int l1) {
  std::vector<std::pair<int, int>> out;
  for (int l = l0; l < l1; ++l)
    for (const auto& r : (*d.level_runs)[l])
      if (r.second > r.first) out.push_back(r);
  std::sort(out.begin(), out.end());
  if (l1 - l0 == 1) return out;
  size_t w = 0;
  for (size_t i = 0; i < out.size(); ++i) {
    if (w && out[w - 1].second == out[i].first)
      out[w - 1].second = out[i].second;
    else
      out[w++] = out[i];
  }
  out.resize(w);
  return out;
}

// What the rows are made from.
struct Layout {
  const SweepDag& d;
  const std::vector<int>& lev;
  const std::vector<Block>& blocks;
  const std::vector<int>& delta;  // of a vertex's work slot (0: it has none)
  int head;                       // levels in blocks; the rest is the dense tail
  int split, part, part_slot;     // rows longer than split are cut; the first part's slot
};

void add_run(SweepRows& R, const std::pair<int, int>& r, int kind, int delta) {
  R.runs.push_back(SweepRun{r.first, r.second - r.first, kind, delta, (int)R.ptr.size() - 1});
}

// The factor's entries [k, e) as a row's, ending it.
void add_row(SweepRows& R, const std::vector<int>& idx, const std::vector<double>& coef, int k, int e) {
  R.idx.insert(R.idx.end(), idx.begin() + k, idx.begin() + e);
  R.coef.insert(R.coef.end(), coef.begin() + k, coef.begin() + e);
  R.ptr.push_back((int)R.idx.size());
}

void reserve_rows(SweepRows& R, const Layout& y, size_t entries) {
  size_t rows = y.d.n;
  for (const Block& b : y.blocks) {
    entries += b.idx.size();
    rows += b.vert.size();
  }
  R.ptr.reserve(rows + 1);
  R.idx.reserve(entries);
  R.coef.reserve(entries);
  R.ptr.push_back(0);
  R.upto.assign(y.d.nlev, 0);
}

// Ends the last run: cuts its rows longer than y.split into parts, a run of
// their own before it, with slots from y.part_slot + parts on.
void end_run(const Layout& y, SweepRows& R, int& parts) {
  SweepRun run = R.runs.back();
  const int k = R.ptr[run.row];
  bool any = false;
  if (y.split)
    for (int q = run.row; q < run.row + run.count && !any; ++q) any = R.ptr[q + 1] - R.ptr[q] > y.split;
  if (!any) return;
  const std::vector<int> ptr(R.ptr.begin() + run.row, R.ptr.end()), idx(R.idx.begin() + k, R.idx.end());
  const std::vector<double> coef(R.coef.begin() + k, R.coef.end());
  R.ptr.resize(run.row + 1);
  R.idx.resize(k);
  R.coef.resize(k);
  R.runs.pop_back();
  const int first = parts;
  for (int q = 0; q < run.count; ++q) {
    if (ptr[q + 1] - ptr[q] <= y.split) continue;
    for (int a = ptr[q]; a < ptr[q + 1]; a += y.part, ++parts)
      add_row(R, idx, coef, a - k, std::min(ptr[q + 1], a + y.part) - k);
  }
  // v0 counts from 0: a part has no vertex
  R.runs.push_back(SweepRun{0, parts - first, kRowPart, y.part_slot + first, run.row});
  run.row = (int)R.ptr.size() - 1;
  R.runs.push_back(run);
  int next = y.part_slot + first;
  for (int q = 0; q < run.count; ++q) {
    if (ptr[q + 1] - ptr[q] <= y.split) {
      add_row(R, idx, coef, ptr[q] - k, ptr[q + 1] - k);
      continue;
    }
    for (int a = ptr[q]; a < ptr[q + 1]; a += y.part) {
      R.idx.push_back(next++);
      R.coef.push_back(1.0);
    }
    R.ptr.push_back((int)R.idx.size());
  }
}

// Blocks upwards, then the dense tail's rows (head inputs only).  Returns the
// number of parts.
int emit_forward(const Layout& y, SweepRows& F) {
  int parts = 0;
  const SweepDag& d = y.d;
  const auto &fptr = *d.fptr, &fidx = *d.fidx;
  const auto& fc = *d.fc;
  std::vector<int> where(d.n);
  reserve_rows(F, y, fidx.size());
  for (const Block& b : y.blocks) {
    const bool multi = b.l1 - b.l0 > 1;
    for (const auto& r : ranges(d, b.l0, b.l0 + 1)) {
      add_run(F, r, kRowPlain, multi ? y.delta[r.first] : 0);
      for (int v = r.first; v < r.second; ++v) add_row(F, fidx, fc, fptr[v], fptr[v + 1]);
      end_run(y, F, parts);
    }
    F.upto[b.l0] = (int)F.runs.size();
    if (!multi) continue;
    const auto rest = ranges(d, b.l0 + 1, b.l1);
    for (const auto& r : rest) {
      add_run(F, r, kRowWork, y.delta[r.first]);
      for (int v = r.first; v < r.second; ++v) {  // the inputs before the block, which come first
        int e = fptr[v];
        while (e < fptr[v + 1] && y.lev[fidx[e]] < b.l0) ++e;
        add_row(F, fidx, fc, fptr[v], e);
      }
      end_run(y, F, parts);
    }
    for (size_t i = 0; i < b.vert.size(); ++i) where[b.vert[i]] = (int)i;
    for (const auto& r : rest) {
      add_run(F, r, kRowFinal, y.delta[r.first]);
      for (int v = r.first; v < r.second; ++v) {
        const int row = where[v];
        for (int e = b.ptr[row]; e < b.ptr[row + 1]; ++e) {
          const int u = b.idx[e];
          F.idx.push_back(y.lev[u] == b.l0 ? u : u + y.delta[u]);
          F.coef.push_back(b.val[e]);
        }
        F.ptr.push_back((int)F.idx.size());
      }
      end_run(y, F, parts);
    }
    for (int l = b.l0 + 1; l < b.l1; ++l) F.upto[l] = (int)F.runs.size();
  }
  if (y.head < d.nlev) {
    for (const auto& r : ranges(d, y.head, d.nlev)) {
      add_run(F, r, kRowPlain, 0);
      for (int v = r.first; v < r.second; ++v) add_row(F, fidx, fc, fptr[v], fptr[v + 1]);
      end_run(y, F, parts);
    }
    for (int l = y.head; l < d.nlev; ++l) F.upto[l] = (int)F.runs.size();
  }
  return parts;
}

// Blocks downwards; a block's last level is its first step.
int emit_backward(const Layout& y, SweepRows& B) {
  int parts = 0;
  const SweepDag& d = y.d;
  const auto &bptr = *d.bptr, &bidx = *d.bidx;
  const auto& bc = *d.bc;
  std::vector<int> where(d.n), tptr, tidx, pos;
  std::vector<double> tval;
  reserve_rows(B, y, bidx.size());
  for (auto it = y.blocks.rbegin(); it != y.blocks.rend(); ++it) {
    const Block& b = *it;
    const int top = b.l1 - 1;
    const bool multi = top > b.l0;
    for (const auto& r : ranges(d, top, b.l1)) {
      add_run(B, r, kRowPlain, multi ? y.delta[r.first] : 0);
      for (int v = r.first; v < r.second; ++v) add_row(B, bidx, bc, bptr[v], bptr[v + 1]);
      end_run(y, B, parts);
    }
    B.upto[top] = (int)B.runs.size();
    if (!multi) continue;
    const auto rest = ranges(d, b.l0, top);
    for (const auto& r : rest) {
      add_run(B, r, kRowWork, y.delta[r.first]);
      for (int v = r.first; v < r.second; ++v) {  // the targets after the block, which come first
        int e = bptr[v];
        while (e < bptr[v + 1] && y.lev[bidx[e]] >= b.l1) ++e;
        add_row(B, bidx, bc, bptr[v], e);
      }
      end_run(y, B, parts);
    }
    // columns of M_B, targets descending (as the plain entries)
    const int m = (int)b.vert.size();
    for (int i = 0; i < m; ++i) where[b.vert[i]] = i;
    tptr.assign(m + 1, 0);
    for (int u : b.idx) tptr[where[u] + 1]++;
    for (int i = 0; i < m; ++i) tptr[i + 1] += tptr[i];
    tidx.resize(b.idx.size());
    tval.resize(b.idx.size());
    pos.assign(tptr.begin(), tptr.end() - 1);
    for (int i = m - 1; i >= 0; --i)
      for (int e = b.ptr[i]; e < b.ptr[i + 1]; ++e) {
        const int c = where[b.idx[e]];
        tidx[pos[c]] = b.vert[i];
        tval[pos[c]] = b.val[e];
        ++pos[c];
      }
    for (const auto& r : rest) {
      add_run(B, r, kRowFinal, y.delta[r.first]);
      for (int v = r.first; v < r.second; ++v) {
        const int c = where[v];
        for (int e = tptr[c]; e < tptr[c + 1]; ++e) {
          const int u = tidx[e];
          B.idx.push_back(y.lev[u] == top ? u : u + y.delta[u]);
          B.coef.push_back(tval[e]);
        }
        B.ptr.push_back((int)B.idx.size());
      }
      end_run(y, B, parts);
    }
    for (int l = b.l0; l < top; ++l) B.upto[l] = (int)B.runs.size();
  }
  return parts;
}

}  // namespace

size_t sweep_fill_limit(const SweepCost& cost, int n, size_t factor_entries) {
  // A direction has at most E = factor + M_B entries, and rows of more than
  // `split` entries add E / part + E / split parts, each an entry and a slot.
  const size_t most = std::numeric_limits<int>::max();
  const size_t per = cost.split ? (size_t)std::min(cost.part, cost.split) / 2 : most;
  const size_t entries = most - most / (per + 1);  // E + E / per <= most
  if (factor_entries >= entries || 2 * (size_t)n + entries / per > most) return 0;
  const size_t want = std::max((size_t)(cost.fill * (double)factor_entries), cost.fill_min);
  return std::min(want, entries - factor_entries);
}

SweepPlan build_sweep_plan(const SweepDag& d, const SweepCost& cost, bool merge) {
  Shared s{d, &cost, std::vector<int>(d.n, 0), std::vector<int>(d.n, -1), std::vector<int>(d.n, 0),
           std::vector<double>(d.n, 0.0), std::vector<double>(d.nlev, 0.0), {}};
  const auto& runs = *d.level_runs;
  const int head = std::min(d.tail_level, d.nlev);
  for (int l = 0; l < d.nlev; ++l)
    for (const auto& r : runs[l]) {
      for (int v = r.first; v < r.second; ++v) s.lev[v] = l;
      const double in = (*d.fptr)[r.second] - (*d.fptr)[r.first], outs = (*d.bptr)[r.second] - (*d.bptr)[r.first];
      s.level_cost[l] += 0.5 * (in + outs) + kRowCost * (r.second - r.first);
    }
  // Blocks: stretches of levels of about equal cost are partitioned by their
  // own thread (the stretches depend on the graph alone).
  std::vector<Block> blocks;
  // A DAG that fills in fast is merged less: while the blocks hold more than the
  // limit, they are cut again with dearer entries.  (Whether they do depends on
  // the graph alone: the threads' total only grows.)
  const size_t limit = sweep_fill_limit(cost, d.n, std::max(d.fidx->size(), d.bidx->size()));
  if (limit == 0) merge = false;
  SweepCost c = cost;
  s.cost = &c;
  for (int round = 0; merge; ++round, c.entries_per_hop *= 0.25) {
    blocks.clear();
    s.held = 0;
    std::fill(s.mark.begin(), s.mark.end(), -1);
    double total = 0.0;
    for (int l = 0; l < head; ++l) total += s.level_cost[l];
    const int stretches = std::max(1, std::min(8, (int)(total / 1e6)));
    std::vector<int> cut{0};
    double sum = 0.0;
    for (int l = 0; l < head; ++l) {
      sum += s.level_cost[l];
      if ((int)cut.size() < stretches && sum >= total * (double)cut.size() / stretches) cut.push_back(l + 1);
    }
    cut.push_back(head);
    std::vector<std::vector<Block>> parts(cut.size() - 1);
    run_threads((int)parts.size(), [&](int i) { partition(s, cut[i], cut[i + 1], limit, parts[i]); });
    if (s.held <= limit) {
      for (auto& p : parts)
        for (auto& b : p) blocks.push_back(std::move(b));
      break;
    }
    if (round == 7) merge = false;
  }
  if (!merge) {
    blocks.clear();
    for (int l = 0; l < head; ++l) blocks.push_back(Block{l, l + 1, {}, {}, {}, {}});
  }
  SweepPlan plan;
  plan.blocks = (int)blocks.size();
  plan.nslots = d.n;

  // slots of the blocks' work values
  std::vector<int> delta(d.n, 0);
  for (const Block& b : blocks) {
    if (b.l1 - b.l0 < 2) continue;
    for (const auto& r : ranges(d, b.l0, b.l1)) {
      for (int v = r.first; v < r.second; ++v) delta[v] = plan.nslots - r.first;
      plan.nslots += r.second - r.first;
    }
  }
  // The directions share no state but the layout; s and y are vectors of their
  // own, so the same slots serve the parts of both.
  const Layout lay{d, s.lev, blocks, delta, head, merge ? cost.split : 0, cost.part, plan.nslots};
  int parts[2] = {0, 0};
  run_threads(2, [&](int i) { parts[i] = i == 0 ? emit_forward(lay, plan.fwd) : emit_backward(lay, plan.bwd); });
  plan.nslots += std::max(parts[0], parts[1]);
  return plan;
}

}  // namespace acg
