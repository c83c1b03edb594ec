// The sweep plan (csrc/acg_plan.h) for tests on the host: test_sweep_plan.py
// compiles this beside acg_plan.cpp and reads the plan's rows through it.
#include "acg_plan.h"

#include <atomic>
#include <cstdlib>
#include <new>
#include <thread>

namespace {
std::atomic<bool> g_fail{false};      // allocations off the main thread fail
std::thread::id g_main;
struct Handle {
  std::vector<std::vector<std::pair<int, int>>> runs;
  std::vector<int> fptr, fidx, bptr, bidx;
  std::vector<double> fc, bc;
  acg::SweepPlan plan;
};
}  // namespace

void* operator new(size_t n) {
  if (g_fail.load(std::memory_order_relaxed) && std::this_thread::get_id() != g_main) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

// levels: nrun triples (level, first, last + 1); null when the plan cannot be built.
void* pc_build(int n, int nlev, int nrun, const int* levels, const int* fptr, const int* fidx, const double* fc,
               const int* bptr, const int* bidx, const double* bc, int tail, const double* cost, int merge, int fail) {
  auto* h = new Handle;
  h->runs.resize(nlev);
  for (int i = 0; i < nrun; ++i) h->runs[levels[3 * i]].emplace_back(levels[3 * i + 1], levels[3 * i + 2]);
  h->fptr.assign(fptr, fptr + n + 1);
  h->bptr.assign(bptr, bptr + n + 1);
  h->fidx.assign(fidx, fidx + fptr[n]);
  h->fc.assign(fc, fc + fptr[n]);
  h->bidx.assign(bidx, bidx + bptr[n]);
  h->bc.assign(bc, bc + bptr[n]);
  const acg::SweepDag d{n, nlev, &h->runs, &h->fptr, &h->fidx, &h->bptr, &h->bidx, &h->fc, &h->bc, tail};
  acg::SweepCost c{cost[0], cost[1], cost[2], (int)cost[3], (int)cost[4], cost[5], (size_t)cost[6]};
  g_main = std::this_thread::get_id();
  g_fail = fail != 0;
  bool ok = true;
  try {
    h->plan = acg::build_sweep_plan(d, c, merge != 0);
  } catch (const std::bad_alloc&) {
    ok = false;
  }
  g_fail = false;
  if (ok) return h;
  delete h;
  return nullptr;
}

// out: slots, blocks, then per direction runs, rows, entries
void pc_dims(const void* p, long long* out) {
  const auto& plan = static_cast<const Handle*>(p)->plan;
  out[0] = plan.nslots;
  out[1] = plan.blocks;
  int at = 2;
  for (const acg::SweepRows* R : {&plan.fwd, &plan.bwd}) {
    out[at++] = (long long)R->runs.size();
    out[at++] = (long long)R->ptr.size() - 1;
    out[at++] = (long long)R->idx.size();
  }
}

// runs: v0, count, kind, delta, row each
void pc_rows(const void* p, int dir, int* runs, int* ptr, int* idx, double* coef) {
  const auto& plan = static_cast<const Handle*>(p)->plan;
  const acg::SweepRows& R = dir == 0 ? plan.fwd : plan.bwd;
  for (const auto& r : R.runs)
    for (int v : {r.v0, r.count, r.kind, r.delta, r.row}) *runs++ = v;
  for (int v : R.ptr) *ptr++ = v;
  for (int v : R.idx) *idx++ = v;
  for (double v : R.coef) *coef++ = v;
}

// The entries a plan's blocks may hold for a factor of this size.
long long pc_fill_limit(const double* cost, int n, long long entries) {
  const acg::SweepCost c{cost[0], cost[1], cost[2], (int)cost[3], (int)cost[4], cost[5], (size_t)cost[6]};
  return (long long)acg::sweep_fill_limit(c, n, (size_t)entries);
}

void pc_free(void* p) { delete static_cast<Handle*>(p); }

}  // extern "C"
