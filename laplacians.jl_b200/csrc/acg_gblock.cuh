// Groups of small graphs: one block runs one graph's whole PCG.
//
// In the group's launch-per-kernel form (acg_group.cuh) every graph shares every
// launch, and the sweeps of the union cost a hand-over between SMs per level of
// the deepest graph.  A small graph needs neither: its block walks the levels
// with block barriers, the swept vector (s, y and z in turn) and, where it fits,
// p in shared memory, and no graph waits for another.  A block is bound by its
// SM's instruction rate (a task is about 200 instructions a warp), so this is for
// graphs of up to some 10,000 vertices; the solver's cost rule decides.  Blocks
// are independent, so the launch may hold more graphs than SMs, largest first.
//
// The arithmetic is the launch-per-kernel form's to the bit: rows are summed by
// the same lanes in the same order (the same task tables, cut per graph), and
// every dot product by the same tree (chunks of kChunk elements on 256 threads,
// warps, then chunks in order).  Some graphs' PCG amplify a change of rounding
// beyond 1e-9 of x at tol 1e-8, so it may not change.
#pragma once
#include "acg_group.cuh"

namespace acg {

constexpr int kGBThreads = 1024;
constexpr int kGBSub = kGBThreads / kVecThreads;  // chunks in flight
constexpr int kGBMaxChunks = 64;                  // at most 131,072 vertices
constexpr int kGBWarps = kVecThreads / 32;        // warps of a chunk
constexpr int kGBWarpsAll = kGBThreads / 32;

struct GBGraph {
  int v0, n;              // vertices [v0, v0 + n)
  int nlev;
  int wf, wb;             // first of the kGBWarpsAll + 1 offsets of its warps' tasks
  int seg;
};

template <typename T>
struct GBArgs {
  const GBGraph* graphs;  // largest first
  const int *lp, *li;
  const T* lv;
  const SweepTask *tf, *tb;  // per graph and warp, in walking order; delta = the step it is taken in
  const int *of, *ob;        // task offsets per warp
  const int *fi, *bi;
  const T *fc, *bc, *g;
  T *r, *p, *q, *x3, *y;  // y: the swept vector of graphs too large for shared memory
  int nall;               // vertices of all graphs (x buffers)
  PcgState* st;
  double eps;
  int init;               // as pcg_scalar_zdot
  int smem_values;        // values the dynamic shared memory holds
};

// NV sums over the graph's vertices as seg_reduce forms them: ld(i) reads what
// vertex i needs, use(i, values, acc) adds to the sums (and may write).  The
// totals are in out[0..NV) (shared) after the block barrier it ends with.
template <int NV, typename L, typename F>
__device__ __forceinline__ void gb_reduce(int n, double* part, double* out, L&& ld, F&& use) {
  constexpr int U = 4;  // vertices whose loads are issued together
  const int t = threadIdx.x & (kVecThreads - 1), sub = threadIdx.x / kVecThreads;
  const int lane = threadIdx.x & 31, w = t >> 5;
  const int nch = (n + kChunk - 1) / kChunk;
  for (int c = sub; c < nch; c += kGBSub) {
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    const int end = min(n, (c + 1) * kChunk);
    for (int i0 = c * kChunk + t; i0 < end; i0 += U * kVecThreads) {
      decltype(ld(0)) val[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * kVecThreads < end) val[u] = ld(i0 + u * kVecThreads);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * kVecThreads < end) use(i0 + u * kVecThreads, val[u], acc);
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], o);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) part[(c * NV + k) * kGBWarps + w] = acc[k];
  }
  __syncthreads();
  // the tree of block_reduce's second step, then the chunks in order
  for (int e = threadIdx.x; e < nch * NV; e += kGBThreads) {
    double* v = part + e * kGBWarps;
    v[0] = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
    for (int c = 0; c < nch; ++c) s += part[(c * NV + threadIdx.x) * kGBWarps];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

// One sweep of the graph, step by step (forward: levels upwards, backward:
// downwards); v holds the swept vector (graph-local indices).  Forward: v[i] =
// r + sum; backward: v[i] = g v[i] + sum in place (a vertex's s is read by its
// own row alone).  A warp's tasks lie one after another, each with the step it
// belongs to; records are loaded two tasks ahead and entries one task ahead,
// across the barriers.
template <typename T, bool kForward>
__device__ __forceinline__ void gb_sweep(const GBArgs<T>& P, const GBGraph& G, T* v) {
  constexpr int U = 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SweepTask* tasks = kForward ? P.tf : P.tb;
  const int* off = kForward ? P.of + G.wf : P.ob + G.wb;
  const int* idx = kForward ? P.fi : P.bi;
  const T* coef = kForward ? P.fc : P.bc;
  const T* aux = kForward ? P.r : P.g;
  int t = __ldg(&off[warp]);
  const int end = __ldg(&off[warp + 1]);
  auto record = [&](int x) {
    SweepTask rec = load_task(tasks, x, end);
    if (x >= end) rec.delta = INT_MAX;
    return rec;
  };
  auto entries = [&](SweepEntries<T, U>& e, const SweepTask& rec) {
    load_entries<T, true, false, U>(e, rec, lane, idx, coef, coef, coef);
    e.a = e.active(lane) && (lane & (e.gw() - 1)) == 0 ? (kForward ? aux[e.v] : __ldg(&aux[e.v])) : T(0);
  };
  SweepEntries<T, U> e0;
  entries(e0, record(t));
  SweepTask r1 = record(t + 1);
  for (int l = 0; l < G.nlev; ++l) {
    while (e0.delta == l) {
      const SweepTask r2 = record(t + 2);
      SweepEntries<T, U> e1;
      entries(e1, r1);
      const int gw = e0.gw();
      T acc = T(0);
#pragma unroll
      for (int j = 0; j < U; ++j)
        if (e0.id[j] >= 0) acc += e0.c[j] * v[e0.id[j] - G.v0];
      for (int k = e0.k0 + U * gw; k < e0.k1; k += 4 * gw) {
        int id[4];
        T c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int kk = k + j * gw;
          id[j] = kk < e0.k1 ? __ldg(&idx[kk]) : -1;
          c[j] = kk < e0.k1 ? __ldg(&coef[kk]) : T(0);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (id[j] >= 0) acc += c[j] * v[id[j] - G.v0];
      }
      __syncwarp();
      acc = group_sum_w(acc, gw);
      if (e0.active(lane) && (lane & (gw - 1)) == 0) {
        const int i = e0.v - G.v0;
        v[i] = kForward ? e0.a + acc : e0.a * v[i] + acc;
      }
      e0 = e1;
      r1 = r2;
      ++t;
    }
    __syncthreads();
  }
}

template <typename T>
struct GB2 {
  T a, b;
};
template <typename T>
struct GB4 {
  T a, b, c, d;
};

template <typename T>
__global__ void __launch_bounds__(kGBThreads, 1) k_group_pcg(const __grid_constant__ GBArgs<T> P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double part[kGBMaxChunks * 3 * kGBWarps];
  __shared__ double tot[3];
  __shared__ PcgState ls;
  const GBGraph G = P.graphs[blockIdx.x];
  const int tid = threadIdx.x, n = G.n;
  if (tid == 0) ls = P.st[G.seg];
  __syncthreads();
  if (ls.done) return;
  T* sm = reinterpret_cast<T*>(smem_raw);
  const bool vin = n <= P.smem_values, pin = 2 * n <= P.smem_values;
  T* v = vin ? sm : P.y + G.v0;
  T* p = pin ? sm + n : P.p + G.v0;
  T *r = P.r + G.v0, *q = P.q + G.v0;
  T* x3 = P.x3 + G.v0;
  const size_t xs = P.nall;
  // the preconditioner and what follows it; init: the pre-loop step
  auto step = [&](int init) -> bool {
    gb_sweep<T, true>(P, G, v);
    gb_sweep<T, false>(P, G, v);
    gb_reduce<1>(n, part, tot, [&](int i) { return v[i]; }, [&](int, T y, double (&a)[1]) { a[0] += (double)y; });
    const double mu = tot[0] / (double)ls.nvert;
    __syncthreads();
    gb_reduce<2>(n, part, tot, [&](int i) { return GB2<T>{v[i], r[i]}; }, [&](int i, const GB2<T>& w, double (&a)[2]) {
      const T z = (T)((double)w.a - mu);
      v[i] = z;
      if (init) p[i] = z;
      a[0] += (double)z * (double)w.b;
      a[1] += fabs((double)z);
    });
    if (tid == 0) {
      ls.mean = mu;
      pcg_scalar_zdot(&ls, tot[0], tot[1], P.eps, init);
    }
    __syncthreads();
    return ls.done != 0;
  };
  bool stop = step(P.init);
  while (!stop) {
    // q = L p, rows as kg_spmv: 8 lanes a row, entries in turn; two rows of a
    // lane's at once, the next two's extents on their way
    {
      constexpr int S = kGBThreads / 8;
      const int gl = tid & 7;
      int row = tid >> 3, e0[2], e1[2];
      auto extent = [&](int first) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = first + h * S;
          e0[h] = i < n ? __ldg(&P.lp[G.v0 + i]) + gl : 0;
          e1[h] = i < n ? __ldg(&P.lp[G.v0 + i + 1]) : 0;
        }
      };
      extent(row);
      for (int base = (tid & ~31) >> 3; base < n; base += 2 * S, row += 2 * S) {
        const int ka[2] = {e0[0], e0[1]}, kb[2] = {e1[0], e1[1]};
        extent(row + 2 * S);
        T acc[2] = {T(0), T(0)};
        for (int k = 0; ka[0] + k < kb[0] || ka[1] + k < kb[1]; k += 16) {
          int id[2][2];
          T c[2][2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int kk = ka[h] + k + 8 * j;
              id[h][j] = kk < kb[h] ? __ldg(&P.li[kk]) : -1;
              c[h][j] = kk < kb[h] ? __ldg(&P.lv[kk]) : T(0);
            }
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (id[h][j] >= 0) acc[h] += c[h][j] * p[id[h][j] - G.v0];
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          acc[h] = group_sum<8>(acc[h]);
          if (row + h * S < n && gl == 0) q[row + h * S] = acc[h];
        }
      }
    }
    __syncthreads();
    gb_reduce<3>(n, part, tot, [&](int i) { return GB2<T>{p[i], q[i]}; }, [&](int, const GB2<T>& w, double (&a)[3]) {
      const double pv = (double)w.a, qv = (double)w.b;
      a[0] += pv * qv;
      a[1] += fabs(pv);
      a[2] += fabs(qv);
    });
    if (tid == 0) pcg_scalar_pq(&ls, tot[0], tot[1], tot[2], P.eps);
    __syncthreads();
    if (ls.done) break;
    {
      const double al = ls.alpha;
      const T* xc = x3 + (size_t)ls.xcur * xs;
      T* xn = x3 + (size_t)ls.xnext * xs;
      gb_reduce<3>(n, part, tot, [&](int i) { return GB4<T>{xc[i], p[i], r[i], q[i]}; },
                   [&](int i, const GB4<T>& w, double (&a)[3]) {
        const T xv = (T)((double)w.a + al * (double)w.b);
        const T rv = (T)((double)w.c + (-al) * (double)w.d);
        xn[i] = xv;
        r[i] = rv;
        a[0] += (double)rv * (double)rv;
        a[1] += fabs((double)xv);
        a[2] += fabs((double)rv);
      });
    }
    if (tid == 0) pcg_scalar_update(&ls, tot[0], tot[1], tot[2]);
    __syncthreads();
    if (ls.done) break;
    stop = step(0);
    if (stop) break;
    const double beta = ls.beta;
    for (int i = tid; i < n; i += kGBThreads) p[i] = (T)((double)v[i] + beta * (double)p[i]);
    __syncthreads();
  }
  if (tid == 0) P.st[G.seg] = ls;
}

}  // namespace acg
