// One-vector PCG as one persistent kernel (src/pcg.jl:256-445).
//
// A solve of one right-hand side is a chain of short dependent steps: as
// separate launches an iteration of a small graph is a dozen kernel launches
// and their drains, 50 us and more where the arithmetic is 1 us.  Here a
// cooperative grid stays on the GPU for the whole PCG and an iteration is
//
//   update    x' = x + alpha p, r' = r - alpha q, |r'|^2, ...       -> reduce
//   forward   the sweep plan's forward tasks (values are their own ready flags)
//   tail      y_T = W w_T, W = M^T diag(g_T) M up to a constant per column: the
//             dense tail's two triangular products as one matrix (k_form_w)
//   backward  the backward tasks; also sum y and y.r                -> reduce
//   p         p' = (y - mean) + beta p                              -> reduce
//   mat-vec   q = L p', p'.q                                        -> reduce
//
// Reductions.  Each block publishes its partial sums, each a slot that starts
// pending; block 0 polls the slots, adds them in block order and publishes the
// totals in one line that every block polls, so all blocks hold the same sums
// and take the same decisions.  (Every block polling every slot was three times
// slower: hundreds of blocks reading the same few lines.)  Publishing is a
// release (fence, then the slots), collecting an acquire (slots, then fence), so
// a reduction is also a grid barrier for the vectors written before it.  A block
// resets its slots once it has the totals; block 0 resets the totals of one
// reduction when every block has published the next, before the fence with which
// it publishes that one's totals.  So a block that has the totals of one
// reduction finds those of the reduction before it pending or new, never old:
// with two reductions an iteration (kWhole) these are the next that it polls.
//
// While it runs, a grid of two blocks per SM leaves next to no registers to other
// streams, so a launch leaves after slice_s seconds, at the end of an iteration,
// and a WHILE node launches the next, which goes on where it left (the vectors,
// the scalars and the reduction slots are in device memory): work that waits gets
// the SMs in between.  A 2048^3 matrix product (0.4 ms alone) beside solves of
// 216,000 vertices (12 ms) took 0.5 ms between the launches of a kernel per step,
// 12 ms beside one launch, and takes 1.5 ms beside launches of a millisecond;
// these cost a solve alone 0.4 to 1 % (grid3(100) 28.07 -> 28.20 ms).
//
// Graphs of up to kDenseWhole vertices have W for the whole graph (k_pcg's
// kWhole): no sweeps and two reductions an iteration.
//
// Every wait is bounded (spin_limit) and raises PcgState::sweep_error; a block
// that sees the flag stops waiting, and all blocks leave.
#pragma once
#include "acg_pcg.cuh"

namespace acg {

constexpr int kDenseWhole = 2048;  // graphs up to this size: W is the whole preconditioner
constexpr int kPersistThreads = 256;
constexpr int kRedPoints = 4;      // reductions of an iteration at most
constexpr int kRedValues = 8;      // values of a reduction at most (one warp of a block each)
constexpr int kWPad = 64;          // W's rows are padded to this many columns

__host__ __device__ constexpr int w_stride(int K) { return (K + kWPad - 1) / kWPad * kWPad; }

// Slots of the reductions: the totals, then each block's partial sums.
__host__ __device__ constexpr int persist_slots(int blocks) { return kRedPoints * kRedValues * (blocks + 1); }

template <typename T>
struct PersistArgs {
  int n, nslots, vs, vl;               // vertices, sweep slots; slot stride of s and y; lanes per mat-vec row
  const int *lp, *li;                  // Laplacian CSR
  const T* lv;
  int ntf, ntb;                        // forward / backward tasks
  const SweepTask *tf, *tb;
  const int *fi, *bi;
  const T *fc, *bc, *g;
  int K, v0;                           // dense tail: vertices [v0, v0 + K)
  const T* W;
  T *r0, *r1, *p0, *p1, *q, *x3, *s, *y;  // r1, p1: the second buffers of kWhole
  T* wt;                               // w_T, packed (pending between iterations)
  double* red;                         // reduction slots (pending at launch)
  PcgState* st;
  double eps;
  int init;                            // as pcg_scalar_zdot: 1 starts the maxtime clock here
  int poll_mode;
  unsigned spin_limit;                 // polls of a sweep value
  unsigned red_limit;                  // polls of a reduction slot
  double slice_s;                      // seconds after which a launch leaves
};

__device__ __forceinline__ bool gave_up(const PcgState* st) { return *((volatile const int*)&st->sweep_error) != 0; }

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ double* red_slot(double* red, int point, int value) {
  return red + kRedPoints * kRedValues + ((size_t)point * kRedValues + value) * gridDim.x;
}

// Publishes the sums of v over the block at reduction `point`.  The block
// barrier inside orders every thread's earlier writes before thread 0's fence.
template <int NV>
__device__ __forceinline__ void red_publish(double* red, int point, double (&v)[NV], double* smem) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr int NW = kPersistThreads / 32;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) smem[k * NW + wid] = v[k];
  __syncthreads();
  if (wid == 0) {
    static_assert(NW == 8 && kRedValues <= 8, "one lane a value, eight warps");
    double t = 0.0;
    if (lane < NV)
#pragma unroll
      for (int w = 0; w < NW; ++w) t += smem[lane * NW + w];
    fence_gpu();
    if (lane < NV) st_relaxed(red_slot(red, point, lane) + blockIdx.x, t);
  }
}

// Collects reduction `point` into smem[0..NV), the same in every block; `last` is
// the reduction before it.  Ends with a block barrier.
template <int NV>
__device__ __forceinline__ void red_collect(double* red, int point, int last, double* smem, PcgState* st,
                                            unsigned spin_limit) {
  constexpr int U = 5;
  const int G = gridDim.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (blockIdx.x == 0) {
    __syncthreads();  // smem of the publish is free
    if (wid < NV) {   // warp k adds value k
      const double* base = red_slot(red, point, wid);
      double sum = 0.0;
      unsigned spins = 0;
      for (int i0 = lane; i0 < G; i0 += 32 * U) {
        double t[U];
        unsigned pend = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          t[u] = 0.0;
          if (i0 + 32 * u < G) pend |= 1u << u;
        }
        while (pend) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if ((pend >> u) & 1u) t[u] = ld_relaxed(base + i0 + 32 * u);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (((pend >> u) & 1u) && !is_pending(t[u])) pend &= ~(1u << u);
          if (pend && (((++spins & 255u) == 0 && gave_up(st)) || spins >= spin_limit)) {
            atomicExch(&st->sweep_error, 1);
#pragma unroll
            for (int u = 0; u < U; ++u)
              if ((pend >> u) & 1u) t[u] = 0.0;
            break;
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) sum += t[u];
      }
      __syncwarp();
      fence_gpu();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) smem[wid] = sum;
    }
    __syncthreads();
    // every block has published `point`, so has the totals of `last`
    if (wid == 0) {
      if (lane < kRedValues) st_relaxed(red + last * kRedValues + lane, pending_value<double>());
      __syncwarp();
      fence_gpu();  // the reset before the totals, for every lane's slot
      if (lane < NV) st_relaxed(red + point * kRedValues + lane, smem[lane]);
    }
  } else {
    __syncthreads();
    if (wid == 0) {
      double t = 0.0;
      if (lane < NV) {
        const double* src = red + point * kRedValues + lane;
        unsigned spins = 0;
        t = ld_relaxed(src);
        while (is_pending(t)) {
          if (((++spins & 255u) == 0 && gave_up(st)) || spins >= spin_limit) {
            atomicExch(&st->sweep_error, 1);
            t = 0.0;
            break;
          }
          if (spins > 32) __nanosleep(spins > 256 ? 200 : 20);
          t = ld_relaxed(src);
        }
        smem[lane] = t;
      }
      __syncwarp();
      fence_gpu();
    }
    __syncthreads();
  }
  if (threadIdx.x < NV) st_relaxed(red_slot(red, point, threadIdx.x) + blockIdx.x, pending_value<double>());
}

// A bounded wait without a call (calls made the sweeps spill around them).
template <typename T>
__device__ __forceinline__ T wait_inline(const T* p, PcgState* st, unsigned spin_limit) {
  T x = ld_relaxed(p);
  for (unsigned spins = 1; is_pending(x); ++spins) {
    if (spins >= 4) __nanosleep(64);
    x = ld_relaxed(p);
    if (is_pending(x) && (((spins & 1023u) == 0 && gave_up(st)) || spins >= spin_limit)) {
      atomicExch(&st->sweep_error, 1);
      return T(0);
    }
  }
  return x;
}

// The tasks of one sweep (k_sweep's loop).  `r` is the residual: the forward
// rows' own term; the backward rows' term is g s, and ysum / yr gather sum y and
// y.r of the rows a lane finishes.  The tail's forward rows go to wt.  (The
// slots are marked pending a reduction earlier: y in the update pass, s and wt
// in the mat-vec.  A mark by the task that fills the other vector's slot, as
// the batched sweeps do it across launches, could land after the other sweep's
// value here.)
constexpr int kPersistUnroll = 2;
template <typename T, bool kForward>
__device__ __forceinline__ void persist_sweep(const PersistArgs<T>& P, const T* r, double& ysum, double& yr) {
  constexpr int U = kPersistUnroll;
  const int lane = threadIdx.x & 31;
  const int W = (int)((gridDim.x * blockDim.x) >> 5);
  const int ntasks = kForward ? P.ntf : P.ntb;
  const SweepTask* tasks = kForward ? P.tf : P.tb;
  const int* idx = kForward ? P.fi : P.bi;
  const T* coef = kForward ? P.fc : P.bc;
  T* out = kForward ? P.s : P.y;
  const size_t vs = P.vs;
  int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  SweepTask r1 = load_task(tasks, t + W, ntasks);
  SweepEntries<T, U> e0;
  T a0, b0;  // own term (forward r, backward g), and r for y.r
  auto fetch = [&](SweepEntries<T, U>& e, T& a, T& b, const SweepTask& rec) {
    load_entries<T, true, false, U>(e, rec, lane, idx, coef, coef, coef);
    const bool lead = e.active(lane) && (lane & (e.gw() - 1)) == 0;
    const bool term = lead && e.term();
    if constexpr (kForward) {
      a = term ? r[e.v] : T(0);
      b = T(0);
    } else {
      a = term ? __ldg(&P.g[e.v]) : T(0);
      b = lead && e.value() ? r[e.v] : T(0);
    }
  };
  fetch(e0, a0, b0, load_task(tasks, t, ntasks));
  for (; t < ntasks; t += W) {
    const SweepTask r2 = load_task(tasks, t + 2 * W, ntasks);
    SweepEntries<T, U> e1;
    T a1, b1;
    fetch(e1, a1, b1, r1);
    const int gw = e0.gw();
    const bool lead = e0.active(lane) && (lane & (gw - 1)) == 0;
    T own = T(0);
    if (!kForward && lead && e0.term()) own = ld_relaxed(&P.s[(size_t)e0.v * vs]);
    T acc = T(0);
    gather_entries<T, U, true>(acc, e0.id, e0.c, out, (int)vs, P.st, P.poll_mode, P.spin_limit);
    for (int k = e0.k0 + U * gw; k < e0.k1; k += 4 * gw) {
      int id[4];
      T c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = k + j * gw;
        id[j] = kk < e0.k1 ? __ldg(&idx[kk]) : -1;
        c[j] = kk < e0.k1 ? __ldg(&coef[kk]) : T(0);
      }
      gather_entries<T, 4, true>(acc, id, c, out, (int)vs, P.st, P.poll_mode, P.spin_limit);
    }
    if (!kForward && is_pending(own)) own = wait_inline(&P.s[(size_t)e0.v * vs], P.st, P.spin_limit);
    __syncwarp();  // reconverge after the divergent waits before the shuffles
    acc = group_sum_w(acc, gw);
    if (lead) {
      const T res = kForward ? a0 + acc : a0 * own + acc;
      if (kForward && e0.value() && e0.v >= P.v0) st_relaxed(&P.wt[e0.v - P.v0], res);
      else st_relaxed(&out[(size_t)e0.slot() * vs], res);
      if (!kForward && e0.value()) {
        ysum += (double)res;
        yr += (double)res * (double)b0;
      }
    }
    e0 = e1;
    a0 = a1;
    b0 = b1;
    r1 = r2;
  }
}

// y[v0 + i] = sum_j W[i][j] w[j] for the rows of this warp, w in shared memory
// (padded with zeros to w_stride(K)); 16 bytes a lane and four loads in flight.
template <typename T>
__device__ __forceinline__ T w_row(const T* __restrict__ Wr, const T* w, int ld, int lane) {
  constexpr int V = 16 / sizeof(T);
  using VT = typename std::conditional<sizeof(T) == 8, double2, float4>::type;
  constexpr int U = 4;
  T acc[U] = {};
  const VT* a = reinterpret_cast<const VT*>(Wr);
  const VT* b = reinterpret_cast<const VT*>(w);
  const int m = ld / V;
  for (int j = lane; j < m; j += 32 * U) {
    VT x[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (j + 32 * u < m) x[u] = __ldg(a + j + 32 * u);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (j + 32 * u < m) {
        const VT z = b[j + 32 * u];
        if constexpr (sizeof(T) == 8) {
          acc[u] += x[u].x * z.x;
          acc[u] += x[u].y * z.y;
        } else {
          acc[u] += x[u].x * z.x;
          acc[u] += x[u].y * z.y;
          acc[u] += x[u].z * z.z;
          acc[u] += x[u].w * z.w;
        }
      }
  }
  return group_sum_w((acc[0] + acc[1]) + (acc[2] + acc[3]), 32);
}

// kWhole: W is the whole preconditioner (K = n): no sweeps, and an iteration is
//   x' and r', y = W r'   (each block forms all of r' in shared memory itself)
//   reduce: the norms, sum y, y.r
//   p' = (y - mean) + beta p and q = L p' in one pass (a neighbour's p' is formed
//   again from its y and p; p in two buffers)
//   reduce: p.q and the L1 norms
// so convergence shows after the product it makes needless.  Otherwise p is
// updated in its own pass: gathering y and p for each entry costs more than
// the barrier once the vectors outgrow L1 (grid3(50): mat-vec 24 us, 8 alone).
template <typename T, bool kWhole>
__global__ void __launch_bounds__(kPersistThreads, 2) k_pcg(const __grid_constant__ PersistArgs<T> P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* w = reinterpret_cast<T*>(smem_raw);
  __shared__ double red_sm[kRedValues * kPersistThreads / 32];
  __shared__ PcgState ls;
  PcgState* gst = P.st;
  if (gst->done) return;  // set before this launch, as resumed: the same in every block
  const int tid = threadIdx.x, lane = tid & 31;
  const int gtid = blockIdx.x * blockDim.x + tid, gsize = gridDim.x * blockDim.x;
  const int n = P.n, K = P.K;
  const int ldw = w_stride(K);
  const size_t vs = P.vs;
  bool first = kWhole || !gst->resumed;
  __shared__ double since;  // ls.elapsed in this launch's first iteration
  if (tid == 0) {
    ls = *gst;
    ls.resumed = 0;
    since = -1.0;
    if (P.init == 1 && first) ls.t_start = globaltimer_ns();
  }
  __syncthreads();
  const T* r = P.r0;  // the residual before the update (kWhole), and the current one
  T* rw = kWhole ? P.r1 : P.r0;
  const T* po = P.p0;
  T* pw = kWhole ? P.p1 : P.p0;
  for (;;) {
    // ---- update: x', r' and their norms
    const double alpha = first ? 0.0 : ls.alpha;
    double nrm[4] = {0.0, 0.0, 0.0, 0.0};  // r'.r', |x'|_1, |r'|_1, r'.1
    if (first) {
      for (int i = gtid; i < n; i += gsize) nrm[3] += (double)r[i];
    } else {
      const T* xc = P.x3 + (size_t)ls.xcur * n;
      T* xn = P.x3 + (size_t)ls.xnext * n;
      for (int i = gtid; i < n; i += gsize) {
        const T xv = (T)((double)xc[i] + alpha * (double)po[i]);
        const T rv = (T)((double)r[i] + (-alpha) * (double)P.q[i]);
        xn[i] = xv;
        rw[i] = rv;
        nrm[0] += (double)rv * (double)rv;
        nrm[1] += fabs((double)xv);
        nrm[2] += fabs((double)rv);
        nrm[3] += (double)rv;
      }
    }
    double ysum = 0.0, yr = 0.0;
    if constexpr (kWhole) {
      for (int j = tid; j < ldw; j += blockDim.x)
        w[j] = j < n ? (first ? r[j] : (T)((double)r[j] + (-alpha) * (double)P.q[j])) : T(0);
      __syncthreads();
    } else {
      const double rsum = nrm[3];
      if (!first) {
        for (int i = gtid; i < P.nslots; i += gsize) P.y[(size_t)i * vs] = pending_value<T>();
        double v[3] = {nrm[0], nrm[1], nrm[2]};
        red_publish<3>(P.red, 0, v, red_sm);
        red_collect<3>(P.red, 0, 3, red_sm, gst, P.red_limit);
        if (tid == 0) pcg_scalar_update(&ls, red_sm[0], red_sm[1], red_sm[2]);
        __syncthreads();
        if (ls.done) break;
      }
      nrm[3] = rsum;
      persist_sweep<T, true>(P, r, ysum, yr);
      for (int j = tid; j < ldw; j += blockDim.x)
        w[j] = j < K ? wait_inline(&P.wt[j], gst, P.spin_limit) : T(0);
      __syncthreads();
    }
    // ---- the dense tail, or the whole preconditioner
    for (int i = gtid >> 5; i < K; i += gsize >> 5) {
      const T res = w_row<T>(P.W + (size_t)i * ldw, w, ldw, lane);
      if (lane == 0) {
        st_relaxed(&P.y[(size_t)(P.v0 + i) * vs], res);
        ysum += (double)res;
        yr += (double)res * (double)(kWhole ? w[i] : r[P.v0 + i]);
      }
    }
    if constexpr (!kWhole) persist_sweep<T, false>(P, r, ysum, yr);
    // ---- mean, rho, beta and the stop rules
    {
      // what may differ between blocks travels as a sum: block 0's clock, and
      // whether a wait gave up
      double el = 0.0;
      if (tid == 0) {
        if (blockIdx.x == 0) el = (double)(globaltimer_ns() - ls.t_start) * 1e-9;
        if (gave_up(gst)) el = -1e300;
      }
      if constexpr (kWhole) {
        double v[7] = {ysum, yr, nrm[3], el, nrm[0], nrm[1], nrm[2]};
        red_publish<7>(P.red, 1, v, red_sm);
        red_collect<7>(P.red, 1, 3, red_sm, gst, P.red_limit);
      } else {
        double v[4] = {ysum, yr, nrm[3], el};
        red_publish<4>(P.red, 1, v, red_sm);
        red_collect<4>(P.red, 1, 0, red_sm, gst, P.red_limit);
      }
      if (tid == 0) {
        ls.mean = red_sm[0] / (double)n;
        ls.elapsed = red_sm[3];
        const double rho = red_sm[1] - ls.mean * red_sm[2];
        bool stop = false;
        if (ls.elapsed < 0.0 || gave_up(gst)) stop = mark_stop(&ls, kSweepTimeout);
        else if (kWhole && !first) stop = pcg_scalar_update(&ls, red_sm[4], red_sm[5], red_sm[6]);
        if (!stop) {
          if (first) pcg_scalar_enter(&ls, rho);
          else if (!pcg_scalar_rho(&ls, rho) && ls.itcnt % 10 != 0) pcg_scalar_tail(&ls, P.eps, ls.elapsed);
        }
      }
      __syncthreads();
      if (ls.done) break;
    }
    const double mu = ls.mean, beta = ls.beta;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // p'.q, |p'|_1, |q|_1, |z|_1
    // ---- p' = z + beta p
    if constexpr (!kWhole) {
      for (int i = gtid; i < n; i += gsize) {
        const T z = (T)((double)P.y[(size_t)i * vs] - mu);
        pw[i] = first ? z : (T)((double)z + beta * (double)pw[i]);
        acc[3] += fabs((double)z);
      }
      for (int j = gtid; j < K; j += gsize) P.wt[j] = pending_value<T>();
      for (int i = gtid; i < P.nslots; i += gsize) P.s[(size_t)i * vs] = pending_value<T>();
      double v[1] = {acc[3]};
      red_publish<1>(P.red, 2, v, red_sm);
      red_collect<1>(P.red, 2, 1, red_sm, gst, P.red_limit);
      acc[3] = 0.0;
      if (tid == 0 && !first && ls.itcnt % 10 == 0) {  // the third L1 test, maxtime, maxits
        ls.sum_abs_z = red_sm[0];
        pcg_scalar_tail(&ls, P.eps, ls.elapsed);
      }
      __syncthreads();
      if (ls.done) break;
    }
    // ---- q = L p'
    {
      const int vl = P.vl, gl = tid & (vl - 1);
      const int groups = gsize / vl;
      constexpr int U = 4;
      int next = (gtid & ~31) / vl + (gtid & 31) / vl;
      int n0 = next < n ? __ldg(&P.lp[next]) : 0, n1 = next < n ? __ldg(&P.lp[next + 1]) : 0;
      for (int base = (gtid & ~31) / vl; base < n; base += groups) {
        const int row = next, k0 = n0, k1 = n1;
        const bool active = row < n;
        next += groups;
        n0 = next < n ? __ldg(&P.lp[next]) : 0;
        n1 = next < n ? __ldg(&P.lp[next + 1]) : 0;
        T sum = T(0);
        if (active) {
          for (int k = k0 + gl; k < k1; k += vl * U) {
            int id[U];
            T c[U], pv[U];
#pragma unroll
            for (int j = 0; j < U; ++j) {
              const int kk = k + j * vl;
              id[j] = kk < k1 ? __ldg(&P.li[kk]) : -1;
              c[j] = kk < k1 ? __ldg(&P.lv[kk]) : T(0);
            }
            if constexpr (kWhole) {
              T yv[U];
#pragma unroll
              for (int j = 0; j < U; ++j)
                if (id[j] >= 0) {
                  yv[j] = P.y[(size_t)id[j] * vs];
                  pv[j] = first ? T(0) : po[id[j]];
                }
#pragma unroll
              for (int j = 0; j < U; ++j) {
                const T z = (T)((double)yv[j] - mu);
                pv[j] = first ? z : (T)((double)z + beta * (double)pv[j]);
              }
            } else {
#pragma unroll
              for (int j = 0; j < U; ++j)
                if (id[j] >= 0) pv[j] = pw[id[j]];
            }
#pragma unroll
            for (int j = 0; j < U; ++j)
              if (id[j] >= 0) sum += c[j] * pv[j];
          }
        }
        sum = group_sum_w(sum, vl);
        if (active && gl == 0) {
          T pn;
          if constexpr (kWhole) {
            const T z = (T)((double)P.y[(size_t)row * vs] - mu);
            pn = first ? z : (T)((double)z + beta * (double)po[row]);
            pw[row] = pn;
            acc[3] += fabs((double)z);
          } else {
            pn = pw[row];
          }
          P.q[row] = sum;
          acc[0] += (double)pn * (double)sum;
          acc[1] += fabs((double)pn);
          acc[2] += fabs((double)sum);
        }
      }
      red_publish<4>(P.red, 3, acc, red_sm);
      red_collect<4>(P.red, 3, kWhole ? 1 : 2, red_sm, gst, P.red_limit);
      if (tid == 0) {
        bool stop = false;
        if (gave_up(gst)) {
          stop = mark_stop(&ls, kSweepTimeout);
        } else if (kWhole && !first && ls.itcnt % 10 == 0) {  // the third L1 test, maxtime, maxits
          ls.sum_abs_z = red_sm[3];
          stop = pcg_scalar_tail(&ls, P.eps, ls.elapsed);
        }
        if (!stop) stop = pcg_scalar_pq(&ls, red_sm[0], red_sm[1], red_sm[2], P.eps);
        if constexpr (!kWhole) {
          // the same in every block: elapsed is block 0's, through a reduction
          if (since < 0.0) since = ls.elapsed;
          if (!stop && ls.elapsed - since > P.slice_s) ls.resumed = 1;
        }
      }
      __syncthreads();
      if (ls.done || (!kWhole && ls.resumed)) break;
    }
    if constexpr (kWhole) {
      const T* t = po;
      po = pw;
      pw = const_cast<T*>(t);
      if (!first) {
        const T* u = r;
        r = rw;
        rw = const_cast<T*>(u);
      }
    }
    first = false;
  }
  if (blockIdx.x == 0 && tid == 0) {
    const int err = gave_up(gst) ? 1 : 0;
    for (int k = 0; k < 16; ++k) ls.counter[k] = 0u;
    ls.sweep_error = err;
    if (err) mark_stop(&ls, kSweepTimeout);
    *gst = ls;
  }
}

// ---- one preconditioner application (LDLsolver, src/approxChol.jl:1347-1366) ----
//
// Two launches instead of a dozen: k_apply_begin takes r in solver order and
// arms the vectors, k_apply runs both sweeps, the tail and the mean removal.
// (One right-hand side of grid3(50), FP64: 277 -> 242 us a call.)
template <typename T>
__global__ void __launch_bounds__(kVecThreads) k_apply_begin(PersistArgs<T> P, const int* __restrict__ perm,
                                                             const double* __restrict__ rext, int nred) {
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gsize = gridDim.x * blockDim.x;
  for (int i = gtid; i < P.n; i += gsize) P.r0[i] = (T)rext[perm[i]];
  for (int i = gtid; i < P.nslots; i += gsize) {
    P.s[(size_t)i * P.vs] = pending_value<T>();
    P.y[(size_t)i * P.vs] = pending_value<T>();
  }
  for (int i = gtid; i < P.K; i += gsize) P.wt[i] = pending_value<T>();
  for (int i = gtid; i < nred; i += gsize) P.red[i] = pending_value<double>();
  if (gtid == 0) *P.st = PcgState{};
}

template <typename T, bool kWhole>
__global__ void __launch_bounds__(kPersistThreads, 2) k_apply(const __grid_constant__ PersistArgs<T> P,
                                                              const int* __restrict__ perm, double* __restrict__ yext) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* w = reinterpret_cast<T*>(smem_raw);
  __shared__ double red_sm[kRedValues * kPersistThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  const int gtid = blockIdx.x * blockDim.x + tid, gsize = gridDim.x * blockDim.x;
  const int K = P.K, ldw = w_stride(K);
  const size_t vs = P.vs;
  double ysum[1] = {0.0}, unused = 0.0;
  if constexpr (!kWhole) persist_sweep<T, true>(P, P.r0, ysum[0], unused);
  for (int j = tid; j < ldw; j += blockDim.x)
    w[j] = j < K ? (kWhole ? P.r0[j] : wait_inline(&P.wt[j], P.st, P.spin_limit)) : T(0);
  __syncthreads();
  for (int i = gtid >> 5; i < K; i += gsize >> 5) {
    const T res = w_row<T>(P.W + (size_t)i * ldw, w, ldw, lane);
    if (lane == 0) {
      st_relaxed(&P.y[(size_t)(P.v0 + i) * vs], res);
      ysum[0] += (double)res;
    }
  }
  if constexpr (!kWhole) persist_sweep<T, false>(P, P.r0, ysum[0], unused);
  red_publish<1>(P.red, 0, ysum, red_sm);
  red_collect<1>(P.red, 0, 1, red_sm, P.st, P.red_limit);
  const double mean = red_sm[0] / (double)P.n;
  for (int i = gtid; i < P.n; i += gsize) yext[perm[i]] = (double)P.y[(size_t)i * vs] - mean;
}

// Ends the loop around k_pcg's launches once the solve is done.  A kernel of its
// own: with the call that sets the condition in k_pcg an iteration took 15 to
// 30 % longer, also where no launch left early (200 x 200 grid 56 -> 68 us,
// matchings of 150,000 vertices 213 -> 278).
static __global__ void k_pcg_loop(const PcgState* st, LoopCtl ctl) {
  if (st->done) clear_loop(ctl);
}

// The one-vector kernels are compiled in acg_persist.cu alone.
#define ACG_PERSIST_KERNELS(INST)                                                                                 \
  INST __global__ void k_pcg<double, true>(const __grid_constant__ PersistArgs<double>);                          \
  INST __global__ void k_pcg<double, false>(const __grid_constant__ PersistArgs<double>);                         \
  INST __global__ void k_pcg<float, true>(const __grid_constant__ PersistArgs<float>);                            \
  INST __global__ void k_pcg<float, false>(const __grid_constant__ PersistArgs<float>);                           \
  INST __global__ void k_apply<double, true>(const __grid_constant__ PersistArgs<double>, const int*, double*);   \
  INST __global__ void k_apply<double, false>(const __grid_constant__ PersistArgs<double>, const int*, double*);  \
  INST __global__ void k_apply<float, true>(const __grid_constant__ PersistArgs<float>, const int*, double*);     \
  INST __global__ void k_apply<float, false>(const __grid_constant__ PersistArgs<float>, const int*, double*);
ACG_PERSIST_KERNELS(extern template)

// mean[k] = the mean of row k of M (K x K, row-major, lower triangular), a
// warp a row.
static __global__ void __launch_bounds__(256) k_row_mean(int K, const double* __restrict__ M, double* __restrict__ mean) {
  const int lane = threadIdx.x & 31, k = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (k >= K) return;
  double sum = 0.0;
  for (int i = lane; i <= k; i += 32) sum += M[(size_t)k * K + i];
  sum = group_sum_w(sum, 32);
  if (lane == 0) mean[k] = sum / K;
}

// W = (M - mean 1^T)^T diag(g) M for the dense tail (or the whole graph): M is
// K x K row-major lower triangular, W's rows are padded with zeros to ldw
// columns.  M^T diag(g) M is the operator; a constant in a column of W only
// shifts all of y, which the mean removal takes out again, and the rows of M
// near the root are nearly constant (all flows to the root, whose own row is
// all ones and is left out).  With these constants in W its entries are far
// larger than what they say of y, and the rounding of each row's sum shows:
// on matchings of 60,000 vertices with lognormal weights one application was
// 4.6e-14 from 64 bits without the means and the root taken out, 6e-16 with
// the two triangular products.  The sums over k carry their rounding errors
// along (two-sum and a product split by fma), since W is used many times; the
// intrinsics keep the compiler from contracting a product into the additions
// around it, which would count its rounding error twice.
// 64 x 64 tiles, 4 x 4 entries a thread, FP64.  Run once per solver.
constexpr int kWTile = 64;
static __global__ void __launch_bounds__(256) k_form_w(int K, int ldw, const double* __restrict__ M,
                                                const double* __restrict__ mean, const double* __restrict__ g,
                                                double* __restrict__ W64, float* __restrict__ W32) {
  __shared__ double A[16][kWTile + 1], B[16][kWTile + 1];
  const int i0 = blockIdx.y * kWTile, j0 = blockIdx.x * kWTile;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[4][4] = {}, low[4][4] = {};
  const int rows = K - 1;  // without the root
  // column j of M has entries in rows k >= j only
  for (int k0 = (j0 / 16) * 16; k0 < rows; k0 += 16) {
    for (int e = threadIdx.x; e < 16 * kWTile; e += 256) {
      const int kk = e / kWTile, c = e % kWTile, k = k0 + kk;
      const bool in = k < rows;
      A[kk][c] = in ? ((i0 + c <= k ? M[(size_t)k * K + i0 + c] : 0.0) - mean[k]) * g[k] : 0.0;
      B[kk][c] = in && j0 + c <= k ? M[(size_t)k * K + j0 + c] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < 16; ++kk)
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const double x = A[kk][ty * 4 + a], z = B[kk][tx * 4 + b], old = acc[a][b];
          const double prod = __dmul_rn(x, z), sum = __dadd_rn(old, prod), t = __dsub_rn(sum, old);
          const double err = __dadd_rn(__dsub_rn(old, __dsub_rn(sum, t)), __dsub_rn(prod, t));
          low[a][b] = __dadd_rn(low[a][b], __dadd_rn(err, __fma_rn(x, z, -prod)));
          acc[a][b] = sum;
        }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + ty * 4 + a, j = j0 + tx * 4 + b;
      if (i < K && j < ldw) {
        const double v = j < K ? acc[a][b] + low[a][b] : 0.0;
        W64[(size_t)i * ldw + j] = v;
        W32[(size_t)i * ldw + j] = (float)v;
      }
    }
}

}  // namespace acg
