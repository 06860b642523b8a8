// batch_kernel.cuh -- many independent 1D tubes advanced in one persistent
// launch.
//
// Each tube is a 1D grid of its own length with its own time t, step size dt
// and end time (the hydro loop main.f90:109-155 per tube: primitive, bound,
// hydrostep, updatetime, compevo, sweep with the 1D predictor of
// muscl.f90:60-69).  A CTA pulls the next tube from a work queue (tubes are
// ordered by estimated work, largest first), stages its conserved state in
// shared memory and runs up to `budget` steps of that tube without leaving
// the SM, then writes the state back: HBM sees each tube once per launch.
//
// Per step, with the tube in shared memory:
//   phase 1  primitives of the n cells and the 2+2 ghost cells (index map of
//            bound, boundary.f90:33-66) into w, and the block's maximum of
//            |u_d| + a; every thread forms dt (hydrostep) and advances t
//            (updatetime) from it;
//   phase 2  each warp updates 30 consecutive cells at a time (muscl.f90:
//            194-215): a lane per cell and interface, face states and fluxes
//            passed on by shuffles (tube_sweep).
// Bound: instruction issue (64 % of the issue slots in FP32, 61 % in FP64, at
// 16 warps per SM; 374 and 673 instructions per cell-update; no HBM traffic to
// speak of).  A lane per interface solves every interface once (1.07 times, with
// the 2 of 32 lanes that only feed their neighbours); a contiguous segment of
// cells per thread, as this kernel first had, solved it (n / NT + 1) / (n /
// NT) times and read w at strides that met in the banks.  4096 tubes of
// 128-4096 cells, FP32: 245 -> 140 ms; 2048 of them in FP64: 299 -> 155 ms.
// A tube longer than the shared-memory capacity keeps q in a global scratch
// slot of its CTA and w in shared memory while w alone fits, else both in
// the slot (same code, generic pointers).
#pragma once

#include <cooperative_groups.h>

#include "batch.h"
#include "fused_kernel.cuh"

namespace evora {
namespace EVORA_FNS {

// The maximum over a tube's cells of |u_d| + a as dt = min(cfl min(dx / s,
// 1e6)): cfl_dt with dx = dy = dz (compparameter's 1D branch), where the
// smallest of the three quotients is the one by the largest speed.
__device__ __forceinline__ double cfl_dt1(const HydroParams& P, double smax, unsigned& err) {
  const double v = fmin2(P.dx / smax, 1e6);
  const double dt = fmin2(P.cfl * v, 1e99);
  if (dt <= 0.0) err |= EVORA_ERR_DT;
  return dt;
}

// Primitives of the n cells of a tube and its 2 + 2 ghosts (the index map of
// bound) into w (field-major, stride n + 4); returns this thread's maximum of
// |u_d| + a over the cells (timestep.f90:40-43), reduced over its warp.  One
// maximum serves the three axes: a sum of |u_d| and a rounds monotonically,
// so the largest |u_d| gives the largest sum.
template <typename T, int NF, int NT>
__device__ __forceinline__ T tube_primitives(const T* qs, T* w, int n, const HydroParams& P, const Gas<T>& c,
                                             bool de, unsigned& err) {
  const int wst = n + 4;
  T smax = (T)0;
  for (int i = threadIdx.x; i < wst; i += NT) {
    bool flip = false;
    const int g = ghost_map(i - 2, n, P.boundtype, 0, flip);
    T qv[6], wv[5];
#pragma unroll
    for (int f = 0; f < NF; ++f) qv[f] = qs[f * n + g];
    prim_k(qv, wv, c, P, de, err);
    if (flip) {
      wv[1] = -wv[1];
      wv[2] = -wv[2];
      wv[3] = -wv[3];
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) w[f * wst + i] = wv[f];
    if (i >= 2 && i < n + 2) {
      T a;
      if constexpr (kFast && sizeof(T) == 8) a = sqrt_fast(c.g * wv[4] * rcp_fast(wv[0]));
      else a = dsqrt(c.g * wv[4] / wv[0]);
      const T s = fmax2(fmax2((T)fabs(wv[1]), (T)fabs(wv[2])), (T)fabs(wv[3])) + a;
      if (s > smax) smax = s;
    }
  }
  return warp_max_pos(smax);
}

// The update of a tube (muscl.f90:60-69, 194-215) from the primitives in w.
// A warp takes 32 consecutive cells: every lane forms the face states of
// its cell, the upper one goes to the next lane by shuffle, a lane solves the
// interface below its cell, and the flux above comes back by shuffle; the
// first and last cell only feed their neighbours, so a chunk updates 30
// cells.  w and q are read and written at consecutive addresses.
template <typename T, int NF, int NT>
__device__ __forceinline__ void tube_sweep_opt(T* qs, const T* w, int n, const HydroParams& P, int limiter,
                                               int solver, bool secondorder, const Gas<T>& c, bool de, double dt,
                                               unsigned& err) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int wst = n + 4;
  const T dt2 = (T)(-0.5 * dt);
  const T dtdx = (T)(dt * P.dxinv);
  const T dxi = (T)P.dxinv;
  for (int c0 = 30 * wid; c0 < n; c0 += 30 * (NT / 32)) {
    const int cc = c0 - 1 + lane;            // this lane's cell, -1 .. n
    const int wi = (cc < n ? cc : n) + 2;    // lanes past the upper ghost repeat it
    T wc[5], fm[5], fp[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) wc[f] = w[f * wst + wi];
    if (secondorder) {
      T s[5], a[5];
      with_limiter<false>(limiter, [&](auto lim) {
#pragma unroll
        for (int f = 0; f < 5; ++f) s[f] = slope_k(w[f * wst + wi - 1], wc[f], w[f * wst + wi + 1], lim);
      });
      pred_k(wc, s, 1, c.g, kFast ? rcp_fast(wc[0]) : (T)0, a);
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        faces1d(wc[f], s[f], dt2, a[f], dxi, fm[f], fp[f]);
      }
    } else {
#pragma unroll
      for (int f = 0; f < 5; ++f) fm[f] = fp[f] = wc[f];
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) fp[f] = __shfl_up_sync(0xffffffffu, fp[f], 1);
    T flo[NF], fhi[NF];
    unsigned e = 0;
    riemann_k<T, NF, 1>(fp, fm, flo, solver, c, e);   // interface cc-1/2
    if (lane > 0 && cc <= n) err |= e;                  // the tube's n + 1 interfaces
#pragma unroll
    for (int f = 0; f < NF; ++f) fhi[f] = __shfl_down_sync(0xffffffffu, flo[f], 1);
    if (lane > 0 && lane < 31 && cc < n) {
      T qv[6];
#pragma unroll
      for (int f = 0; f < NF; ++f) qv[f] = qs[f * n + cc];
      if (de) {
        T wd[5];
        unsigned e2 = 0;
        prim_k(qv, wd, c, P, de, e2);   // dual-energy resync of q (comp.f90:60-72)
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) qs[f * n + cc] = axpy_k<kFast>(qv[f], dtdx, flo[f] - fhi[f]);
    }
  }
}

// The usual options (minmod, HLLC, second order) as constants, so that their
// sweep has no branches on them.
template <typename T, int NF, int NT>
__device__ __forceinline__ void tube_sweep(T* qs, const T* w, int n, const HydroParams& P, const Gas<T>& c, bool de,
                                           double dt, unsigned& err) {
  if (P.limiter == 1 && P.solver == 2 && P.secondorder && !de)
    tube_sweep_opt<T, NF, NT>(qs, w, n, P, 1, 2, true, c, false, dt, err);
  else
    tube_sweep_opt<T, NF, NT>(qs, w, n, P, P.limiter, P.solver, P.secondorder != 0, c, de, dt, err);
}

// compparameter for a tube of n cells (parameter.f90:192-205, 1D branch);
// bt: its boundary type (0: the batch's).
template <typename T>
__device__ __forceinline__ HydroParams tube_params(const BatchArgs<T>& A, int n, int bt) {
  HydroParams P = A.P;
  if (bt) P.boundtype = bt;
  P.nx = n;
  P.ny = 1;
  P.nz = 1;
  P.dx = (A.xmax - A.xmin) / n;
  P.dy = P.dx;
  P.dz = P.dx;
  {
    double ymax = P.dy, zmax = P.dz;
    P.dy = (ymax - 0.0) / 1;
    P.dz = (zmax - 0.0) / 1;
  }
  P.dxinv = 1.0 / P.dx;
  P.dyinv = 1.0 / P.dy;
  P.dzinv = 1.0 / P.dz;
  return P;
}

// The most steps a tube of n cells runs in this launch.
template <typename T>
__device__ __forceinline__ int tube_budget(const BatchArgs<T>& A, int n) {
  int budget = A.budget;
  if (A.quantum > 0) {
    const long long b = A.quantum / n;
    budget = (int)(b < 1 ? 1 : (b < budget ? b : budget));
  }
  if (A.steps_per_cell > 0.0) budget = max(1, (int)(A.steps_per_cell * n));
  return budget;
}

// A tube's bookkeeping after a launch (one thread).
template <typename T>
__device__ __forceinline__ void tube_close(const BatchArgs<T>& A, TubeState* ts, int n, double t, double dt, int steps,
                                           unsigned err, int go) {
  ts->err |= err;
  ts->t = t;
  ts->dt = dt;
  ts->k += steps;
  if (err) ts->status = TUBE_ERROR;
  else if (!go) ts->status = TUBE_DONE;
  atomicAdd((unsigned long long*)A.cell_updates, (unsigned long long)n * (unsigned long long)steps);
}

template <typename T, int NF, int NT>
__device__ __forceinline__ void tube_run(const BatchArgs<T>& A, T* qs, T* w, int tb, T* red,
                                         unsigned* s_err) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  TubeState* ts = A.tubes + tb;
  const int n = ts->n;
  const long long off = ts->offset;
  const HydroParams P = tube_params(A, n, ts->bt);
  const Gas<T> c = Gas<T>::make(P);
  const bool de = P.dualenergy != 0;
  // stage q into qs (field-major, stride n)
  for (int f = 0; f < NF; ++f)
    for (int i = tid; i < n; i += NT) qs[f * n + i] = A.q[(size_t)f * A.ntot + off + i];
  double t = ts->t, dt = ts->dt, tend = ts->tend;
  unsigned err = 0;
  int steps = 0, go = 1;
  if (tid == 0) *s_err = 0u;
  const int budget = tube_budget(A, n);
  __syncthreads();
  while (steps < budget) {
    // ---- phase 1: primitives (+ ghosts) and the CFL maximum
    const T sm = tube_primitives<T, NF, NT>(qs, w, n, P, c, de, err);
    if (lane == 0) red[wid] = sm;
    if (err) atomicOr(s_err, err);
    __syncthreads();
    // every thread forms dt and advances t from the warps' maxima
    unsigned e = *s_err;
    const double smax = (double)warp_max_pos(lane < NT / 32 ? red[lane] : (T)0);
    double d = cfl_dt1(P, smax, e), tt = t;
    int g2 = 1;
    if (!e) update_time(tend, tt, d, g2);
    if (!e && g2 && !(tt > t)) e |= EVORA_ERR_DT;   // dt below the resolution of t: no progress
    if (e) {                       // an error stops the tube before its update
      err |= e;
      break;
    }
    dt = d;
    t = tt;
    go = g2;
    // ---- phase 2: the update
    tube_sweep<T, NF, NT>(qs, w, n, P, c, de, dt, err);
    ++steps;
    if (__syncthreads_or(err != 0) || !go) break;   // a Riemann error stops the tube after its step
  }
  if (err) atomicOr(s_err, err);
  // write back
  for (int f = 0; f < NF; ++f)
    for (int i = tid; i < n; i += NT) A.q[(size_t)f * A.ntot + off + i] = qs[f * n + i];
  __syncthreads();
  if (tid == 0) tube_close(A, ts, n, t, dt, steps, *s_err, go);
}

template <typename T, int NF, int NT>
__global__ void __launch_bounds__(NT) k_tubes(BatchArgs<T> A) {
  extern __shared__ __align__(16) unsigned char sraw[];
  __shared__ int s_tube;
  __shared__ T red[NT / 32];
  __shared__ unsigned s_err;
  for (;;) {
    if (threadIdx.x == 0) {
      const int i = atomicAdd(A.head, 1);
      s_tube = i < A.ntubes ? A.order[i] : -1;
    }
    __syncthreads();
    const int tb = s_tube;
    __syncthreads();
    if (tb < 0) break;
    if (A.tubes[tb].status != TUBE_RUNNING) continue;
    const int n = A.tubes[tb].n;
    T* qs;
    T* w;
    if (n <= A.cap) {
      qs = reinterpret_cast<T*>(sraw);
      w = qs + NF * A.cap;
    } else if (n <= A.capw) {
      // the primitives (read three times per cell and step by the sweeps)
      // in shared memory, the state in the CTA's scratch slot
      w = reinterpret_cast<T*>(sraw);
      qs = A.gscratch + (size_t)blockIdx.x * (size_t)(NF + 5) * (A.nmax + 4);
    } else {
      qs = A.gscratch + (size_t)blockIdx.x * (size_t)(NF + 5) * (A.nmax + 4);
      w = qs + (size_t)NF * (A.nmax + 4);
    }
    tube_run<T, NF, NT>(A, qs, w, tb, red, &s_err);
  }
}

// ---- lines of cells shared by the CTAs of a thread-block cluster: several
// steps of a resident 1D grid in one launch, and tubes of batches too small
// to give every SM one (the loop main.f90:109-155).
//
// Rank r of the cluster keeps the cells [r m, r m + its cells) in shared
// memory over the steps.  Per step it forms the primitives of its cells,
// stores the two at either end into its neighbours' halos (or, at the ends of
// the line, mirrors them into its own) and its warps' maxima and errors into
// every rank, all through distributed shared memory; one cluster barrier; dt
// from all maxima; the sweep; one block barrier.  Halos, maxima and errors are
// double-buffered by the step's parity: a rank that is one barrier ahead
// writes the other copy.
// Bound: the latency of the step's dependent chain.  Resident grid, 1024 FP64
// cells: 9.0 (five launches per step) -> 2.2 us per step; by size and number of
// ranks: steps1d_plan (fused_inst.cuh).
template <typename T, int NT>
struct LineMax {
  T smax[2][16 * (NT / 32)];
  unsigned err[2][16 * (NT / 32)];
};

// The line and its running time; every thread of the cluster holds the same.
struct LineRun {
  double t, dt, tend;
  int go;        // updatetime's flag
  int active;    // the last step asked for was run (or ended in an error of its update)
  int k;         // steps done
  unsigned err;
};

// Up to nsteps steps of the line of n cells at q (field stride fs) by the
// first ranks of the cluster, m cells each; the other ranks only keep step.
// TUBE: a step whose update fails counts, and one that does not advance t
// raises EVORA_ERR_DT (tube_run); else the control block's rules
// (step_begin, step_time, step_end).  smem: steps1d_smem(NF, m) bytes.
template <typename T, int NF, int NT, bool TUBE>
__device__ __forceinline__ void line_steps(const HydroParams& P, const Gas<T>& c, bool de, T* q, int64_t fs, int n,
                                           int m, int nsteps, bool runnable, unsigned char* smem, LineMax<T, NT>& mx,
                                           LineRun& L) {
  namespace cg = cooperative_groups;
  constexpr int NW = NT / 32;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), nr = (int)cl.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int used = (n + m - 1) / m;              // ranks that have cells (each >= 2)
  const int x0 = rank * m;
  const int mine = rank < used ? (n - x0 < m ? n - x0 : m) : 0;
  const int wlen = 5 * (m + 4);                  // one copy of the primitives
  T* const w0 = reinterpret_cast<T*>(smem);
  T* const qs = w0 + 2 * wlen;                   // field-major, stride mine
  const int wst = mine + 4;
  // the neighbours' primitives and row strides
  const bool periodic = P.boundtype == 2;
  const int lr = rank > 0 ? rank - 1 : (periodic ? used - 1 : -1);
  const int ur = rank < used - 1 ? rank + 1 : (periodic ? 0 : -1);
  auto cells_of = [&](int r) { return n - r * m < m ? n - r * m : m; };
  T* const wl = lr >= 0 ? cl.map_shared_rank(w0, lr) : w0;
  T* const wu = ur >= 0 ? cl.map_shared_rank(w0, ur) : w0;
  const int ml = lr >= 0 ? cells_of(lr) : mine, mu = ur >= 0 ? cells_of(ur) : mine;
  unsigned err_step = 0;   // this thread's errors of the last sweep, not yet exchanged
  for (int f = 0; f < NF; ++f)
    for (int i = tid; i < mine; i += NT) qs[f * mine + i] = q[f * fs + x0 + i];
  cl.sync();   // every rank is here before any stores into its shared memory
  for (int s = 0;; ++s) {
    const int par = s & 1;
    T* const w = w0 + par * wlen;
    // another step, unless the run has ended (step_begin); the round after
    // the last step only exchanges its errors
    const bool step = s < nsteps && L.go != 0 && runnable;
    L.active = step ? 1 : (s < nsteps ? 0 : L.active);
    T smax = (T)0;
    unsigned e = 0;
    if (step) {
      for (int i = tid; i < mine; i += NT) {
        T qv[6], wv[5];
#pragma unroll
        for (int f = 0; f < NF; ++f) qv[f] = qs[f * mine + i];
        prim_k(qv, wv, c, P, de, e);
#pragma unroll
        for (int f = 0; f < 5; ++f) w[f * wst + i + 2] = wv[f];
        T a;
        if constexpr (kFast && sizeof(T) == 8) a = sqrt_fast(c.g * wv[4] * rcp_fast(wv[0]));
        else a = dsqrt(c.g * wv[4] / wv[0]);
        const T sp = fmax2(fmax2((T)fabs(wv[1]), (T)fabs(wv[2])), (T)fabs(wv[3])) + a;
        if (sp > smax) smax = sp;
        // bound (boundary.f90:33-66) and the ranks' halos
        if (i < 2) {
          T* d = lr >= 0 ? wl + par * wlen + ml + 2 + i : w + 1 - i;
          const int st = lr >= 0 ? ml + 4 : wst;
#pragma unroll
          for (int f = 0; f < 5; ++f) d[f * st] = wv[f];
        }
        if (i >= mine - 2) {
          const int j = mine - 1 - i;
          T* d = ur >= 0 ? wu + par * wlen + 1 - j : w + mine + 2 + j;
          const int st = ur >= 0 ? mu + 4 : wst;
          const bool flip = ur < 0 && P.boundtype == 3;
#pragma unroll
          for (int f = 0; f < 5; ++f) d[f * st] = flip && f >= 1 && f <= 3 ? -wv[f] : wv[f];
        }
      }
      smax = warp_max_pos(smax);
    }
    // a sweep's errors in the upper, the primitives' in the lower half
    const unsigned eall = __reduce_or_sync(0xffffffffu, (err_step << 16) | e);
    if (lane < nr) {
      LineMax<T, NT>* r = cl.map_shared_rank(&mx, lane);
      r->smax[par][rank * NW + wid] = smax;
      r->err[par][rank * NW + wid] = eall;
    }
    cl.sync();
    T g = (T)0;
    unsigned ge = 0;
    for (int i = lane; i < nr * NW; i += 32) {
      g = fmax2(g, mx.smax[par][i]);
      ge |= mx.err[par][i];
    }
    ge = __reduce_or_sync(0xffffffffu, ge);
    if (ge >> 16) {   // the last sweep failed: nothing after it
      L.err |= ge >> 16;
      if (TUBE) ++L.k;
      if (s < nsteps) L.active = 0;
      break;
    }
    if (s > 0) ++L.k;
    if (!step) break;
    const double gm = (double)warp_max_pos(g);
    unsigned ed = ge & 0xffffu;
    double d = 0.0, t = L.t;
    int go = L.go;
    if (!ed) d = cfl_dt1(P, gm, ed);
    if (!ed) update_time(L.tend, t, d, go);
    if (TUBE && !ed && go && !(t > L.t)) ed |= EVORA_ERR_DT;   // dt below the resolution of t: no progress
    if (ed) {         // hydrostep's errors: no update
      L.err |= ed;
      L.active = 0;
      break;
    }
    L.t = t;
    L.dt = d;
    L.go = go;
    err_step = 0;
    if (mine > 0) tube_sweep<T, NF, NT>(qs, w, mine, P, c, de, d, err_step);
    __syncthreads();
  }
  for (int f = 0; f < NF; ++f)
    for (int i = tid; i < mine; i += NT) q[f * fs + x0 + i] = qs[f * mine + i];
  cl.sync();   // no rank goes on while its shared memory may be written
}

template <typename T, int NF, int NT>
__global__ void __launch_bounds__(NT) k_steps1d(HydroParams P, T* __restrict__ q, GridCtl* ctl, int nsteps, int m) {
  extern __shared__ __align__(16) unsigned char sraw[];
  __shared__ LineMax<T, NT> mx;
  LineRun L{ctl->t, ctl->dt, ctl->tend, ctl->go, ctl->active, 0, 0u};
  line_steps<T, NF, NT, false>(P, Gas<T>::make(P), NF == 6 && P.dualenergy != 0, q, P.nx, P.nx, m, nsteps,
                               ctl->err == 0 && ctl->dump == 0, sraw, mx, L);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->t = L.t;
    ctl->dt = L.dt;
    ctl->go = L.go;
    ctl->active = L.active;
    ctl->k += L.k;
    ctl->err |= L.err;
    ctl->errnext = 0u;
    ctl->snext[0] = ctl->snext[1] = ctl->snext[2] = 0ull;
  }
}

// The tubes of a small batch, a cluster per tube: a CTA per tube leaves most SMs
// idle and the longest tube takes its 20 us per step (8000 cells FP32); 8 CTAs
// take 3.7.  A rank takes at least 64 cells.  By size and count: cluster_ranks
// (fused_inst.cuh).
template <typename T, int NF, int NT>
__global__ void __launch_bounds__(NT) k_tubes_cluster(BatchArgs<T> A) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char sraw[];
  __shared__ LineMax<T, NT> mx;
  __shared__ int s_tube;
  cg::cluster_group cl = cg::this_cluster();
  const int nr = (int)cl.num_blocks();
  for (;;) {
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
      const int i = atomicAdd(A.head, 1);
      s_tube = i < A.ntubes ? A.order[i] : -1;
    }
    cl.sync();
    const int tb = *cl.map_shared_rank(&s_tube, 0);
    cl.sync();   // all have read it
    if (tb < 0) break;
    TubeState* ts = A.tubes + tb;
    if (ts->status != TUBE_RUNNING) continue;
    const int n = ts->n;
    const HydroParams P = tube_params(A, n, ts->bt);
    int m = (n + nr - 1) / nr;
    if (m < 64) m = 64;
    while (n % m == 1) ++m;   // every used rank has two cells or more
    LineRun L{ts->t, ts->dt, ts->tend, 1, 1, 0, 0u};
    line_steps<T, NF, NT, true>(P, Gas<T>::make(P), P.dualenergy != 0, A.q + ts->offset, A.ntot, n, m,
                                tube_budget(A, n), true, sraw, mx, L);
    if (cl.block_rank() == 0 && threadIdx.x == 0) tube_close(A, ts, n, L.t, L.dt, L.k, L.err, L.go);
  }
}

}  // namespace EVORA_FNS
}  // namespace evora
