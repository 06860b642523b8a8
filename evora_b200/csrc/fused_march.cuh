// fused_march.cuh -- the 2D update (muscl.f90:171-290 with the 2D predictor
// 70-88) with a warp per strip of columns, marching up the rows.
//
// Lane l of a warp holds column X0 - 2 + l; 28 of the 32 columns are updated,
// the two at either end only feed their neighbours.  Per row the lane has the
// primitives of its column in rows c-1, c, c+1 in registers; x neighbours, x
// face states and x fluxes pass between lanes by shuffles, y faces and fluxes
// stay in the lane.  No shared memory and no barrier inside the march, and
// every interface is solved once (1.14 times with the end lanes; rows above
// and below a chunk are recomputed: (R + 2) / R face states).
//
// Bound: instruction issue on large grids, the latency of the row's dependent
// chain on small ones, where the rows per warp (R) are chosen so that the
// warps fill the SMs (choose_rows, fused.cu).  The tile program this
// replaces in 2D (fused_tile) has a CTA of 128 or 256 threads go through four
// barriers for one tile and solves the halo's primitives 1.7 times.  us per
// step, FP32 / FP64, the tile program with its control kernel -> this:
// 64^2 8.8 / 11.0 -> 5.5 / 6.2, 512^2 22.7 / 43.2 -> 14.7 / 23.2,
// 1024^2 64.3 / 156 -> 31.7 / 72, 1400^2 119 / 289 -> 55 / 130.
#pragma once

#include "fused_kernel.cuh"

namespace evora {
namespace EVORA_FNS {

constexpr int kMarchCols = 28;    // columns a warp updates
constexpr int kMarchWarps = 4;    // warps per CTA

// Warp gw of the grid's strips x chunks (A.zc rows per chunk).  cm: running
// maxima of |u_d| + a of the written cells.
// RC > 0: that many rows per warp, the rows unrolled (their chains overlap).
template <typename T, int NF, bool OPT, int RC = 0>
__device__ __forceinline__ void march2d(const FusedArgs<T>& A, int gw, T* cm, unsigned& cerr) {
  const HydroParams& P = A.P;
  const int nx = P.nx, ny = P.ny, R = RC > 0 ? RC : A.zc;
  const int lane = threadIdx.x & 31;
  const int nstrips = (nx + kMarchCols - 1) / kMarchCols;
  const int X0 = (gw % nstrips) * kMarchCols, Y0 = (gw / nstrips) * R;
  if (Y0 >= ny) return;
  const int ye = ny - Y0 < R ? ny - Y0 : R;
  const int64_t n = A.n;
  const int x = X0 - 2 + lane;
  const bool owned = lane >= 2 && lane < 30 && x < nx;
  if (ctl_skip(A.ctl)) {
    if (owned)
      for (int y = Y0; y < Y0 + ye; ++y) {
        const int64_t idx = (int64_t)y * nx + x;
#pragma unroll
        for (int f = 0; f < NF; ++f) A.qout[f * n + idx] = A.qin[f * n + idx];
      }
    return;
  }
  const Gas<T> c = Gas<T>::make(P);
  const bool de = NF == 6 && P.dualenergy != 0;
  const int solver = OPT ? 2 : P.solver;
  const double dtd = A.ctl->dt;
  const T dt2 = (T)(-0.5 * dtd);
  const T dtdx = (T)(dtd * P.dxinv), dtdy = (T)(dtd * P.dyinv);
  unsigned err = 0;
  // lanes past the grid's two upper ghost columns repeat the outer one
  bool flip = false;
  const int mx = ghost_map(x > nx + 1 ? nx + 1 : x, nx, P.boundtype, 0, flip);
  auto row = [&](int y) {
    bool fl = false;
    return (int64_t)ghost_map(y > ny + 1 ? ny + 1 : y, ny, P.boundtype, 1, fl) * nx + mx;
  };
  auto load = [&](int y, T* qv) {
    const T* p = A.qin + row(y);
#pragma unroll
    for (int f = 0; f < NF; ++f) qv[f] = p[f * n];   // coherent loads: step_head
  };
  auto convert = [&](T* qv, T* wv) {
    prim_k(qv, wv, c, P, de, err);
    if (flip) {
      wv[1] = -wv[1];
      wv[2] = -wv[2];
      wv[3] = -wv[3];
    }
  };
  T wm[5], wc[5], wp[5], qv[6], qn[6];
  load(Y0 - 2, qv);
  load(Y0 - 1, qn);
  convert(qv, wm);
  load(Y0, qv);
  convert(qn, wc);
  load(Y0 + 1, qn);
  convert(qv, wp);
  T yu[5], fy[NF], qacc[NF];   // upper y face of row r-1, flux r-3/2, row r-1 after its x term
#pragma unroll
  for (int f = 0; f < 5; ++f) yu[f] = (T)0;
#pragma unroll
  for (int f = 0; f < NF; ++f) fy[f] = qacc[f] = (T)0;
#pragma unroll (RC > 0 ? RC + 2 : 1)
  for (int it = 0; it < (RC > 0 ? RC + 2 : ye + 2); ++it) {
    const int r = Y0 - 1 + it;
    if (RC > 0 && r > Y0 + ye) break;
    const bool inner = it >= 1 && (RC == 0 || it <= RC) && r < Y0 + ye;
    T qc[6];
    if (inner) load(r, qc);
    // slopes, predictor and faces of row r
    T wl[5], wr[5], wv[5], face[3][2][5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      wl[f] = __shfl_up_sync(0xffffffffu, wc[f], 1);
      wr[f] = __shfl_down_sync(0xffffffffu, wc[f], 1);
    }
    cell_faces_g<T, 2, OPT>(
        [&](int f, int dx, int dy, int) -> T {
          return dx < 0 ? wl[f] : (dx > 0 ? wr[f] : (dy < 0 ? wm[f] : (dy > 0 ? wp[f] : wc[f])));
        },
        P, dt2, wv, face);
    // the interface below row r completes row r-1
    if (it >= 1) {
      T fn[NF];
      unsigned e = 0;
      riemann_k<T, NF, 2>(yu, face[1][0], fn, solver, c, e);
      if (owned) err |= e;
      if (it >= 2 && owned) {
        const int64_t idx = (int64_t)(r - 1) * nx + x;
        T qo[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
          qo[f] = axpy_k<kFast>(qacc[f], dtdy, fy[f] - fn[f]);
          A.qout[f * n + idx] = qo[f];
        }
        if (A.cfl_next) {
          T s[3];
          cfl_speeds<T, NF>(qo, P, de, cerr, s);
          if (s[0] > cm[0]) cm[0] = s[0];
          if (s[1] > cm[1]) cm[1] = s[1];
          if (s[2] > cm[2]) cm[2] = s[2];
        }
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) fy[f] = fn[f];
    }
    if (inner) {
      T lo[5], fx[NF];
#pragma unroll
      for (int f = 0; f < 5; ++f) lo[f] = __shfl_up_sync(0xffffffffu, face[0][1][f], 1);
      unsigned e = 0;
      riemann_k<T, NF, 1>(lo, face[0][0], fx, solver, c, e);
      if (lane >= 2 && lane <= 30 && x <= nx) err |= e;
      if (de) {
        T wd[5];
        unsigned e2 = 0;
        prim_k(qc, wd, c, P, de, e2);   // dual-energy resync of q (comp.f90:60-72)
      }
#pragma unroll
      for (int f = 0; f < NF; ++f)
        qacc[f] = axpy_k<kFast>(qc[f], dtdx, fx[f] - __shfl_down_sync(0xffffffffu, fx[f], 1));
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      yu[f] = face[1][1][f];
      wm[f] = wc[f];
      wc[f] = wp[f];
    }
    if (r < Y0 + ye) {   // row r+2; the one after it is loaded while row r+1 is computed
      convert(qn, wp);
      if (r + 1 < Y0 + ye) load(r + 3, qn);
    }
  }
  if (err) atomicOr(&A.ctl->err, err);
}

// A CTA's maxima and errors into its grid's control block (all threads).
template <typename T>
__device__ __forceinline__ void march_maxima(GridCtl* ctl, const T* cm, unsigned cerr, T (*red)[kMarchWarps]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const T m = warp_max_pos(cm[d]);
    if (lane == 0) red[d][wid] = m;
  }
  if (cerr) atomicOr(&ctl->errnext, cerr);
  __syncthreads();
  if (threadIdx.x < 3) {
    T m = red[threadIdx.x][0];
#pragma unroll
    for (int k = 1; k < kMarchWarps; ++k) m = fmax2(m, red[threadIdx.x][k]);
    atomicMax(&ctl->snext[threadIdx.x], ordered_bits((double)m));
  }
}

// OPT: grids with the usual options (minmod, HLLC, second order), as
// constants (1024^2 FP32: 43 -> 33 us).  CTAs per SM: FP32 needs 115 registers,
// so 4; FP64 at 3 (168 registers) or 4 (128, with spills) takes 27 or 30 us at
// 512^2, 78.5 or 77.6 at 1024^2.
template <typename T, int NF, bool OPT, int RC>
__global__ void __launch_bounds__(32 * kMarchWarps, RC > 0 ? 2 : (sizeof(T) == 4 ? 4 : 3)) k_march2d(FusedArgs<T> A) {
  __shared__ T red[3][kMarchWarps];
  T cm[3] = {(T)0, (T)0, (T)0};
  unsigned cerr = 0;
  step_head();
  march2d<T, NF, OPT, RC>(A, blockIdx.x * kMarchWarps + (threadIdx.x >> 5), cm, cerr);
  if (A.cfl_next) march_maxima(A.ctl, cm, cerr, red);
  step_tail(A);
}

}  // namespace EVORA_FNS
}  // namespace evora
