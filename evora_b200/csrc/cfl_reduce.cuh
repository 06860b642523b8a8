// cfl_reduce.cuh -- reductions of the signal speeds |u_d| + a, and the CFL
// maxima of the next step as the epilogue of a physics substep.
#pragma once

#include "hydro_math.cuh"

namespace evora {

// The largest of a non-negative value (no NaN) over a warp, or over red[0..NW)
// for every lane: values >= 0 order like their bits, which one (FP32) or two
// (FP64: high words, then the low words of those that have the largest)
// warp reductions of unsigned words take.
__device__ __forceinline__ float warp_max_pos(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ double warp_max_pos(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return __hiloint2double((int)mh, (int)ml);
}

// The next step's hydrostep maxima (timestep.f90:26-57) from the kernel that
// writes a step's final state, so that the step needs no CFL kernel (a pass
// over the state: 23 to 27 us at 128^3) and one control kernel instead of
// three.  Per cell add(): the state as it is stored (rounded to T), its
// pressure as pressure() gives it (comp.f90:45-85; with dual energy the kin/E
// switch), the speeds in FP64.  FAST: the fast forms (not STRICT grids).
template <typename T, bool FAST>
struct CflEpilogue {
  double m[3] = {0.0, 0.0, 0.0};
  unsigned err = 0;

  // v: q(1:6), S read with dual energy only; pg = rho^(g-1) of the cell
  // (read with dual energy in the fast form)
  __device__ __forceinline__ void add(const double* v, double pg, const HydroParams& P, const Gas<double>& c) {
    double q[6], w[5], a;
#pragma unroll
    for (int f = 0; f < 6; ++f) q[f] = (double)(T)v[f];
    if constexpr (FAST) {
      const double ri = rcp_fast(q[0]);
#pragma unroll
      for (int d = 1; d < 4; ++d) w[d] = q[d] * ri;
      const double kin = 0.5 * sq3(q[1], q[2], q[3]) * ri;
      w[4] = c.g1 * (q[4] - kin);
      if (P.dualenergy && kin * rcp_fast(q[4]) > c.de_thresh1) w[4] = q[5] * pg;
      if (w[4] <= 0.0) err |= EVORA_ERR_PRESSURE;
      a = sqrt_fast(c.g * w[4] * ri);
    } else {
      q2w(q, w, c, P.dualenergy != 0, err);
      a = sqrt(c.g * w[4] / w[0]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double s = fabs(w[d + 1]) + a;
      if (s > m[d]) m[d] = s;
    }
  }

  // One block's maxima into ctl->snext, errors into ctl->errnext (all threads;
  // red: 3 x 32 doubles of shared memory).  A block that raises no maximum
  // leaves the words alone: thousands of blocks share the three.
  __device__ __forceinline__ void finish(GridCtl* ctl, double (*red)[32]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double b = warp_max_pos(m[d]);
      if (lane == 0) red[d][wid] = b;
    }
    if (err) atomicOr(&ctl->errnext, err);
    __syncthreads();
    if (threadIdx.x < 3) {
      double b = 0.0;
      for (int k = 0; k < nw; ++k) b = fmax2(b, red[threadIdx.x][k]);
      if (ordered_bits(b) > __ldcg(&ctl->snext[threadIdx.x])) atomicMax(&ctl->snext[threadIdx.x], ordered_bits(b));
    }
  }
};

}  // namespace evora
