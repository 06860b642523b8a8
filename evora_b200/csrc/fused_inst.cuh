// fused_inst.cuh -- one arithmetic instantiation of the fused backend: the
// update kernels for NF = 5/6 fields and 1, 2, 3 dimensions, and the CFL
// kernel, compiled with this translation unit's floating-point flags.
// Requires EVORA_FNS (namespace), EVORA_T (state type) and the tile shape
// EVORA_TX, EVORA_TY, EVORA_ZC.
#pragma once

#include <cudaTypedefs.h>

#include <algorithm>

#include "batch_kernel.cuh"
#include "conduction.h"
#include "fused.h"
#include "fused_kernel.cuh"
#include "fused_march.cuh"
#include "fused_tma.cuh"
#if EVORA_PRECISION_F32
#include "fused_pair.cuh"
#endif

namespace evora {
namespace EVORA_FNS {

using TT = EVORA_T;

// Tile table of this precision: (TX, TY, ZC, CTAs per SM, TMA, PIPE).
// TMA = 1: the tensor-staged 3D kernel of fused_tma.cuh (FP32; in FP64 it took
// 3.35 ms per 256^3 launch against 2.11), for grids tiled by whole tiles (the
// plan falls back to entry 0 elsewhere).  PIPE = 1: the two-barrier pipelined
// 3D march of fused_kernel.cuh (FP32; in FP64 it measured no faster than the
// three-barrier march, 2.113 against 2.114 ms per 256^3 launch).  Entry 0 is the
// default for grids the TMA kernel does not take; evora_grid_autotune times
// all entries on the grid itself.  The entries are the 3D kernels'; 1D and 2D
// grids have one kernel each.
template <int I> struct Tile;
#if EVORA_PRECISION_F32
template <> struct Tile<0> { static constexpr int TX = 32, TY = 8, ZC = 32, MINB = 3, TMA = 0, PIPE = 1; };
template <> struct Tile<1> { static constexpr int TX = 16, TY = 16, ZC = 32, MINB = 3, TMA = 0, PIPE = 1; };
template <> struct Tile<2> { static constexpr int TX = 32, TY = 8, ZC = 32, MINB = 2, TMA = 0, PIPE = 1; };
template <> struct Tile<3> { static constexpr int TX = 16, TY = 8, ZC = 32, MINB = 4, TMA = 0, PIPE = 1; };
template <> struct Tile<4> { static constexpr int TX = 32, TY = 8, ZC = 32, MINB = 2, TMA = 1, PIPE = 1; };
// two cells per thread on packed FP32 pairs (fused_pair.cuh)
template <> struct Tile<5> { static constexpr int TX = 32, TY = 8, ZC = 32, MINB = 3, TMA = 2, PIPE = 1; };
constexpr int kTiles = 6;
#else
template <> struct Tile<0> { static constexpr int TX = 16, TY = 8, ZC = 32, MINB = 3, TMA = 0, PIPE = 0; };
template <> struct Tile<1> { static constexpr int TX = 32, TY = 4, ZC = 32, MINB = 3, TMA = 0, PIPE = 0; };
template <> struct Tile<2> { static constexpr int TX = 16, TY = 8, ZC = 16, MINB = 3, TMA = 0, PIPE = 0; };
template <> struct Tile<3> { static constexpr int TX = 16, TY = 8, ZC = 64, MINB = 3, TMA = 0, PIPE = 0; };
template <> struct Tile<4> { static constexpr int TX = 16, TY = 8, ZC = 32, MINB = 2, TMA = 0, PIPE = 0; };
constexpr int kTiles = 5;
#endif

// The shared-memory layout of the k_fused kernel of entry C.
template <class C, int NF>
using TileSmem = FusedSmem<TT, NF, C::TX, C::TY, kSmemDq<TT, C::PIPE != 0>>;

// cuTensorMapEncodeTiled from the driver (no link against libcuda).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// The 4D map (x, y, z, field) of an SoA state q[f][z][y][x] with a box of
// one halo'd plane of all fields, as fused_tma.cuh stages it.
template <int NF, int TX, int TY>
bool encode_state_map(const HydroParams& P, const void* q, CUtensorMap* map) {
  using S = TmaSmem<TT, NF, TX, TY>;
  auto enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)P.nx, (cuuint64_t)P.ny, (cuuint64_t)P.nz, (cuuint64_t)NF};
  const cuuint64_t es = sizeof(TT);
  const cuuint64_t strides[3] = {es * P.nx, es * P.nx * P.ny, es * P.nx * P.ny * P.nz};
  const cuuint32_t box[4] = {(cuuint32_t)S::SX, (cuuint32_t)S::RY, 1, (cuuint32_t)NF};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, sizeof(TT) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                         4, const_cast<void*>(q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Whether the TMA kernel of this shape takes the grid: whole tiles in x and
// y, a 3D grid, 16-byte aligned rows.
template <int TX, int TY>
bool tma_fits(const HydroParams& P, int dim) {
  return dim == 3 && P.nx % TX == 0 && P.ny % TY == 0 && ((size_t)P.nx * sizeof(TT)) % 16 == 0;
}

// Launches a 2D update.  With a step control tail the launch may overlap the
// end of the previous one (step_head), which hides the gap between two
// launches (1024^2 FP64: 78 -> 72 us).  In 3D the same lost: CTAs placed while
// the previous update's last ones still run crowd onto the SMs that are free
// first (100 x 75 x 61 FP32: 90 -> 112 us).
template <class Kernel, class... Args>
void launch_step(const FusedPlan& pl, Kernel k, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = pl.grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = pl.tail ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, args...);   // errors: cudaGetLastError
}

template <int NF, int DIM, int I>
void launch(const FusedPlan& pl, const void* qin, void* qout, GridCtl* ctl, cudaStream_t st) {
  FusedArgs<TT> A{pl.P, (const TT*)qin, (TT*)qout, ctl, pl.n, pl.cfl_fused, pl.zc, pl.tail};
  if constexpr (DIM == 1) {
    k_fused1d<TT, NF><<<pl.grid, pl.threads, 0, st>>>(A);
  } else if constexpr (DIM == 2) {
    const bool opt = pl.P.limiter == 1 && pl.P.solver == 2 && pl.P.secondorder;
    auto k = opt ? k_march2d<TT, NF, true, 0> : k_march2d<TT, NF, false, 0>;
    if (pl.unrolled && pl.zc == 1) k = opt ? k_march2d<TT, NF, true, 1> : k_march2d<TT, NF, false, 1>;
    if (pl.unrolled && pl.zc == 2) k = opt ? k_march2d<TT, NF, true, 2> : k_march2d<TT, NF, false, 2>;
    launch_step(pl, k, pl.threads, 0, st, A);
  } else {
    using C = Tile<I>;
#if EVORA_PRECISION_F32
    if constexpr (C::TMA == 2 && DIM == 3 && NF == 5) {
      CUtensorMap map;
      if (encode_state_map<5, C::TX, C::TY>(pl.P, qin, &map)) {
        k_fused_pair<C::TX, C::TY, C::ZC, C::MINB><<<pl.grid, pl.threads, pl.smem, st>>>(A, map);
        return;
      }
      k_fused<TT, NF, DIM, C::TX, C::TY, C::ZC, 2, C::PIPE != 0>
          <<<pl.grid, C::TX * C::TY, sizeof(TileSmem<C, NF>), st>>>(A);
      return;
    }
#endif
    if constexpr (C::TMA == 1 && DIM == 3) {
      CUtensorMap map;
      if (encode_state_map<NF, C::TX, C::TY>(pl.P, qin, &map)) {
        k_fused_tma<TT, NF, C::TX, C::TY, C::ZC, C::MINB><<<pl.grid, pl.threads, pl.smem, st>>>(A, map);
        return;
      }
      // the map was checked at plan time; should it fail here, the same
      // tile runs without tensor staging
      k_fused<TT, NF, DIM, C::TX, C::TY, C::ZC, C::MINB, C::PIPE != 0>
          <<<pl.grid, pl.threads, sizeof(TileSmem<C, NF>), st>>>(A);
    } else {
      k_fused<TT, NF, DIM, C::TX, C::TY, C::ZC, C::MINB, C::PIPE != 0><<<pl.grid, pl.threads, pl.smem, st>>>(A);
    }
  }
}

template <int NF, int DIM, int I>
FusedLaunch pick_one(int* tx, int* ty, int* zc, size_t* smem, int* threads, int* minb) {
  if constexpr (DIM == 1) {
    *tx = 128; *ty = 1; *zc = 1; *smem = 0; *threads = 128; *minb = 1;
  } else if constexpr (DIM == 2) {
    // the march: warps of kMarchCols columns, zc rows each (set by the plan)
    *tx = kMarchCols; *ty = 1; *zc = 1; *smem = 0; *threads = 32 * kMarchWarps; *minb = 1;
  } else {
    using C = Tile<I>;
    *tx = C::TX; *ty = C::TY; *zc = DIM == 3 ? C::ZC : 1; *minb = C::MINB;
    *smem = sizeof(TileSmem<C, NF>);
    *threads = C::TX * C::TY;
    auto k = k_fused<TT, NF, DIM, C::TX, C::TY, C::ZC, C::TMA == 2 ? 2 : C::MINB, C::PIPE != 0>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
    cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
#if EVORA_PRECISION_F32
    if constexpr (C::TMA == 2 && DIM == 3 && NF == 5) {
      *smem = sizeof(PairSmem<float, C::TX, C::TY>);
      *threads = C::TX / 2 * C::TY;
      auto kp = k_fused_pair<C::TX, C::TY, C::ZC, C::MINB>;
      cudaFuncSetAttribute(kp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
      cudaFuncSetAttribute(kp, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
#endif
    if constexpr (C::TMA == 1 && DIM == 3) {
      *smem = sizeof(TmaSmem<TT, NF, C::TX, C::TY>);
      auto kt = k_fused_tma<TT, NF, C::TX, C::TY, C::ZC, C::MINB>;
      cudaFuncSetAttribute(kt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
      cudaFuncSetAttribute(kt, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
  }
  return &launch<NF, DIM, I>;
}

int tiles() { return kTiles; }

// Whether tile entry `tile` can run this grid (TMA entries need whole tiles
// and an encodable tensor map).
bool tile_fits(const HydroParams& P, int nf, int dim, int tile) {
#if EVORA_PRECISION_F32
  if (tile == 5) {
    using C5 = Tile<5>;
    if (nf != 5 || !pair_config(P) || !tma_fits<C5::TX, C5::TY>(P, dim)) return false;
    CUtensorMap map;
    return encode_state_map<5, C5::TX, C5::TY>(P, reinterpret_cast<const void*>((uintptr_t)1 << 20), &map);
  }
#endif
  using C = Tile<4>;
  if (tile != 4 || C::TMA == 0) return true;
  if (!tma_fits<C::TX, C::TY>(P, dim)) return false;
  // encode against an aligned dummy address: only shapes and strides are checked
  CUtensorMap map;
  const void* fake = reinterpret_cast<const void*>((uintptr_t)1 << 20);
  return nf == 5 ? encode_state_map<5, C::TX, C::TY>(P, fake, &map) : encode_state_map<6, C::TX, C::TY>(P, fake, &map);
}

FusedLaunch pick(int nf, int dim, int tile, int* tx, int* ty, int* zc, size_t* smem, int* threads, int* minb) {
  if (nf == 5 && dim == 3) {
    switch (tile) {
      case 1: return pick_one<5, 3, 1>(tx, ty, zc, smem, threads, minb);
      case 2: return pick_one<5, 3, 2>(tx, ty, zc, smem, threads, minb);
      case 3: return pick_one<5, 3, 3>(tx, ty, zc, smem, threads, minb);
      case 4: return pick_one<5, 3, 4>(tx, ty, zc, smem, threads, minb);
#if EVORA_PRECISION_F32
      case 5: return pick_one<5, 3, 5>(tx, ty, zc, smem, threads, minb);
#endif
      default: return pick_one<5, 3, 0>(tx, ty, zc, smem, threads, minb);
    }
  }
  if (nf == 5) {
    if (dim == 1) return pick_one<5, 1, 0>(tx, ty, zc, smem, threads, minb);
    return pick_one<5, 2, 0>(tx, ty, zc, smem, threads, minb);
  }
  if (dim == 1) return pick_one<6, 1, 0>(tx, ty, zc, smem, threads, minb);
  if (dim == 2) return pick_one<6, 2, 0>(tx, ty, zc, smem, threads, minb);
  switch (tile) {
    case 1: return pick_one<6, 3, 1>(tx, ty, zc, smem, threads, minb);
    case 2: return pick_one<6, 3, 2>(tx, ty, zc, smem, threads, minb);
    case 3: return pick_one<6, 3, 3>(tx, ty, zc, smem, threads, minb);
    case 4: return pick_one<6, 3, 4>(tx, ty, zc, smem, threads, minb);
    default: return pick_one<6, 3, 0>(tx, ty, zc, smem, threads, minb);
  }
}

// ---- multi-grid batches: per step one persistent launch over the tiles of
// the 3D members (the tile program of entry 0) and one over the strips of the
// 2D members (the march), each pulling items from an atomic work queue; every
// grid keeps its own dt, control block and ping-pong parity (MultiGridDesc).
//
// The two launches share no data; the batch runs them in parallel branches of
// its graph, so that one's CTAs start as the other's run out of items.
// 12 grids (3.6 M cells in 2D, 1.1 M in 3D), FP32: 425 -> 219 us per
// step (one launch over tiles of both kinds, 32 planes per 3D item, before).
template <typename Args>
__device__ __forceinline__ void multi_args(Args& A, const MultiGridDesc& d) {
  // the parameters by all threads, word by word
  static_assert(sizeof(HydroParams) % 4 == 0, "copied by words");
  const unsigned* src = reinterpret_cast<const unsigned*>(&d.P);
  unsigned* dst = reinterpret_cast<unsigned*>(&A.P);
  for (int i = threadIdx.x; i < (int)(sizeof(HydroParams) / 4); i += blockDim.x) dst[i] = src[i];
  if (threadIdx.x == 0) {
    A.qin = (const TT*)d.q[d.par];
    A.qout = (TT*)d.q[d.par ^ 1];
    A.ctl = d.ctl;
    A.n = d.n;
    A.cfl_next = 1;
    A.zc = d.zc;
    A.tail = 0;
  }
}

template <int NF>
__global__ void __launch_bounds__(Tile<0>::TX* Tile<0>::TY, Tile<0>::MINB)
    k_multi(const MultiGridDesc* grids, const MultiGridItem* items, int* meta) {
  using C = Tile<0>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<FusedSmem<TT, NF, C::TX, C::TY>*>(smem_raw);
  __shared__ __align__(16) unsigned char a_raw[sizeof(FusedArgs<TT>)];
  __shared__ int s_item;
  auto& A = *reinterpret_cast<FusedArgs<TT>*>(a_raw);
  const int nitems = meta[kMetaItems3];
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&meta[kMetaNext3], 1);
    __syncthreads();
    if (s_item >= nitems) break;
    const MultiGridItem w = items[s_item];
    multi_args(A, grids[w.grid]);
    __syncthreads();
    fused_tile<TT, NF, 3, C::TX, C::TY, C::ZC>(A, sm, threadIdx.x, w.bx, w.by, w.bz);
    __syncthreads();   // the shared state is reused by the next item
  }
}

// A 2D item: kMarchWarps warps of the march from warp bx on.
template <int NF>
__global__ void __launch_bounds__(32 * kMarchWarps, sizeof(TT) == 4 ? 4 : 3)
    k_multi2d(const MultiGridDesc* grids, const MultiGridItem* items, int* meta) {
  __shared__ __align__(16) unsigned char a_raw[sizeof(FusedArgs<TT>)];
  __shared__ TT red[3][kMarchWarps];
  __shared__ int s_item;
  auto& A = *reinterpret_cast<FusedArgs<TT>*>(a_raw);
  const int nitems = meta[kMetaItems2];
  items += meta[kMetaItems3];
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&meta[kMetaNext2], 1);
    __syncthreads();
    if (s_item >= nitems) break;
    const MultiGridItem w = items[s_item];
    multi_args(A, grids[w.grid]);
    __syncthreads();
    TT cm[3] = {(TT)0, (TT)0, (TT)0};
    unsigned cerr = 0;
    const int gw = w.bx + (int)(threadIdx.x >> 5);
    if (A.P.limiter == 1 && A.P.solver == 2 && A.P.secondorder) march2d<TT, NF, true>(A, gw, cm, cerr);
    else march2d<TT, NF, false>(A, gw, cm, cerr);
    march_maxima(A.ctl, cm, cerr, red);
    __syncthreads();   // the shared state is reused by the next item
  }
}

template <int NF>
void multi_launch(const MultiGridDesc* grids, const MultiGridItem* items, int* meta, bool has3, bool has2, int sms,
                  cudaStream_t st3, cudaStream_t st2) {
  using C = Tile<0>;
  if (has3)
    k_multi<NF><<<sms * C::MINB, C::TX * C::TY, sizeof(FusedSmem<TT, NF, C::TX, C::TY>), st3>>>(grids, items, meta);
  if (has2)
    k_multi2d<NF><<<sms * (sizeof(TT) == 4 ? 4 : 3), 32 * kMarchWarps, 0, st2>>>(grids, items, meta);
}

MultiLaunch multi_pick(int nf, MultiShape* s) {
  using C = Tile<0>;
  s->tx = C::TX;
  s->ty = C::TY;
  s->ctas_per_sm = C::MINB;
  s->cols2 = kMarchCols;
  s->warps2 = kMarchWarps;
  if (nf == 5) {
    cudaFuncSetAttribute(k_multi<5>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(FusedSmem<TT, 5, C::TX, C::TY>));
    cudaFuncSetAttribute(k_multi<5>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    return &multi_launch<5>;
  }
  cudaFuncSetAttribute(k_multi<6>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(FusedSmem<TT, 6, C::TX, C::TY>));
  cudaFuncSetAttribute(k_multi<6>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  return &multi_launch<6>;
}

// hydrostep part 1 on the SoA state: maxima of |u_d| + a (per cell in the
// working precision, cfl_speeds; maxima and dt in FP64).
template <int NF>
__global__ void k_cfl_soa(HydroParams P, const TT* __restrict__ q, int64_t n, GridCtl* ctl) {
  if (ctl_skip(ctl)) return;
  double m0 = 0.0, m1 = 0.0, m2 = 0.0, vmin = 1e99;
  unsigned err = 0;
  const Units U = units_of(P, ctl);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    TT qv[6], s[3];
#pragma unroll
    for (int f = 0; f < NF; ++f) qv[f] = __ldg(q + f * n + i);
    cfl_speeds<TT, NF>(qv, P, P.dualenergy != 0, err, s);
    const double s0 = s[0], s1 = s[1], s2 = s[2];
    if (s0 > m0) m0 = s0;
    if (s1 > m1) m1 = s1;
    if (s2 > m2) m2 = s2;
    if (P.conduction) {
      // thermalstep (timestep.f90:84-93): min over cells of rho / kappa
      double qd[6], w[5];
#pragma unroll
      for (int f = 0; f < NF; ++f) qd[f] = (double)qv[f];
      q2w(qd, w, Gas<double>::make(P), P.dualenergy != 0, err);
      const double v = kFast ? thermal_v_fast(U, w[0], w[4]) : thermal_v(U, w[0], w[4]);
      if (v < vmin) vmin = v;
    }
  }
  if (P.conduction) {
    for (int off = 16; off > 0; off >>= 1) vmin = fmin2(vmin, __shfl_xor_sync(0xffffffffu, vmin, off));
    if ((threadIdx.x & 31) == 0) atomicMin(&ctl->vcond, ordered_bits(vmin));
  }
  for (int off = 16; off > 0; off >>= 1) {
    m0 = fmax2(m0, __shfl_xor_sync(0xffffffffu, m0, off));
    m1 = fmax2(m1, __shfl_xor_sync(0xffffffffu, m1, off));
    m2 = fmax2(m2, __shfl_xor_sync(0xffffffffu, m2, off));
  }
  __shared__ double red[3][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) { red[0][wid] = m0; red[1][wid] = m1; red[2][wid] = m2; }
  __syncthreads();
  if (wid == 0) {
    m0 = lane < nw ? red[0][lane] : 0.0;
    m1 = lane < nw ? red[1][lane] : 0.0;
    m2 = lane < nw ? red[2][lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) {
      m0 = fmax2(m0, __shfl_xor_sync(0xffffffffu, m0, off));
      m1 = fmax2(m1, __shfl_xor_sync(0xffffffffu, m1, off));
      m2 = fmax2(m2, __shfl_xor_sync(0xffffffffu, m2, off));
    }
    if (lane == 0) {
      atomicMax(&ctl->smax[0], ordered_bits(m0));
      atomicMax(&ctl->smax[1], ordered_bits(m1));
      atomicMax(&ctl->smax[2], ordered_bits(m2));
    }
  }
  if (err) atomicOr(&ctl->err, err);
}

void cfl(const FusedPlan& pl, const void* q, GridCtl* ctl, cudaStream_t st) {
  int64_t blocks = (pl.n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (pl.nf == 5) k_cfl_soa<5><<<(int)blocks, 256, 0, st>>>(pl.P, (const TT*)q, pl.n, ctl);
  else k_cfl_soa<6><<<(int)blocks, 256, 0, st>>>(pl.P, (const TT*)q, pl.n, ctl);
}

// ---- dynamic shared memory of the kernels below
// A launch is refused when it asks for more than its kernel's limit, and the
// limit belongs to the kernel, not to a plan: batches, servers and grids of
// other lengths share it, in other threads too.  So it is always the most that
// the device gives (its opt-in size less the kernel's static memory), set once
// by each plan and never to a plan's own size.
template <class Kernel>
void allow_smem(Kernel k) {
  int dev = 0, most = 0;
  cudaFuncAttributes a;
  if (cudaGetDevice(&dev) == cudaSuccess && cudaFuncGetAttributes(&a, k) == cudaSuccess &&
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess)
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
  cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  cudaGetLastError();
}

// ---- 1D grids: several steps in one launch
constexpr size_t kSteps1dSmem = 220 * 1024;   // + 6 KB static: within allow_smem's limit
size_t steps1d_smem(int nf, int m) { return ((size_t)10 * (m + 4) + (size_t)nf * m) * sizeof(TT); }

template <int NF, int NT>
void steps1d_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int ranks, size_t smem, cudaStream_t st) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(ranks);
  cfg->blockDim = dim3(NT);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = ranks;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

template <int NF, int NT>
void steps1d_launch(const FusedPlan& pl, void* q, GridCtl* ctl, int nsteps, int m, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  steps1d_config<NF, NT>(&cfg, &at, pl.ranks1d, steps1d_smem(NF, m), st);
  cudaLaunchKernelEx(&cfg, k_steps1d<TT, NF, NT>, pl.P, (TT*)q, ctl, nsteps, m);   // errors: cudaGetLastError
}

template <int NF>
void steps1d_allow() {
  allow_smem(k_steps1d<TT, NF, 256>);
  allow_smem(k_steps1d<TT, NF, 512>);
  cudaFuncSetAttribute(k_steps1d<TT, NF, 512>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

template <int NF>
bool steps1d_wide(int m) {   // whether this device schedules clusters of 16 such CTAs
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  steps1d_allow<NF>();
  steps1d_config<NF, 512>(&cfg, &at, 16, steps1d_smem(NF, m), nullptr);
  int count = 0;
  const bool ok = cudaOccupancyMaxActiveClusters(&count, k_steps1d<TT, NF, 512>, &cfg) == cudaSuccess;
  cudaGetLastError();
  return ok && count > 0;
}

// Ranks of the cluster that k_steps1d runs a 1D grid with, 0 if the grid
// does not fit one.  us per step, FP64 / FP32, by ranks:
//      cells        1            2            4            8           16
//         64  1.73 / 1.34  1.78 / 1.42  1.85 / 1.46  1.97 / 1.57  2.25 / 1.85
//        200  2.01 / 1.49  1.80 / 1.42  1.84 / 1.44  1.96 / 1.59  2.24 / 1.82
//        400  2.78 / 1.84  2.07 / 1.55  1.82 / 1.46  1.99 / 1.59  2.26 / 1.84
//       1024  5.24 / 2.93  3.49 / 2.18  2.39 / 1.76  2.18 / 1.64  2.23 / 1.74
//       8000   - / -        - / -        - / 4.63    5.51 / 3.21  4.55 / 3.43
//      23000   - / -        - / -        - / -        - / 6.00    7.25 / 4.59
// against 9 to 13 with separate kernels.  The smallest count within 5 % of
// the best up to 8, the largest portable cluster; 16, where the device has
// room for it, once a rank of 8 would hold more than 1000 (FP64) or 2000
// (FP32) cells.
int steps1d_plan(const FusedPlan& pl) {
  if (pl.dim != 1) return 0;
  auto per_rank = [&](int r) { return (int)((pl.n + r - 1) / r); };
  auto fits = [&](int r) {
    const int m = per_rank(r);
    return pl.n - (int64_t)(r - 1) * m >= 2 && steps1d_smem(pl.nf, m) <= kSteps1dSmem;
  };
  int r = pl.n <= 96 ? 1 : (pl.n <= 300 ? 2 : (pl.n <= 700 ? 4 : 8));
  if (per_rank(8) > (sizeof(TT) == 8 ? 1000 : 2000) && fits(16) &&
      (pl.nf == 5 ? steps1d_wide<5>(per_rank(16)) : steps1d_wide<6>(per_rank(16))))
    return 16;
  return fits(r) ? r : 0;
}

void steps1d(FusedPlan& pl, void* q, GridCtl* ctl, int nsteps, cudaStream_t st) {
  if (!pl.allowed1d) {   // at a grid's first step: it loads the kernels (15 ms the first time)
    if (pl.nf == 5) steps1d_allow<5>();
    else steps1d_allow<6>();
    pl.allowed1d = true;
  }
  // warps for one round of 30 cells each, as far as 16 of them go
  const int m = (int)((pl.n + pl.ranks1d - 1) / pl.ranks1d);
  if (pl.nf == 5) {
    if (m <= 240) steps1d_launch<5, 256>(pl, q, ctl, nsteps, m, st);
    else steps1d_launch<5, 512>(pl, q, ctl, nsteps, m, st);
  } else {
    if (m <= 240) steps1d_launch<6, 256>(pl, q, ctl, nsteps, m, st);
    else steps1d_launch<6, 512>(pl, q, ctl, nsteps, m, st);
  }
}

// ---- batched tubes
BatchArgs<TT> batch_args(const BatchPlan& pl, void* q) {
  BatchArgs<TT> A;
  A.P = pl.P;
  A.xmin = pl.xmin;
  A.xmax = pl.xmax;
  A.q = (TT*)q;
  A.ntot = pl.ntot;
  A.tubes = pl.tubes;
  A.order = pl.order;
  A.ntubes = pl.ntubes;
  A.head = pl.head;
  A.budget = pl.budget;
  A.quantum = pl.quantum;
  A.steps_per_cell = pl.steps_per_cell;
  A.cap = pl.cap;
  A.capw = pl.capw;
  A.gscratch = (TT*)pl.gscratch;
  A.nmax = pl.nmax;
  A.cell_updates = pl.cell_updates;
  return A;
}

template <int NF, int NT>
void batch_launch(const BatchPlan& pl, void* q, cudaStream_t st) {
  k_tubes<TT, NF, NT><<<pl.ctas, NT, pl.smem, st>>>(batch_args(pl, q));
}

// Cells per rank of the longest tube, as k_tubes_cluster splits it (at most).
int cluster_cells(int nmax, int ranks) { return std::max(64, (nmax + ranks - 1) / ranks) + 1; }

// Estimated us per step of a tube of n cells by a CTA, and by ranks of m cells.
double cta_us(int n) {
  return sizeof(TT) == 4 ? std::max(n <= 120 ? 1.1 : 1.75, 0.95 + 1.9e-3 * n)
                         : std::max(n <= 120 ? 1.4 : 2.3, 1.2 + 3.75e-3 * n);
}
double cluster_us(int m) { return sizeof(TT) == 4 ? 1.75 + 1.78e-3 * m : 1.9 + 3.5e-3 * m; }

// CTAs per tube (k_tubes_cluster, 512 threads each): 2, 4 or 8, or 0 for a CTA
// per tube (k_tubes), by the shortest estimated time of the launch.
// pl.clusters has the clusters of each size that run at once (74, 33 and 15 of
// 2, 4 and 8 CTAs: one CTA fits an SM, and the SMs of a GPC that do not make up
// a whole cluster stay idle); more tubes than that wait for one another, so the
// queue is played through: each tube goes to the cluster that is free first.
// n, steps: the running tubes' lengths and steps in the launch (their relation
// is enough), in queue order.
// us per step of equal tubes, measured, FP32 / FP64:
//     cells       CTA          2            4            8 CTAs, all at once
//        60   1.1 / 1.4    1.8 / 2.0    1.8 / 2.0    1.8 / 2.1
//       150   1.8 / 2.3    1.8 / 2.0    1.8 / 2.0    1.8 / 2.1
//       500   1.9 / 3.1    2.0 / 2.5    1.9 / 2.3    1.9 / 2.2
//      1000   2.9 / 5.0    2.5 / 3.5    2.0 / 2.6    2.0 / 2.5
//      2500   5.8 / 10.5   3.8 / 6.1    2.8 / 4.1    2.2 / 2.8
//      8000  20.2 / 36.6    - / -       5.2 / -      3.7 / 5.6
// and twice or three times that in two or three turns.  With every tube a
// cluster up to two CTAs per SM, the rule before, 148 FP32 tubes of 1000 cells
// took 4.9 (now 2.9), 37 of 2500 6.5 (3.8), 24 of 60 3.5 (1.1).
template <int NF>
int cluster_ranks(const BatchPlan& pl, const int* n, const double* steps, int running, int sms) {
  if (running < 1 || running > sms) return 0;   // not even a CTA per tube at once: measured with fewer
  double best = 0.0;
  int nmax = 0, ranks = 0;
  for (int i = 0; i < running; ++i) {
    best = std::max(best, steps[i] * cta_us(n[i]));
    nmax = std::max(nmax, n[i]);
  }
  for (int e = 1; e <= 3; ++e) {
    double busy[128] = {};   // until when each cluster is
    const int at_once = std::min(pl.clusters[e], 128);
    if (at_once < 1 || steps1d_smem(NF, cluster_cells(nmax, 1 << e)) > kSteps1dSmem) continue;
    for (int i = 0; i < running; ++i)
      *std::min_element(busy, busy + at_once) += steps[i] * cluster_us(cluster_cells(n[i], 1 << e));
    const double t = *std::max_element(busy, busy + at_once);
    if (t < best) {
      best = t;
      ranks = 1 << e;
    }
  }
  return ranks;
}

template <int NF>
void cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int tubes, int ranks, size_t smem,
                    cudaStream_t st) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(tubes * ranks);
  cfg->blockDim = dim3(512);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = ranks;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// The clusters that run at once, with the most shared memory a launch asks
// for.  A batch of more tubes than SMs never asks; loading the kernel for it
// would cost its first creation some 5 ms.
template <int NF>
void cluster_plan(BatchPlan* pl) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (pl->ntubes > sms) return;
  allow_smem(k_tubes_cluster<TT, NF, 512>);
  for (int i = 1; i <= 3; ++i) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config<NF>(&cfg, &at, 1, 1 << i, kSteps1dSmem, nullptr);
    int count = 0;
    if (cudaOccupancyMaxActiveClusters(&count, k_tubes_cluster<TT, NF, 512>, &cfg) != cudaSuccess) count = 0;
    pl->clusters[i] = count;
  }
  cudaGetLastError();
}

template <int NF>
void cluster_launch(const BatchPlan& pl, void* q, int running, int nmax, int ranks, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  cluster_config<NF>(&cfg, &at, running, ranks, steps1d_smem(NF, cluster_cells(nmax, ranks)), st);
  cudaLaunchKernelEx(&cfg, k_tubes_cluster<TT, NF, 512>, batch_args(pl, q));   // errors: cudaGetLastError
}

int batch_cluster_ranks(const BatchPlan& pl, const int* n, const double* steps, int running, int sms) {
  return pl.nf == 5 ? cluster_ranks<5>(pl, n, steps, running, sms) : cluster_ranks<6>(pl, n, steps, running, sms);
}

void batch_cluster(const BatchPlan& pl, void* q, int running, int nmax, int ranks, cudaStream_t st) {
  if (pl.nf == 5) cluster_launch<5>(pl, q, running, nmax, ranks, st);
  else cluster_launch<6>(pl, q, running, nmax, ranks, st);
}

template <int NF, int NT>
BatchLaunch batch_pick_one(BatchPlan* pl) {
  pl->threads = NT;
  pl->smem = ((size_t)NF * pl->cap + 5 * ((size_t)pl->cap + 4)) * sizeof(TT);
  pl->capw = std::max(pl->cap, (int)(pl->smem / (5 * sizeof(TT))) - 4);
  allow_smem(k_tubes<TT, NF, NT>);
  cluster_plan<NF>(pl);
  return &batch_launch<NF, NT>;
}

BatchLaunch batch_pick(int nf, int threads, BatchPlan* pl) {
  if (nf == 5) {
    if (threads == 128) return batch_pick_one<5, 128>(pl);
    if (threads == 512) return batch_pick_one<5, 512>(pl);
    if (threads == 768) return batch_pick_one<5, 768>(pl);
    return batch_pick_one<5, 256>(pl);
  }
  if (threads == 128) return batch_pick_one<6, 128>(pl);
  if (threads == 512) return batch_pick_one<6, 512>(pl);
  return batch_pick_one<6, 256>(pl);
}

template <int NF, int NT>
int max_ctas_one(size_t smem) {
  int nb = 0;
  allow_smem(k_tubes<TT, NF, NT>);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_tubes<TT, NF, NT>, NT, smem);
  return nb;
}

int batch_max_ctas_per_sm(int nf, int threads, size_t smem) {
  if (nf == 5) {
    if (threads == 128) return max_ctas_one<5, 128>(smem);
    if (threads == 512) return max_ctas_one<5, 512>(smem);
    if (threads == 768) return max_ctas_one<5, 768>(smem);
    return max_ctas_one<5, 256>(smem);
  }
  if (threads == 128) return max_ctas_one<6, 128>(smem);
  if (threads == 512) return max_ctas_one<6, 512>(smem);
  return max_ctas_one<6, 256>(smem);
}

}  // namespace EVORA_FNS
}  // namespace evora
