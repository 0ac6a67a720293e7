// One persistent stage kernel for every 2-D arena of an element pool.
//
// A pool keeps the solves of each (physics, p, q) in an arena of its own;
// the plain pool path launches one persistent stage kernel per arena and
// stage.  Here the 2-D arenas (Euler 2-D and shallow water, p = 1..7,
// q = p + 2) share ONE launch per LSRK stage: the kernel walks a device-side
// list of (arena, tile) work items and runs, for each, the fused stage body
// (stage2d_tile, stage2d.cuh) compiled for that arena's (physics, p, q) at a
// common launch shape of 128 threads per CTA.  The body of a work item is a
// CTA-uniform branch, so a launch mixes orders freely; per element the
// arithmetic is that of the body alone (each pencil's operations and their
// order do not depend on the thread count), so a solve's result is the same
// in either path.  Included by one compilation unit per working precision.
#pragma once

#include "dispatch.cuh"

namespace dgmx {

constexpr int kFusedBodies = 14;   // Euler 2-D p = 1..7, shallow water p = 1..7
constexpr int kFusedThreads = 128;
// CTAs per SM the register allocation is held to
constexpr int kFusedMinBlocks64 = 4, kFusedMinBlocksMixed = 5;

// A work item is a tile of an arena, or, in FP32 and in a pool of more tiles
// than the grid has CTAs, two tiles of a solve that follow one another where
// their shared memory leaves the CTAs per SM as they are: a barrier interval
// then has two rounds of modal rows to hide its loads behind (24 solves of 8 to
// 64 elements a side, 40 steps: 27.8 -> 26.0 ms; FP64, with its bodies' spills,
// 42 -> 46).
template <bool MIXED, int B>
struct FusedCfg {
  static constexpr int PHYS = B < 7 ? DGMX_EULER2D : DGMX_SHALLOW;
  static constexpr int P = B % 7 + 1, L = P + 1, Q = P + 2;
  static constexpr int EPB = stage2d_epb(phys_nf(PHYS), L);
  static constexpr bool PAIR =
      MIXED && CfgD<PHYS, L, Q, 2 * EPB, kFusedThreads, 0, MIXED>::SMEM <= 228 * 1024 / kFusedMinBlocksMixed - 1024;
  using C = CfgD<PHYS, L, Q, PAIR ? 2 * EPB : EPB, kFusedThreads, 0, MIXED>;
};

template <bool MIXED, int B = 0>
constexpr size_t fused_smem() {
  if constexpr (B < kFusedBodies) {
    constexpr size_t here = FusedCfg<MIXED, B>::C::SMEM, rest = fused_smem<MIXED, B + 1>();
    return here > rest ? here : rest;
  } else {
    return 0;
  }
}

template <bool MIXED, int B = 0>
__device__ __forceinline__ void fused_dispatch(int body, unsigned char *raw, const StageArgs &a, int item,
                                               int tid) {
  if constexpr (B < kFusedBodies) {
    if (body == B) {
      using F = FusedCfg<MIXED, B>;
      const int e0 = item / 2 * F::EPB, end = e0 + (item % 2 ? 2 : 1) * F::EPB;
      SmemD<typename F::C> sm(raw, end < a.ne ? end : a.ne);
      stage2d_tile<typename F::C, F::PHYS>(sm, a, e0, tid);
    } else {
      fused_dispatch<MIXED, B + 1>(body, raw, a, item, tid);
    }
  }
}

// args: [stage][arena] stage arguments; bodies[arena]: body index;
// items[0 .. *nitems): (arena, 2 tile + (1: and the tile behind it)).
template <bool MIXED>
__global__ void __launch_bounds__(kFusedThreads, MIXED ? kFusedMinBlocksMixed : kFusedMinBlocks64) fused_stage_kernel(const StageArgs *args, int narena,
                                                                       const int *bodies, const int2 *items,
                                                                       const int *nitems, int stage) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_release();
  const int n = *nitems;
  for (int t = blockIdx.x; t < n; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    const int2 it = items[t];
    fused_dispatch<MIXED>(bodies[it.x], smem_raw, args[(size_t)stage * narena + it.x], it.y, threadIdx.x);
  }
}

// Constant tables of every body's (L, Q) in this compilation unit's module
// (the two physics share them).
template <bool MIXED, int B = 0>
static cudaError_t fused_upload() {
  if constexpr (B < 7) {
    using F = FusedCfg<MIXED, B>;
    const Tables1D t = make_tables(F::L, F::Q, F::Q - 1);
    cudaError_t e = upload_tables_lq<F::L, F::Q, typename F::C::R>(t);
    if (e == cudaSuccess) e = upload_tables2_lq<F::L, F::Q, typename F::C::R>(t);
    if (e != cudaSuccess) return e;
    return fused_upload<MIXED, B + 1>();
  } else {
    return cudaSuccess;
  }
}

template <bool MIXED, int B = 0>
constexpr int fused_epb(int body) {
  if constexpr (B < kFusedBodies) return body == B ? FusedCfg<MIXED, B>::EPB : fused_epb<MIXED, B + 1>(body);
  else return 1;
}

template <bool MIXED, int B = 0>
constexpr bool fused_pair(int body) {
  if constexpr (B < kFusedBodies) return body == B ? FusedCfg<MIXED, B>::PAIR : fused_pair<MIXED, B + 1>(body);
  else return false;
}

template <bool MIXED>
struct FusedHost {
  static cudaError_t init() {
    cudaError_t e = fused_upload<MIXED>();
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(fused_stage_kernel<MIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)fused_smem<MIXED>());
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fused_stage_kernel<MIXED>, kFusedThreads,
                                                      fused_smem<MIXED>()) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static cudaError_t launch(const StageArgs *args, int narena, const int *bodies, const int2 *items,
                            const int *nitems, int stage, int grid, cudaStream_t s) {
    return launch_dependent(fused_stage_kernel<MIXED>, (unsigned)grid, kFusedThreads, fused_smem<MIXED>(), s, args,
                            narena, bodies, items, nitems, stage);
  }
};

}  // namespace dgmx
