// Launchers for one kernel instantiation and the registry hook used by the
// per-physics compilation units (k_*.cu).
#pragma once

#include "ns.cuh"
#include "pipeline.cuh"
#include "form3.cuh"
#include "stage2.cuh"
#include "stage2d.cuh"

namespace dgmx {

// Launch of a kernel that calls pdl_wait (kernels.cuh), allowed to start
// before the kernel ahead of it on the stream has drained.
template <class... P>
inline cudaError_t launch_dependent(void (*k)(P...), unsigned grid, int nt, size_t smem, cudaStream_t s,
                                    const P &...a) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3((unsigned)nt);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, a...);
}

// Every k_*.cu is its own device module with its own copy of the __constant__
// tables, whose host shadows have internal linkage.  The uploader must have
// internal linkage too: an ordinary (weak) template instantiation would be
// merged across compilation units by the linker and write only one module's
// tables.
template <int L, int Q, class T>
static cudaError_t upload_tables_lq(const Tables1D &t) {
  auto put = [](const auto &sym, const std::vector<double> &v, size_t n) {
    std::vector<T> c(n);
    for (size_t i = 0; i < n; ++i) c[i] = T(v[i]);
    return cudaMemcpyToSymbol(sym, c.data(), sizeof(T) * n);
  };
  cudaError_t e;
  if ((e = put(cB<T, L, Q>, t.B, (size_t)L * Q)) != cudaSuccess) return e;
  if ((e = put(cBg<T, L, Q>, t.Bg, (size_t)L * (Q - 1))) != cudaSuccess) return e;
  if ((e = put(cD<T, L, Q>, t.D, (size_t)Q * Q)) != cudaSuccess) return e;
  if ((e = put(cG2GL<T, L, Q>, t.g2gl, (size_t)Q * (Q - 1))) != cudaSuccess) return e;
  if ((e = put(cGL2G<T, L, Q>, t.gl2g, (size_t)(Q - 1) * Q)) != cudaSuccess) return e;
  if ((e = put(cW<T, L, Q>, t.w, (size_t)Q)) != cudaSuccess) return e;
  std::vector<double> end(2 * L);
  for (int a = 0; a < L; ++a) { end[a] = t.B[a * Q + 0]; end[L + a] = t.B[a * Q + Q - 1]; }
  if ((e = put(cEnd<T, L, Q>, end, (size_t)2 * L)) != cudaSuccess) return e;
  // projection with the GLL weights folded in, and lift with 1/w_end folded in
  std::vector<double> bw((size_t)L * Q), gw((size_t)2 * Q * (Q - 1));
  for (int a = 0; a < L; ++a)
    for (int i = 0; i < Q; ++i) bw[(size_t)a * Q + i] = t.B[(size_t)a * Q + i] * t.w[i];
  for (int end_ = 0; end_ < 2; ++end_)
    for (size_t k = 0; k < (size_t)Q * (Q - 1); ++k) gw[end_ * Q * (Q - 1) + k] = t.g2gl[k] / t.w[end_ ? Q - 1 : 0];
  if ((e = put(cBw<T, L, Q>, bw, (size_t)L * Q)) != cudaSuccess) return e;
  return put(cG2GLw<T, L, Q>, gw, (size_t)2 * Q * (Q - 1));
}

// Tables of the second-form stage kernel (only its compilation unit
// instantiates them: constant memory is 64 KB per module): the weighted
// derivative E = B W D and the lift-projection BwG = B W G2GL (L rows each).
template <int L, int Q, class T>
static cudaError_t upload_tables2_lq(const Tables1D &t) {
  std::vector<T> e2((size_t)L * Q), bwg((size_t)L * (Q - 1));
  for (int a = 0; a < L; ++a) {
    for (int j = 0; j < Q; ++j) {
      double acc = 0.0;
      for (int i = 0; i < Q; ++i) acc += t.B[(size_t)a * Q + i] * t.w[i] * t.D[(size_t)i * Q + j];
      e2[(size_t)a * Q + j] = T(acc);
    }
    for (int g = 0; g < Q - 1; ++g) {
      double acc = 0.0;
      for (int i = 0; i < Q; ++i) acc += t.B[(size_t)a * Q + i] * t.w[i] * t.g2gl[(size_t)i * (Q - 1) + g];
      bwg[(size_t)a * (Q - 1) + g] = T(acc);
    }
  }
  cudaError_t e = cudaMemcpyToSymbol(cE2<T, L, Q>, e2.data(), sizeof(T) * e2.size());
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(cBwG<T, L, Q>, bwg.data(), sizeof(T) * bwg.size());
}

// Whether CV::MINB CTAs of the FP32 viscous kernels' tile CV fit one SM's
// shared memory (3-D Navier-Stokes only: other physics have no such kernels).
template <bool NS, class CV>
struct ViscPairFits {
  static constexpr bool value = false;
};
template <class CV>
struct ViscPairFits<true, CV> {
  static constexpr bool value = CV::MINB * (NsCfg<CV, float>::Grad::SMEM + 1024) <= 228 * 1024 &&
                                CV::MINB * (NsCfg<CV, float>::Visc::SMEM + 1024) <= 228 * 1024;
};

template <int PHYS, int L, int Q, int EPB, int MINB, bool MIXED = false, int NT_ = 0>
struct Launch {
  using C = Cfg<PHYS, L, Q, EPB, MINB, MIXED, NT_>;
  // The separate viscous kernels serve the 3xTF32 form of 3-D Navier-Stokes
  // at p >= 5 (1-D operators of at least 7 x 7).
  static constexpr bool kVisc32 = PHYS == DGMX_NS3D && L >= 6 && !MIXED && MINB == 0;
  // Their tile.  Above 512 quadrature points one thread
  // per point (and its registers) leaves one CTA per SM, whose barriers then
  // idle the SM; 256 threads (about three points each) and four CTAs per SM
  // (the traces read from global memory and the lean viscous layout,
  // NsCfg::Grad::TRG and NsCfg::Visc::LEAN, ~50 KB each) let CTAs' barrier
  // waits overlap the others' work (p = 7, q = 9: 15 % faster than 384 x 3).
  using CV2 = Cfg<PHYS, L, Q, EPB, 4, MIXED, 256>;
  static constexpr bool kViscPair = C::QD > 512 && EPB == 1 && ViscPairFits<PHYS == DGMX_NS3D && !MIXED, CV2>::value;
  using CV = std::conditional_t<kViscPair, CV2, C>;
  static dim3 grid(int ne) { return dim3((unsigned)((ne + EPB - 1) / EPB)); }
  static dim3 vgrid(const StageArgs &a) { return a.vtiles ? dim3((unsigned)a.nvtiles) : grid(a.ne); }
  // tables, projections and trace kernels (all that another form's tile of
  // the same (L, Q) takes from this one)
  static cudaError_t init_aux(const Tables1D &t) {
    cudaError_t e = upload_tables_lq<L, Q, typename C::R>(t);
    if (e != cudaSuccess) return e;
    const int sm = (int)C::SMEM;
    if ((e = cudaFuncSetAttribute(traces_modal_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
    if constexpr (!MIXED) {
      if ((e = cudaFuncSetAttribute(traces_nodal_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
      if ((e = cudaFuncSetAttribute(forward_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
      if ((e = cudaFuncSetAttribute(backward_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
    }
    return cudaSuccess;
  }
  static KernelOps aux() {
    KernelOps o;
    o.traces_modal = traces_modal; o.traces_nodal = traces_nodal; o.forward = forward; o.backward = backward;
    return o;
  }
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = init_aux(t);
    if (e != cudaSuccess) return e;
    const int sm = (int)C::SMEM;
    if ((e = cudaFuncSetAttribute(stage_kernel<C, PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
    if constexpr (!MIXED)
      if ((e = cudaFuncSetAttribute(rhs_nodal_kernel<C, PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm))) return e;
    if constexpr (kVisc32) {
      // the 3xTF32 viscous kernels and their FP32 tables
      using N = NsCfg<CV, float>;
      if ((e = upload_tables_lq<L, Q, float>(t)) != cudaSuccess) return e;
      const int sg = (int)N::Grad::SMEM, sv = (int)N::Visc::SMEM;
      if ((e = cudaFuncSetAttribute(ns_grad_kernel<CV, PHYS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sg))) return e;
      if ((e = cudaFuncSetAttribute(ns_grad_kernel<CV, PHYS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sg))) return e;
      if ((e = cudaFuncSetAttribute(ns_visc_kernel<CV, PHYS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sv))) return e;
      if ((e = cudaFuncSetAttribute(ns_visc_kernel<CV, PHYS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sv))) return e;
    }
    return cudaSuccess;
  }
  static cudaError_t ns_grad32(const StageArgs &a, bool nodal, cudaStream_t s) {
    if constexpr (kVisc32) {
      using N = NsCfg<CV, float>;
      if (nodal) ns_grad_kernel<CV, PHYS, true><<<grid(a.ne), CV::NT, N::Grad::SMEM, s>>>(a);
      else ns_grad_kernel<CV, PHYS, false><<<grid(a.ne), CV::NT, N::Grad::SMEM, s>>>(a);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t ns_visc32(const StageArgs &a, bool nodal, cudaStream_t s) {
    if constexpr (kVisc32) {
      using N = NsCfg<CV, float>;
      if (nodal) ns_visc_kernel<CV, PHYS, true><<<vgrid(a), CV::NT, N::Visc::SMEM, s>>>(a);
      else ns_visc_kernel<CV, PHYS, false><<<vgrid(a), CV::NT, N::Visc::SMEM, s>>>(a);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) {
    stage_kernel<C, PHYS><<<grid(a.ne), C::NT, C::SMEM, s>>>(a);
    return cudaGetLastError();
  }
  static cudaError_t traces_modal(const StageArgs &a, const double *X, void *T, cudaStream_t s) {
    traces_modal_kernel<C><<<grid(a.ne), C::NT, C::SMEM, s>>>(a, X, static_cast<typename C::R *>(T));
    return cudaGetLastError();
  }
  static cudaError_t traces_nodal(const StageArgs &a, cudaStream_t s) {
    if constexpr (!MIXED) {
      traces_nodal_kernel<C><<<grid(a.ne), C::NT, C::SMEM, s>>>(a);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    if constexpr (!MIXED) {
      rhs_nodal_kernel<C, PHYS><<<grid(a.ne), C::NT, C::SMEM, s>>>(a);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t forward(const StageArgs &a, const double *Un, double *Um, cudaStream_t s) {
    if constexpr (!MIXED) {
      forward_kernel<C><<<grid(a.ne), C::NT, C::SMEM, s>>>(a, Un, Um);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t backward(const StageArgs &a, const double *Um, double *Un, cudaStream_t s) {
    if constexpr (!MIXED) {
      backward_kernel<C><<<grid(a.ne), C::NT, C::SMEM, s>>>(a, Um, Un);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    stage_kernel<C, PHYS><<<g, C::NT, C::SMEM, s>>>(a);
    return cudaGetLastError();
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage_kernel<C, PHYS>, C::NT, C::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static KernelOps ops() {
    KernelOps o;
    o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.epb = EPB; o.nt = C::NT; o.smem = C::SMEM; o.minb = MINB; o.mixed = MIXED;
    o.init = init; o.stage = stage; o.traces_modal = traces_modal; o.traces_nodal = traces_nodal;
    o.rhs_nodal = rhs_nodal; o.forward = forward; o.backward = backward;
    if constexpr (kVisc32) { o.ns_grad32 = ns_grad32; o.ns_visc32 = ns_visc32; }
    return o;
  }
};

// Elements per CTA: pack small elements so a CTA has >= ~128 threads.
constexpr int default_epb(int dim, int Q) {
  return dim == 3 ? (Q * Q * Q >= 100 ? 1 : (Q * Q * Q >= 50 ? 2 : 4))
                  : (Q * Q >= 100 ? 1 : (128 / (Q * Q) > 8 ? 8 : 128 / (Q * Q)));
}


// Streaming multiprocessors of the current device (cached per device).
inline int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return sm_count(0);
  if (!cached[dev]) cached[dev] = sm_count(dev);
  return cached[dev];
}

// The persistent pipelined stage kernel (stage_pipe_kernel) for LSRK and
// right-hand-side stages; other stage kinds run the plain kernel of the
// same tile.
template <int PHYS, int L, int Q, int EPB, int MINB, bool MIXED = false>
struct PLaunch {
  using Base = Launch<PHYS, L, Q, EPB, MINB, MIXED>;
  using C = typename Base::C;
  using P = Pipe<C>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init(t);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(stage_pipe_kernel<C, PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)P::SMEM);
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage_pipe_kernel<C, PHYS>, C::NT, P::SMEM) !=
        cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    if (a.kind != kLSRK && a.kind != kRHS) return Base::stage(a, s);
    stage_pipe_kernel<C, PHYS><<<g, C::NT, P::SMEM, s>>>(a);
    return cudaGetLastError();
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) {
    static int bps = 0;
    if (!bps) bps = blocks_per_sm();
    const int tiles = (a.ne + EPB - 1) / EPB;
    const int g = tiles < sm_count() * bps ? tiles : sm_count() * bps;
    return stage_grid(a, g, s);
  }
  static KernelOps ops() {
    KernelOps o = Base::ops();
    o.smem = P::SMEM; o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.warp = 2;
    return o;
  }
};

// Threads of a third-form tile: about one per modal row, 64 to 256.
constexpr int form3_threads(int L) {
  const int t = (5 * L * L + 31) / 32 * 32;
  return t < 64 ? 64 : (t > 256 ? 256 : t);
}
// CTAs per SM that smem bytes and a cap of r registers per thread allow.
constexpr int form3_blocks(size_t smem, int nt, int r) {
  const int per_part = 16384 / (32 * r), by_regs = per_part * 4 / ((nt + 31) / 32);
  const int by_smem = (int)((228 * 1024) / (smem + 1024));
  const int b = by_regs < by_smem ? by_regs : by_smem;
  return b < 1 ? 1 : b;
}

// Euler 3-D in the third form: every stage kind, boundary sides and the
// right-hand side on GLL values.  The projections and trace kernels come from
// the plain tile.
template <int PHYS, int L, int Q, bool MIXED, int NT = form3_threads(L), int REGS = MIXED ? 72 : 112>
struct Launch3 {
  using Base = Launch<PHYS, L, Q, default_epb(3, Q), 0, MIXED>;
  using C0 = Cfg3<PHYS, L, Q, NT, 0, MIXED>;
  using C = Cfg3<PHYS, L, Q, NT, form3_blocks(Stage3<C0>::SMEM, NT, REGS), MIXED>;
  using N = Stage3<C>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init_aux(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, typename C::R>(t);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(stage3_kernel<C, PHYS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)N::SMEM);
    if constexpr (!MIXED)
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(stage3_kernel<C, PHYS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)N::SMEM);
    return e;
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    return launch_dependent(stage3_kernel<C, PHYS, false>, (unsigned)g, NT, N::SMEM, s, a);
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) { return stage_grid(a, a.ne, s); }
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    if constexpr (!MIXED) {
      return launch_dependent(stage3_kernel<C, PHYS, true>, (unsigned)a.ne, NT, N::SMEM, s, a);
    } else {
      return cudaErrorNotSupported;
    }
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage3_kernel<C, PHYS, false>, NT, N::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static KernelOps ops() {
    KernelOps o = Base::aux();
    o.epb = 1; o.nt = NT; o.minb = C::MINB; o.smem = N::SMEM; o.preferred = 1; o.mixed = MIXED;
    o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.rhs_nodal = rhs_nodal;
    return o;
  }
};
template <int PHYS, int P, int Q, bool MIXED = false>
void reg3() {
  const int key = PHYS + (MIXED ? kMixedKey : 0);
  constexpr int NT = form3_threads(P + 1);
  register_ops(key, P + 1, Q, Launch3<PHYS, P + 1, Q, MIXED>::ops());
  register_ops(key, P + 1, Q, Launch3<PHYS, P + 1, Q, MIXED, NT, MIXED ? 56 : 80>::ops());
  if constexpr (MIXED && P >= 6) {
    // 512 threads where no SM has more than one CTA (p = 7, 8 to 125 elements:
    // 9.2 to 9.4 us a stage against 12.9 to 16.6 with 256, p = 6 9.2 to 9.4
    // against 11.1 to 14.1; 216 elements 17.6 and 17.4 against 16.2 and 14.4)
    KernelOps o = Launch3<PHYS, P + 1, Q, MIXED, 512, 128>::ops();
    o.preferred = 0;
    o.small = 1;
    register_ops(key, P + 1, Q, o);
  }
}

// The second-form stage kernel (stage2.cuh) for LSRK and right-hand-side
// stages; other stage kinds, and every other kernel of the handle, come from
// the third-form tile of the same (L, Q).
template <int PHYS, int L, int Q, int EPB, int NT, int MINB, bool MIXED = false, int VD = 0>
struct Launch2 {
  static_assert(EPB == 1, "the third form's tiles hold one element");
  using Base = Launch3<PHYS, L, Q, MIXED>;
  using C = Cfg2<PHYS, L, Q, EPB, NT, MINB, MIXED, VD>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init(t);
    if (e != cudaSuccess) return e;
    if ((e = upload_tables2_lq<L, Q, typename C::R>(t)) != cudaSuccess) return e;
    if constexpr (NODAL2)
      if ((e = cudaFuncSetAttribute(rhs2_kernel<C, PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM)) != cudaSuccess)
        return e;
    return cudaFuncSetAttribute(stage2_kernel<C, PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
  }
  // right-hand side on GLL values in this form where its stage is the default
  static constexpr bool NODAL2 = !MIXED && L <= 5 && (5 * L * L <= NT);
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    if constexpr (NODAL2) {
      rhs2_kernel<C, PHYS><<<(unsigned)a.ne, NT, C::SMEM, s>>>(a);
      return cudaGetLastError();
    } else {
      return cudaErrorNotSupported;
    }
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage2_kernel<C, PHYS>, NT, C::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    if (a.kind != kLSRK && a.kind != kRHS) return Base::stage_grid(a, g, s);
    return launch_dependent(stage2_kernel<C, PHYS>, (unsigned)g, NT, C::SMEM, s, a);
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) {
    if (a.kind != kLSRK && a.kind != kRHS) return Base::stage(a, s);
    return launch_dependent(stage2_kernel<C, PHYS>, (unsigned)((a.ne + EPB - 1) / EPB), NT, C::SMEM, s, a);
  }
  static KernelOps ops() {
    KernelOps o = Base::ops();
    o.epb = EPB; o.nt = NT; o.minb = MINB; o.smem = C::SMEM; o.preferred = 0;
    if constexpr (NODAL2) o.rhs_nodal = rhs_nodal;
    o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.warp = 3;
    return o;
  }
};

template <int PHYS, int P, int Q, int EPB, int NT, int MINB, bool MIXED, int VD = 0>
void reg2_variant(int preferred = 0, int small = 0) {
  using C = Cfg2<PHYS, P + 1, Q, EPB, NT, MINB, MIXED, VD>;
  if constexpr (C::SMEM <= 227 * 1024 && (MINB == 0 || (65536 / (NT * MINB) >= 40 &&
                                                        (int)((228 * 1024) / (C::SMEM + 1024)) >= MINB)))
  {
    KernelOps o = Launch2<PHYS, P + 1, Q, EPB, NT, MINB, MIXED, VD>::ops();
    o.preferred = preferred;
    o.small = small;
    register_ops(PHYS + (MIXED ? kMixedKey : 0), P + 1, Q, o);
  }
}

// CTAs per SM of NT threads that a cap of R registers per thread allows: a
// warp's registers come from one of the SM's four 16K-register scheduler
// partitions, so ceil(warps / 4) warps of 32 x R registers share 16K;
// clipped to what the tile's shared memory allows.
template <class C>
constexpr int blocks_for_regs(int nt, int r) {
  const int per_part = 16384 / (32 * r), warps = (nt + 31) / 32;
  const int by_regs = per_part * 4 / warps;
  const int by_smem = (int)((228 * 1024) / (C::SMEM + 1024));
  return by_regs < by_smem ? by_regs : by_smem;
}

// Second-form variants of a 3-D Euler (p, q): one element per CTA at two
// thread counts, uncapped and with the CTAs per SM that caps of 96 and 80
// (and for the FP32 form 64) registers per thread allow; for the FP32 form
// also the volume pass with one direction per thread (fewer registers) at
// caps of 80, 64 and 56.  Appended variants keep the earlier indices.
template <int PHYS, int P, int Q, bool MIXED = false>
void reg2() {
  constexpr int NTA = ((P + 1) * (P + 1) * 5 + 31) / 32 * 32;   // one thread per modal row
  constexpr int NTB = NTA + 32;
  using CA = Cfg2<PHYS, P + 1, Q, 1, NTA, 0, MIXED>;
  using CB = Cfg2<PHYS, P + 1, Q, 1, NTB, 0, MIXED>;
  constexpr int A96 = blocks_for_regs<CA>(NTA, 96), A80 = blocks_for_regs<CA>(NTA, 80);
  constexpr int B96 = blocks_for_regs<CB>(NTB, 96), B80 = blocks_for_regs<CB>(NTB, 80);
  constexpr int B64 = blocks_for_regs<CB>(NTB, 64), A64 = blocks_for_regs<CA>(NTA, 64);
  reg2_variant<PHYS, P, Q, 1, NTA, 0, MIXED>();
  // up to p = 4 the default (p = 3, 32^3: FP64 239 us against the third form's
  // 314, FP32 190 against 214; p = 2, 20^3: 37.5 against 54 and 33 against 41; p = 4,
  // 16^3: 76 against 94 and, 18^3, 71 against 82; at p = 5, 14^3, 87 against 91 and
  // 57 against 57); a mesh of one wave takes the uncapped tile (p = 3, 8^3: 6.7 us
  // against 7.9 to 11.8 for the capped ones).  FP64 at p = 4, where shared memory
  // holds five CTAs at 80 registers as at 96: the wider tile at 96 for every mesh
  // (5^3 8.8 us, uncapped 8.6; 8^3 12.3 / 15.8; 16^3 76 / 81; 30^3 467 / 510).
  constexpr bool WIDE = !MIXED && P <= 4 && A80 == A96;
  constexpr int PREF = P <= 4 ? 2 : 0, ONE_WAVE = P <= 4 && !WIDE ? 4 : 0;
  reg2_variant<PHYS, P, Q, 1, NTB, 0, MIXED>(0, MIXED ? 0 : ONE_WAVE);
  static_assert(!WIDE || B96 >= 2, "a preferred tile");
  if constexpr (B96 >= 2) reg2_variant<PHYS, P, Q, 1, NTB, B96, MIXED>(WIDE ? PREF : 0, MIXED ? ONE_WAVE : 0);
  if constexpr (A96 >= 2) reg2_variant<PHYS, P, Q, 1, NTA, A96, MIXED>();
  if constexpr (B80 >= 2 && B80 != B96) reg2_variant<PHYS, P, Q, 1, NTB, B80, MIXED>();
  if constexpr (A80 >= 2 && A80 != A96) reg2_variant<PHYS, P, Q, 1, NTA, A80, MIXED>(MIXED ? 0 : PREF);
  if constexpr (MIXED && B64 >= 2 && B64 != B80) reg2_variant<PHYS, P, Q, 1, NTB, B64, MIXED>();
  // FP32 with the volume's three directions spread over three warps
  if constexpr (MIXED && A80 >= 2) reg2_variant<PHYS, P, Q, 1, NTA, A80, MIXED, 1>();
  if constexpr (MIXED && B80 >= 2) reg2_variant<PHYS, P, Q, 1, NTB, B80, MIXED, 1>();
  if constexpr (MIXED && A64 >= 2 && A64 != A80) reg2_variant<PHYS, P, Q, 1, NTA, A64, MIXED, 1>();
  constexpr int A56 = blocks_for_regs<CA>(NTA, 56);
  if constexpr (MIXED && B64 >= 2 && B64 != B80) reg2_variant<PHYS, P, Q, 1, NTB, B64, MIXED, 1>();
  if constexpr (MIXED && A56 >= 2 && A56 != A64) reg2_variant<PHYS, P, Q, 1, NTA, A56, MIXED, 1>(PREF);
  // FP64 at 72 registers: one more CTA per SM for a few dozen bytes of spills
  constexpr int A72 = blocks_for_regs<CA>(NTA, 72), B72 = blocks_for_regs<CB>(NTB, 72);
  if constexpr (!MIXED && A72 >= 2 && A72 != A80) reg2_variant<PHYS, P, Q, 1, NTA, A72, MIXED>();
  if constexpr (!MIXED && B72 >= 2 && B72 != B80) reg2_variant<PHYS, P, Q, 1, NTB, B72, MIXED>();
}

// Navier-Stokes 3-D in the third form: ns_flux_kernel, then ns_update_kernel
// as the stage kernel (every stage kind).  The projections and trace kernels
// come from the plain tile.
//
// Threads and register caps, measured as flux + update per stage: p = 7 (12^3)
// flux 256 at 112 with update 256 at 64 registers 232 us, 320 at 96 248, 384
// at 80 246, update 128 at 96 234; p = 5 (14^3) flux 256 at 80 with update 128
// at 96 171 us, 192 at 96 187; p = 3 (16^3) flux 96 at 80 with update 64 at 96
// 90 us, 128 at 96 92.  Above p = 3 an element has more pencils than 256
// threads take in a round, below p = 7 smaller caps buy more CTAs per SM.
template <int PHYS, int L, int Q, int NTF = (L < 5 ? form3_threads(L) : (L == 5 ? 160 : 256)), int RF = (L < 8 ? 80 : 112),
          int NTU = (L < 5 ? 64 : (L < 8 ? 128 : 256)), int RU = (L < 8 ? 96 : 64)>
struct Launch3Ns {
  using Base = Launch<PHYS, L, Q, default_epb(3, Q), 0>;
  using C0 = Cfg3<PHYS, L, Q, 64, 0, false>;
  using CF = Cfg3<PHYS, L, Q, NTF, form3_blocks(NsFlux<C0>::SMEM, NTF, RF), false>;
  using CU = Cfg3<PHYS, L, Q, NTU, form3_blocks(NsUpdate<C0, false>::SMEM, NTU, RU), false>;
  using F = NsFlux<CF>;
  using CN = Cfg3<PHYS, L, Q, NTU, form3_blocks(NsUpdate<C0, true>::SMEM, NTU, 112), false>;
  using N = NsUpdate<CU, false>;
  using NN = NsUpdate<CN, true>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init_aux(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, double>(t);
    // the FP32 viscous form's
    if (e == cudaSuccess) e = upload_tables_lq<L, Q, float>(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, float>(t);
    auto attr = [&](auto k, size_t smem) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    };
    attr(ns_flux_kernel<CF, PHYS, false, false>, F::SMEM);
    attr(ns_flux_kernel<CF, PHYS, true, false>, F::SMEM);
    attr(ns_flux_kernel<CF, PHYS, false, true>, F::SMEM);
    attr(ns_flux_kernel<CF, PHYS, true, true>, F::SMEM);
    attr(ns_update_kernel<CU, PHYS, false>, N::SMEM);
    attr(ns_update_kernel<CN, PHYS, true>, NN::SMEM);
    return e;
  }
  template <bool F32>
  static cudaError_t flux(const StageArgs &a, bool nodal, cudaStream_t s) {
    const unsigned g = a.vtiles ? a.nvtiles : a.ne;
    return launch_dependent(nodal ? ns_flux_kernel<CF, PHYS, true, F32> : ns_flux_kernel<CF, PHYS, false, F32>, g, NTF,
                            F::SMEM, s, a);
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    return launch_dependent(ns_update_kernel<CU, PHYS, false>, (unsigned)g, NTU, N::SMEM, s, a);
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) {
    return stage_grid(a, a.ne, s);
  }
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    return launch_dependent(ns_update_kernel<CN, PHYS, true>, (unsigned)a.ne, NTU, NN::SMEM, s, a);
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ns_update_kernel<CU, PHYS, false>, NTU, N::SMEM) !=
        cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static KernelOps ops() {
    KernelOps o = Base::aux();
    o.epb = 1; o.nt = NTF; o.minb = CF::MINB; o.smem = F::SMEM; o.preferred = 1;
    o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.rhs_nodal = rhs_nodal;
    o.ns_visc = flux<false>; o.ns_visc32 = flux<true>;
    if constexpr (L >= 6) {
      // 3xTF32: at q = 9 the first-form stage tile runs 512 threads (one per
      // point, 736, would get 80 registers and spill about 1 KB each)
      static const KernelOps tensor = Launch<PHYS, L, Q, default_epb(3, Q), 0, false, Q == 9 ? 512 : 0>::ops();
      o.tensor = &tensor;
    }
    return o;
  }
};
template <int PHYS, int P, int Q>
void reg3_ns() {
  register_ops(PHYS, P + 1, Q, Launch3Ns<PHYS, P + 1, Q>::ops());
  // p = 3: 512 elements 21 us against 29, 1728 46 against 50, 2744 66 against 67,
  // 4096 95 against 94.  p = 1 and 2, one wave of its CTAs: 216 elements 11.9 and
  // 14.4 us against 12.4 and 16.2, 729 12.8 and 17.6 against 16.0 and 23.7; 1000
  // 21.3 and 27.2 against 17.4 and 26.1, 8000 91 and 127 against 68 and 109
  KernelOps o = Launch3Ns<PHYS, P + 1, Q, (P < 4 ? 128 : 256), (P < 4 ? 96 : 112), 128, 80>::ops();
  if (P < 4) o.small = P == 3 ? 14 : 5;
  register_ops(PHYS, P + 1, Q, o);
}

// Elements per CTA of a 2-D tile: about 128 modal rows.
constexpr int stage2d_epb(int nf, int L) { return 128 / (nf * L) > 1 ? 128 / (nf * L) : 1; }

// Euler 2-D and shallow water (stage2d.cuh): every stage kind, boundary sides,
// sources and the right-hand side on GLL values.  The projections and trace
// kernels come from the plain tile.
template <int PHYS, int L, int Q, bool MIXED, int EPB = stage2d_epb(phys_nf(PHYS), L), int NT = 128, int MINB = 4>
struct Launch2D {
  using Base = Launch<PHYS, L, Q, default_epb(2, Q), 0, MIXED>;
  using C = CfgD<PHYS, L, Q, EPB, NT, MINB, MIXED>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init_aux(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, typename C::R>(t);
    auto attr = [&](auto k) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    };
    attr(stage2d_kernel<C, PHYS>);
    if constexpr (!MIXED) {
      attr(rhs2d_kernel<C, PHYS, false>);
      attr(rhs2d_kernel<C, PHYS, true>);
    }
    return e;
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    return launch_dependent(stage2d_kernel<C, PHYS>, (unsigned)g, NT, C::SMEM, s, a);
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) { return stage_grid(a, (a.ne + EPB - 1) / EPB, s); }
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    if constexpr (!MIXED) {
      const unsigned g = (a.ne + EPB - 1) / EPB;
      return launch_dependent(a.Tin ? rhs2d_kernel<C, PHYS, false> : rhs2d_kernel<C, PHYS, true>, g, NT, C::SMEM, s, a);
    } else {
      return cudaErrorNotSupported;
    }
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage2d_kernel<C, PHYS>, NT, C::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static KernelOps ops() {
    KernelOps o = Base::aux();
    o.epb = EPB; o.nt = NT; o.minb = MINB; o.smem = C::SMEM; o.mixed = MIXED; o.preferred = 1;
    o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.rhs_nodal = rhs_nodal; o.self_traces = !MIXED;
    return o;
  }
};

// Navier-Stokes 2-D: ns2d_flux_kernel, then the face terms and update of
// stage2d_kernel.
template <int PHYS, int L, int Q, int EPB = stage2d_epb(4, L), int NT = 128, int MINB = 4>
struct Launch2DNs {
  using Base = Launch<PHYS, L, Q, default_epb(2, Q), 0>;
  using C = CfgD<PHYS, L, Q, EPB, NT, MINB, false>;
  using N = NsFlux2<C>;
  static cudaError_t init(const Tables1D &t) {
    cudaError_t e = Base::init_aux(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, double>(t);
    // the FP32 viscous form's
    if (e == cudaSuccess) e = upload_tables_lq<L, Q, float>(t);
    if (e == cudaSuccess) e = upload_tables2_lq<L, Q, float>(t);
    auto attr = [&](auto k, size_t smem) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    };
    attr(ns2d_flux_kernel<C, PHYS, false, false>, N::SMEM);
    attr(ns2d_flux_kernel<C, PHYS, true, false>, N::SMEM_NODAL);
    attr(ns2d_flux_kernel<C, PHYS, false, true>, N::SMEM);
    attr(ns2d_flux_kernel<C, PHYS, true, true>, N::SMEM_NODAL);
    attr(stage2d_kernel<C, PHYS>, C::SMEM);
    attr(rhs2d_kernel<C, PHYS, false>, C::SMEM);
    return e;
  }
  template <bool F32>
  static cudaError_t flux(const StageArgs &a, bool nodal, cudaStream_t s) {
    const unsigned g = a.vtiles ? a.nvtiles : (a.ne + EPB - 1) / EPB;
    return launch_dependent(nodal ? ns2d_flux_kernel<C, PHYS, true, F32> : ns2d_flux_kernel<C, PHYS, false, F32>, g, NT,
                            nodal ? N::SMEM_NODAL : N::SMEM, s, a);
  }
  static cudaError_t stage_grid(const StageArgs &a, int g, cudaStream_t s) {
    return launch_dependent(stage2d_kernel<C, PHYS>, (unsigned)g, NT, C::SMEM, s, a);
  }
  static cudaError_t stage(const StageArgs &a, cudaStream_t s) { return stage_grid(a, (a.ne + EPB - 1) / EPB, s); }
  static cudaError_t rhs_nodal(const StageArgs &a, cudaStream_t s) {
    return launch_dependent(rhs2d_kernel<C, PHYS, false>, (unsigned)((a.ne + EPB - 1) / EPB), NT, C::SMEM, s, a);
  }
  static int blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage2d_kernel<C, PHYS>, NT, C::SMEM) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    return n > 0 ? n : 1;
  }
  static KernelOps ops() {
    KernelOps o = Base::aux();
    o.epb = EPB; o.nt = NT; o.minb = MINB; o.smem = N::SMEM; o.preferred = 1;
    o.init = init; o.stage = stage; o.stage_grid = stage_grid; o.blocks_per_sm = blocks_per_sm;
    o.rhs_nodal = rhs_nodal;
    o.ns_visc = flux<false>; o.ns_visc32 = flux<true>;
    return o;
  }
};

// 2-D tiles of one (physics, p, q): E elements (128 modal rows) at 128 threads;
// 256, where every interval's tasks run side by side, for a mesh of one CTA per
// SM or less (16 x 16, p = 4: 6.5 us a stage against 7.4); and 64.  In FP64,
// where the registers hold an SM to 16 warps, eight 64-thread CTAs of E elements
// have twice the elements in flight, two rounds of rows per interval to hide
// loads and FP64 chains behind: up to p = 5 the default above what one wave of
// 128-thread CTAs holds (us a stage, 128 / 64 threads: p = 1, 100 x 100 9.5 /
// 10.1, 200 x 200 22.3 / 22.3; p = 2, 150 x 150 21.7 / 19.9, 300 x 300 91 / 80;
// p = 3, 100 x 100 16.1 / 17.2, 200 x 200 51.5 / 48.0; p = 4, 60 x 60 16.4 / 14.9,
// 100 x 100 26.0 / 23.3, 300 x 300 209 / 176; p = 5, 80 x 80 24.2 / 22.5, 160 x 160
// 76.3 / 71.2), unless fewer than seven fit the shared memory.  At p = 6, where
// it spills 680 bytes (128 threads 276), only while one wave of it holds the mesh:
// 50 x 50 20.3 / 19.9, 60 x 60 21.9 / 20.5, but 75 x 75 29.7 / 33.6, 120 x 120 62.6
// / 69.3, 200 x 200 175 / 181.
template <int PHYS, int P, int Q, bool MIXED = false>
void reg2d() {
  constexpr int E = stage2d_epb(phys_nf(PHYS), P + 1), B = MIXED ? 6 : 4;
  const int key = PHYS + (MIXED ? kMixedKey : 0);
  using Half = Launch2D<PHYS, P + 1, Q, MIXED, MIXED ? (E + 1) / 2 : E, 64, 2 * B>;
  KernelOps wide = Launch2D<PHYS, P + 1, Q, MIXED, E, 256, 1>::ops(),
            full = Launch2D<PHYS, P + 1, Q, MIXED, E, 128, B>::ops(), half = Half::ops();
  wide.preferred = half.preferred = 0;
  wide.small = E;
  if (!MIXED && 7 * (half.smem + 1024) <= 228 * 1024) {
    full.small = B * E;
    if (P < 6) half.preferred = 2; else half.small = 7 * E;
  }
  register_ops(key, P + 1, Q, wide);
  register_ops(key, P + 1, Q, full);
  register_ops(key, P + 1, Q, half);
}
template <int PHYS, int P, int Q>
void reg2d_ns() {
  constexpr int E = stage2d_epb(4, P + 1);
  register_ops(PHYS, P + 1, Q, Launch2DNs<PHYS, P + 1, Q, E, 128, 5>::ops());
  register_ops(PHYS, P + 1, Q, Launch2DNs<PHYS, P + 1, Q, (E + 1) / 2, 64, 8>::ops());
}

template <int PHYS, int P, int Q, int EPB, int MINB, bool MIXED>
void reg_pipe() {
  using C = Cfg<PHYS, P + 1, Q, EPB, MINB, MIXED>;
  using PP = Pipe<C>;
  if constexpr (PP::OK && PP::SMEM <= 227 * 1024 && (MINB == 0 || 65536 / (C::NT * MINB) >= 48)) {
    if constexpr (MINB == 0 || (228 * 1024) / (PP::SMEM + 1024) >= MINB)
      register_ops(PHYS + (MIXED ? kMixedKey : 0), P + 1, Q, PLaunch<PHYS, P + 1, Q, EPB, MINB, MIXED>::ops());
  }
}

}  // namespace dgmx
