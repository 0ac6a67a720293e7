// Fused DG stage kernel for 2-D quadrilaterals (sm_100a), FP64 and the mixed
// FP32 form: Euler and shallow water, every stage kind, boundary sides,
// sources, and the right-hand side on GLL values.
//
// Same arithmetic contract as stage_tile (stage.cuh) with the element's
// operators ordered so that a stage takes five barrier intervals instead of
// about fourteen and shared memory carries only what changes hands:
//   1. numerical flux at the face points and, beside it, modal rows -> values
//      along j (one thread per modal row, read from global memory by it);
//   2. one thread per point column and flux direction: the column's values
//      along i, the contravariant fluxes at its points and their projection
//      along i, all in registers; beside it the projection of the face terms;
//   3. one thread per modal row: projection along j, face terms, stage update,
//      end values along j of the next state;
//   4. end values along i;  5. next traces.
// Navier-Stokes runs intervals 1 (faces) and 3 to 5 on the volume part that
// ns2d_flux_kernel (below) leaves.
// Operators are folded into even and odd parts (form3.cuh).  The two flux
// directions of a column go to two threads: each evaluates the column's state
// again, which is cheaper than holding both directions' sums (2 NF L values)
// and gives the interval twice the threads.
#pragma once

#include "form3.cuh"
#include "ns.cuh"

namespace dgmx {

template <int PHYS, int L_, int Q_, int EPB_, int NT_, int MINB_, bool MIXED_>
struct CfgD {
  static constexpr bool MIXED = MIXED_;
  static constexpr int PHYSICS = PHYS, DIM = 2;
  using R = std::conditional_t<MIXED_, float, double>;
  static constexpr int NF = phys_nf(PHYS), L = L_, Q = Q_, G = Q_ - 1, EPB = EPB_, NT = NT_;
  static constexpr int MINB = MINB_ > 0 ? MINB_ : 1, MINB_REQ = MINB_;
  static constexpr int NFACE = 4, GF = G, LD = L * L, QD = Q * Q;
  static constexpr int BANKS = 128 / (int)sizeof(R);
  static constexpr int PQ = Q % 2 == 0 ? Q + 1 : Q;                  // rows of Q: odd pitch
  static constexpr int MF = G > L ? G : L, PF = MF % 2 == 0 ? MF + 1 : MF;   // face lines, G -> L in place
  static constexpr int S_T = NF * L * PQ, S_F = NFACE * NF * PF;
  // regions of one element: row values T (later the next state), projected
  // fluxes X0 and X1, face terms XL, end lines FP
  static constexpr int O_T = 0, O_X0 = S_T, O_X1 = 2 * S_T, O_XL = 3 * S_T, O_FP = O_XL + S_F;
  // element pitch = Q (mod banks): a warp's columns read consecutive banks
  static constexpr int SLOT = align_to(O_FP + S_F, Q, BANKS);
  static constexpr size_t DATA = ((size_t)EPB * SLOT * sizeof(R) + 15) / 16 * 16;
  // element and class; the mixed form's element mean (four values)
  static constexpr size_t SMEM = DATA + (size_t)EPB * (MIXED_ ? 32 : 16);
  // flux constants of the right-hand side on GLL values (direction d, field n at
  // NF d + n) in the place of the end lines, which only stages use
  static constexpr int O_CST = O_FP;
  // those constants up to p = 4: above, this form rounds no more than the
  // derivative-first form without (1.24, 1.68, 1.19 times its distance from a
  // 64-bit evaluation at p = 2, 3, 4, with the constants 0.69; 0.92 at p = 5)
  static constexpr bool SHIFT = L <= 5;
};

template <class C>
struct SmemD {
  using T = typename C::R;
  T *base;
  int *eid, *cls;
  T *mean;
  int end;   // first element behind the tile's own
  __device__ SmemD(unsigned char *raw, int end_) : end(end_) {
    base = reinterpret_cast<T *>(raw);
    eid = reinterpret_cast<int *>(raw + C::DATA);
    cls = eid + C::EPB;
    mean = reinterpret_cast<T *>(reinterpret_cast<unsigned char *>(eid) + 16 * C::EPB);
  }
  __device__ T *slot(int s) const { return base + (size_t)s * C::SLOT; }
};

template <class C>
__device__ __forceinline__ void sd_load(const SmemD<C> &sm, const StageArgs &a, int e0, int tid) {
  for (int s = tid; s < C::EPB; s += C::NT) {
    const int e = e0 + s, c = e < sm.end ? a.links[(size_t)e * 4].cls : -1;   // -1: unallocated
    sm.cls[s] = c >= 0 ? c : 0;
    sm.eid[s] = c >= 0 ? e : -1;
  }
}

// Trace values of GLL values (Field layout) at Gauss point g of face f of
// element e (GL2G, src/Quad.cpp:884-905).
template <class C>
__device__ __forceinline__ void sd_nodal_trace(const StageArgs &a, int e, int f, int g, double *U) {
  constexpr int Q = C::Q, L = C::L;
  // faces: 0 j=0, 1 i=Q-1, 2 j=Q-1, 3 i=0; the line's points along i (0, 2) or j
  const int at = f == 1 ? (Q - 1) * Q : (f == 2 ? Q - 1 : 0), st = f % 2 == 0 ? Q : 1;
#pragma unroll
  for (int n = 0; n < C::NF; ++n) U[n] = 0.0;
#pragma unroll
  for (int x = 0; x < Q; ++x) {
    double c = cGL2G<double, L, Q>[x];
#pragma unroll
    for (int h = 1; h < C::G; ++h) c = g == h ? cGL2G<double, L, Q>[h * Q + x] : c;
#pragma unroll
    for (int n = 0; n < C::NF; ++n) U[n] = fma(c, __ldg(a.Xn + ((size_t)n * a.ne + e) * C::QD + at + x * st), U[n]);
  }
}

// ---- interval 1a: (F^ - F(U_own)).n J_side/J_el at face point g of face f ------
// SELF: both sides' traces are interpolated here from the GLL values instead
// of being read from trace buffers.  KEEP: the element's own flux at a point
// of faces 0 and 3 becomes the constants of its volume fluxes along j and i
// (pencil.cuh; their outward normal times J_side/J_el is -metric[d]).  Where it
// is not finite, neither is the face's term, nor then the element's result.
template <class C, int PHYS, bool KEEP, bool SELF>
__device__ __forceinline__ void sd_face_point(const SmemD<C> &sm, const StageArgs &a, int e0, int w) {
  using T = typename C::R;
  constexpr int NF = C::NF, G = C::G;
  const int s = w / (4 * G), rem = w - s * 4 * G, f = rem / G, g = rem - f * G, e = e0 + s;
  if (e >= sm.end) return;
  const int cls = __ldg(&a.links[(size_t)e * 4].cls);
  if (cls < 0) return;   // unallocated
  const FaceLink *lp = a.links + (size_t)e * 4 + f;
  const FaceLink lk{__ldg(&lp->elem), __ldg(&lp->face), __ldg(&lp->perm), cls};
  const GeomClass *gc = a.classes + cls;
  const int gn = __ldg(a.perm + lk.perm + g);
  T Uo[5], Un[5];
  if constexpr (SELF) {
    sd_nodal_trace<C>(a, e, f, g, Uo);
    sd_nodal_trace<C>(a, lk.elem, lk.face, gn, Un);
  } else {
    const T *Tin = trace_in<C>(a);
    const T *to = Tin + ((size_t)e * 4 + f) * NF * G + g, *tn = Tin + ((size_t)lk.elem * 4 + lk.face) * NF * G + gn;
#pragma unroll
    for (int k = 0; k < NF; ++k) { Uo[k] = to[k * G]; Un[k] = tn[k * G]; }
  }
  const T nm[3] = {T(__ldg(&gc->nrm[f][0])), T(__ldg(&gc->nrm[f][1])), T(0)};
  const T jr = T(__ldg(&gc->jr[f]));
  const bool master = (__ldg(&gc->master) >> f) & 1;
  if constexpr (!C::MIXED) {
    const int bt = (__ldg(&gc->bc) >> (4 * f)) & 15;
    if (bt) ghost_state<2, NF>(a.bckind[bt], a.bcpar[bt], Uo, nm, false, Un);
  }
  T UL[5], UR[5], Fh[5], FL[5], FR[5];
#pragma unroll
  for (int k = 0; k < NF; ++k) { UL[k] = master ? Uo[k] : Un[k]; UR[k] = master ? Un[k] : Uo[k]; }
  T *eo = sm.slot(s) + C::O_XL + f * NF * C::PF + g;
  bool ok;
  if constexpr (C::MIXED) {
    const RefState<T> ref = *reinterpret_cast<const RefState<T> *>(a.uref + kUrefStride * solve_of(a, e) + 10);
    ok = face_flux_pert<PHYS, T>(ref, UL, UR, nm, T(a.gamma), a.flux, Fh, FR);
#pragma unroll
    for (int k = 0; k < NF; ++k) eo[k * C::PF] = (master ? Fh[k] : FR[k] - Fh[k]) * jr;
  } else {
    ok = face_flux<PHYS, T>(UL, UR, nm, T(a.gamma), a.flux, Fh, FL, FR);
#pragma unroll
    for (int k = 0; k < NF; ++k) eo[k * C::PF] = (master ? Fh[k] - FL[k] : FR[k] - Fh[k]) * jr;
    if (KEEP && g == G / 2 && f % 3 == 0)
#pragma unroll
      for (int k = 0; k < NF; ++k)
        sm.slot(s)[C::O_CST + (f == 0 ? NF : 0) + k] = jr * (master ? -FL[k] : FR[k]);
    if constexpr (is_ns(PHYS)) {
      // BR1 viscous lift: the central average leaves (V_own + V_nbr)/2, zero
      // on boundary sides (src/Navier_Stokes.cpp:113-252)
      if (!((__ldg(&gc->bc) >> (4 * f)) & 15)) {
        const double *vo = a.V + ((size_t)e * 4 + f) * (NF - 1) * G + g;
        const double *vn = a.V + ((size_t)lk.elem * 4 + lk.face) * (NF - 1) * G + gn;
#pragma unroll
        for (int k = 1; k < NF; ++k) eo[k * C::PF] = fma(0.5 * jr, vo[(k - 1) * G] + vn[(k - 1) * G], eo[k * C::PF]);
      }
    }
  }
  if (!ok) {
    atomicOr(a.err, 1);
    atomicMin(a.err + 1, e);
  }
}

// ---- interval 1b: modal row (n, a) -> values along j ----------------------------
template <class C>
__device__ __forceinline__ void sd_state_row(const SmemD<C> &sm, const StageArgs &a, int e0, int w) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q, RPS = C::NF * L;
  const int s = w / RPS, r = w - s * RPS, e = e0 + s;
  if (e >= sm.end) return;
  double x[L];
  ld_row<L>(a.X + ((size_t)e * RPS + r) * L, x);
  if constexpr (C::MIXED)   // the constant mode is left out; its value:
    if (r % L == 0) {
      sm.mean[4 * s + r / L] = T(0.5 * x[0]);
      x[0] = 0.0;
    }
  T v[L], u[Q];
#pragma unroll
  for (int k = 0; k < L; ++k) v[k] = T(x[k]);
  eo_expand<L, Q>(v, u);
  st_pencil<Q>(sm.slot(s) + C::O_T + r * C::PQ, 1, u);
}

// ---- interval 2: one column of points, one flux direction -----------------------
// Contravariant flux G = metric[R] . F(U) of one point, less the constants c
// (SHIFT), into g[n].
template <class C, int PHYS, bool SHIFT>
__device__ __forceinline__ void sd_point_flux(const typename C::R *U, const typename C::R *m, typename C::R gamma,
                                              const RefState<typename C::R> &ref, const typename C::R *c,
                                              typename C::R *g) {
  using T = typename C::R;
  T F[3][5];
  if constexpr (C::MIXED) volume_flux_pert<PHYS, T>(ref, U, gamma, F);
  else volume_flux<PHYS, T>(U, gamma, F);
#pragma unroll
  for (int n = 0; n < C::NF; ++n) g[n] = fma(m[1], F[1][n], SHIFT ? fma(m[0], F[0][n], -c[n]) : m[0] * F[0][n]);
}

// X_R[n][a] = sum_i C[a][i] G_R[n][i] along the column's points, C = E for the
// flux along i (R = 0), P for the one along j.
template <class C, int PHYS, int R, bool NODAL>
__device__ __forceinline__ void sd_column(const SmemD<C> &sm, const StageArgs &a, int s, int j) {
  using T = typename C::R;
  constexpr int NF = C::NF, L = C::L, Q = C::Q, PQ = C::PQ;
  const GeomClass *gc = a.classes + sm.cls[s];
  const T m[2] = {T(__ldg(&gc->metric[3 * R])), T(__ldg(&gc->metric[3 * R + 1]))};
  const T gamma = T(a.gamma);
  // FP64 above L = 5: the sums alone take 128 registers' worth at L = 8, so
  // the column's modal values are read again for each pair of points
  // (volatile keeps the compiler from holding them all)
  constexpr bool REREAD = !C::MIXED && L > 5;
  T v[NF][L];
  const T *t = sm.slot(s) + C::O_T + j;
  const double *xn = nullptr;
  if constexpr (NODAL) {
    xn = a.Xn + (size_t)(sm.eid[s] >= 0 ? sm.eid[s] : 0) * C::QD + j;
  } else if constexpr (!REREAD) {
#pragma unroll
    for (int n = 0; n < NF; ++n) ld_pencil<L>(t + n * L * PQ, PQ, v[n]);
  }
  auto val = [&](int n, int b) -> T {
    if constexpr (REREAD) return *(const volatile T *)(t + (n * L + b) * PQ);
    else return v[n][b];
  };
  T acc[NF][L];
#pragma unroll
  for (int n = 0; n < NF; ++n) zero<L>(acc[n]);
  // The mixed form's fluxes are about the element's mean, the right-hand
  // side's on GLL values less the element's constants (pencil.cuh).  FP64
  // stages leave them whole: their own update of the state rounds more than
  // the operators do (0.96 of the derivative-first form's distance from a
  // 64-bit evaluation).
  RefState<T> ref;
  if constexpr (C::MIXED) ref = element_reference<PHYS, T>(sm.mean + 4 * s, gamma);
  const T *cst = sm.slot(s) + C::O_CST + NF * R;
#pragma unroll
  for (int i = 0; i < (Q + 1) / 2; ++i) {
    const bool mid = 2 * i + 1 == Q;
    T Up[5], Um[5], Gp[5], Gm[5];
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      if constexpr (NODAL) {
        Up[n] = T(xn[(size_t)n * a.ne * C::QD + i * Q]);
        if (!mid) Um[n] = T(xn[(size_t)n * a.ne * C::QD + (Q - 1 - i) * Q]);
      } else {
        T e = T(0), o = T(0);
#pragma unroll
        for (int b = 0; b < L; b += 2) e = fma(cB<T, L, Q>[b * Q + i], val(n, b), e);
        if (!mid)
#pragma unroll
          for (int b = 1; b < L; b += 2) o = fma(cB<T, L, Q>[b * Q + i], val(n, b), o);
        Up[n] = e + o;
        Um[n] = e - o;
      }
    }
    sd_point_flux<C, PHYS, NODAL && C::SHIFT>(Up, m, gamma, ref, cst, Gp);
    if (!mid) sd_point_flux<C, PHYS, NODAL && C::SHIFT>(Um, m, gamma, ref, cst, Gm);
#pragma unroll
    for (int n = 0; n < NF; ++n) {
      const T sum = mid ? Gp[n] : Gp[n] + Gm[n], dif = mid ? T(0) : Gp[n] - Gm[n];
#pragma unroll
      for (int b = 0; b < L; ++b) {
        const bool sym = (b % 2 == 0) != (R == 0);
        if (mid && !sym) continue;
        acc[n][b] = fma(R == 0 ? cE2<T, L, Q>[b * Q + i] : cBw<T, L, Q>[b * Q + i], sym ? sum : dif, acc[n][b]);
      }
    }
  }
  T *x = sm.slot(s) + (R == 0 ? C::O_X0 : C::O_X1) + j;
#pragma unroll
  for (int n = 0; n < NF; ++n) st_pencil<L>(x + n * L * PQ, PQ, acc[n]);
}

// Projection of one face's terms of one field, in place: XL[b] = sum_g BwG[b][g] E[g].
template <class C>
__device__ __forceinline__ void sd_lift(const SmemD<C> &sm, int w) {
  using T = typename C::R;
  constexpr int L = C::L, G = C::G, Q = C::Q, N = 4 * C::NF;
  const int s = w / N;
  T *p = sm.slot(s) + C::O_XL + (w - s * N) * C::PF;
  T v[G], z[L];
  ld_pencil<G>(p, 1, v);
#pragma unroll
  for (int b = 0; b < L; ++b) {
    T acc = T(0);
#pragma unroll
    for (int g = 0; g < G; ++g) acc = fma(cBwG<T, L, Q>[b * G + g], v[g], acc);
    z[b] = acc;
  }
  st_pencil<L>(p, 1, z);
}

// Adds the projected face terms to row (n, a): faces 0 (j=0) and 2 (j=Q-1)
// hold lines over a, 3 (i=0) and 1 (i=Q-1) over b.
template <class C>
__device__ __forceinline__ void sd_add_faces(const SmemD<C> &sm, int s, int n, int aa, typename C::R (&R)[C::L]) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q, FB = C::NF * C::PF;
  const T *xl = sm.slot(s) + C::O_XL + n * C::PF;
  const T x0 = xl[aa], x2 = xl[2 * FB + aa];
  const T e0 = end_value<T, L, Q>(0, aa), e1 = end_value<T, L, Q>(1, aa);
#pragma unroll
  for (int b = 0; b < L; ++b) {
    T acc = R[b];
    acc = fma(cEnd<T, L, Q>[b], x0, acc);
    acc = fma(cEnd<T, L, Q>[L + b], x2, acc);
    acc = fma(e0, xl[3 * FB + b], acc);
    acc = fma(e1, xl[FB + b], acc);
    R[b] = acc;
  }
}

// ---- interval 3: row (n, a) of the projected right-hand side ---------------------
template <class C>
__device__ __forceinline__ void sd_rhs_row(const SmemD<C> &sm, int s, int n, int aa, typename C::R (&R)[C::L]) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q;
  const T *sl = sm.slot(s);
  T v[Q], sf[(Q + 1) / 2], df[Q / 2];
  zero<L>(R);
  ld_pencil<Q>(sl + C::O_X0 + (n * L + aa) * C::PQ, 1, v);
  eo_fold<Q>(v, sf, df);
  eo_project<L, Q, false>(sf, df, R);
  ld_pencil<Q>(sl + C::O_X1 + (n * L + aa) * C::PQ, 1, v);
  eo_fold<Q>(v, sf, df);
  eo_project<L, Q, true>(sf, df, R);
  sd_add_faces<C>(sm, s, n, aa, R);
}

template <class C>
__device__ __forceinline__ void sd_update_row(const SmemD<C> &sm, const StageArgs &a, int w) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q, RPS = C::NF * L;
  const int s = w / RPS, r = w - s * RPS, n = r / L, aa = r - n * L;
  const int e = sm.eid[s];
  if (e < 0) return;
  T R[L], nx[L];
  const size_t gi = ((size_t)e * RPS + r) * L;
  // the registers' rows are asked for before the row's own work
  const bool lsrk = a.kind == kLSRK;
  double x[L];
  T ut[L];
  ld_row<L>(a.X + gi, x);
  if (lsrk) {
    if constexpr (C::MIXED) ld_row<L>(a.Utf + gi, ut); else ld_row<L>(a.Ut + gi, ut);
  }
  if constexpr (is_ns(C::PHYSICS)) {   // the volume part was left by ns2d_flux_kernel
    ld_row<L>(a.Pv + gi, R);
    sd_add_faces<C>(sm, s, n, aa, R);
  } else {
    sd_rhs_row<C>(sm, s, n, aa, R);
  }
  const double dt = a.dts ? a.dts[solve_of(a, e)] : a.dt;
  if constexpr (C::MIXED) {
    if (a.Ssrc)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= float(a.src_scale * a.Ssrc[gi + k]);
    if (a.Rsub)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= float(a.Rsub[gi + k]);
    const double ref0 = aa == 0 ? a.uref[kUrefStride * solve_of(a, e) + 5 + n] : 0.0;
    if (a.kind == kRHS) {
#pragma unroll
      for (int k = 0; k < L; ++k) a.A[gi + k] = R[k];
    } else {
      const float c0 = float(a.c0), mdt = -float(dt);
#pragma unroll
      for (int k = 0; k < L; ++k) {
        ut[k] = fmaf(mdt, R[k], c0 * ut[k]);
        x[k] = fma(a.c1, double(ut[k]), x[k]);
      }
      st_row<L>(a.Utf + gi, ut);
      st_row<L>(a.U + gi, x);
    }
#pragma unroll
    for (int k = 0; k < L; ++k) nx[k] = float(k == 0 ? x[k] - ref0 : x[k]);
  } else {
    if (a.Ssrc)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= a.src_scale * a.Ssrc[gi + k];
    if (a.Rcap)   // first right-hand side (shallow-water balance)
#pragma unroll
      for (int k = 0; k < L; ++k) a.Rcap[gi + k] = R[k];
    if (a.Rsub)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= a.Rsub[gi + k];
    if (lsrk) {
#pragma unroll
      for (int k = 0; k < L; ++k) {
        ut[k] = fma(-dt, R[k], a.c0 * ut[k]);
        nx[k] = fma(a.c1, ut[k], x[k]);
      }
      st_row<L>(a.Ut + gi, ut);
      st_row<L>(a.U + gi, nx);
    } else {
      double u[L], acc[L];
      const bool to_u = a.kind == kTVD2 || a.kind == kRK43;
      if (a.kind != kTVD0 && a.kind != kRK40 && a.kind != kRHS) ld_row<L>(a.U + gi, u);
      if (a.kind == kRK41 || a.kind == kRK43) ld_row<L>(a.A + gi, acc);
#pragma unroll
      for (int k = 0; k < L; ++k) nx[k] = f3_stage_value(a, dt, R[k], x[k], u[k], acc[k]);
      if (a.kind != kRHS) st_row<L>((to_u ? a.U : a.Ut) + gi, nx);
      if (a.kind == kRK40 || a.kind == kRK41 || a.kind == kRHS) st_row<L>(a.A + gi, acc);
    }
  }
  // the next state's row, and its end values along j (faces 0 and 2)
  T *sl = sm.slot(s);
  st_pencil<L>(sl + C::O_T + r * C::PQ, 1, nx);
  T f0 = T(0), f2 = T(0);
#pragma unroll
  for (int k = 0; k < L; ++k) {
    f0 = fma(cEnd<T, L, Q>[k], nx[k], f0);
    f2 = fma(cEnd<T, L, Q>[L + k], nx[k], f2);
  }
  T *fp = sl + C::O_FP + n * C::PF + aa;
  fp[0] = f0;
  fp[2 * C::NF * C::PF] = f2;
}

// ---- intervals 4 and 5: next traces -------------------------------------------------
template <class C>
__device__ __forceinline__ void sd_ends(const SmemD<C> &sm, int w) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q, RPS = C::NF * L;
  const int s = w / RPS, r = w - s * RPS, n = r / L, b = r - n * L;
  T *sl = sm.slot(s);
  const T *u = sl + C::O_T + n * L * C::PQ + b;
  T lo = T(0), hi = T(0);
#pragma unroll
  for (int k = 0; k < L; ++k) {
    const T v = u[k * C::PQ];
    lo = fma(cEnd<T, L, Q>[k], v, lo);
    hi = fma(cEnd<T, L, Q>[L + k], v, hi);
  }
  T *fp = sl + C::O_FP + n * C::PF + b;
  fp[3 * C::NF * C::PF] = lo;
  fp[C::NF * C::PF] = hi;
}
template <class C>
__device__ __forceinline__ void sd_trace(const SmemD<C> &sm, typename C::R *Tout, int w) {
  using T = typename C::R;
  constexpr int L = C::L, Q = C::Q, G = C::G, N = 4 * C::NF;
  const int s = w / N, fn = w - s * N, e = sm.eid[s];
  if (e < 0) return;
  T v[L], out[G];
  ld_pencil<L>(sm.slot(s) + C::O_FP + fn * C::PF, 1, v);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    T acc = T(0);
#pragma unroll
    for (int b = 0; b < L; ++b) acc = fma(cBg<T, L, Q>[b * G + g], v[b], acc);
    out[g] = acc;
  }
  st_row<G>(Tout + ((size_t)e * N + fn) * G, out);
}

template <class C, int PHYS, bool NODAL, bool SELF>
__device__ __forceinline__ void sd_front(const SmemD<C> &sm, const StageArgs &a, int e0, int tid) {
  constexpr int NT = C::NT, NC = C::EPB * C::Q;
  sd_load<C>(sm, a, e0, tid);
  pdl_wait();
  for (int w = tid; w < C::EPB * 4 * C::G; w += NT) sd_face_point<C, PHYS, NODAL && C::SHIFT && !is_ns(PHYS), SELF>(sm, a, e0, w);
  // from the last thread down: a tile with threads enough for both does the
  // rows beside the face points
  if constexpr (!NODAL && !is_ns(PHYS))
    for (int w = NT - 1 - tid; w < C::EPB * C::NF * C::L; w += NT) sd_state_row<C>(sm, a, e0, w);
  __syncthreads();
  if constexpr (!is_ns(PHYS)) for (int w = tid; w < 2 * NC; w += NT) {
    const int c = w < NC ? w : w - NC, s = c / C::Q, j = c - s * C::Q;
    if (sm.eid[s] < 0) continue;
    if (w < NC) sd_column<C, PHYS, 0, NODAL>(sm, a, s, j);
    else sd_column<C, PHYS, 1, NODAL>(sm, a, s, j);
  }
  // from the last thread down: the columns leave the last warps idle
  for (int w = NT - 1 - tid; w < C::EPB * 4 * C::NF; w += NT) sd_lift<C>(sm, w);
  __syncthreads();
}

// One fused stage of the EPB elements from e0.
template <class C, int PHYS>
__device__ __forceinline__ void stage2d_tile(const SmemD<C> &sm, const StageArgs &a, int e0, int tid) {
  constexpr int NT = C::NT, NR = C::EPB * C::NF * C::L;
  sd_front<C, PHYS, false, false>(sm, a, e0, tid);
  for (int w = tid; w < NR; w += NT) sd_update_row<C>(sm, a, w);
  __syncthreads();
  for (int w = tid; w < NR; w += NT) sd_ends<C>(sm, w);
  __syncthreads();
  for (int w = tid; w < C::EPB * 4 * C::NF; w += NT) sd_trace<C>(sm, trace_out<C>(a), w);
}

template <class C, int PHYS>
__global__ void __launch_bounds__(C::NT, C::MINB) stage2d_kernel(StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemD<C> sm(smem_raw, a.ne);
  pdl_release();
  const int ntile = a.tiles ? *a.ntiles : (int)gridDim.x;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    if (t != (int)blockIdx.x) __syncthreads();
    stage2d_tile<C, PHYS>(sm, a, (a.tiles ? a.tiles[t] : t) * C::EPB, threadIdx.x);
  }
}

// Domain::time_derivative on GLL values.  SELF: one launch, every face's two
// traces interpolated where the flux is taken (GL2G is Q products per value,
// less than writing, launching and reading a trace buffer); otherwise the own
// and neighbour traces come from a.Tin (element partitions, whose ghost
// slots hold traces only).
template <class C, int PHYS, bool SELF>
__global__ void __launch_bounds__(C::NT, C::MINB) rhs2d_kernel(StageArgs a) {
  constexpr int NT = C::NT, L = C::L, Q = C::Q, RPS = C::NF * L;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemD<C> sm(smem_raw, a.ne);
  const int tid = threadIdx.x, e0 = blockIdx.x * C::EPB;
  sd_front<C, PHYS, true, SELF>(sm, a, e0, tid);
  for (int w = tid; w < C::EPB * RPS; w += NT) {
    const int s = w / RPS, r = w - s * RPS, e = sm.eid[s];
    if (e < 0) continue;
    double R[L], u[Q];
    const size_t gi = ((size_t)e * RPS + r) * L;
    if constexpr (is_ns(PHYS)) {
      ld_row<L>(a.Pv + gi, R);
      sd_add_faces<C>(sm, s, r / L, r % L, R);
    } else {
      sd_rhs_row<C>(sm, s, r / L, r % L, R);
    }
    if (a.Ssrc)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= a.src_scale * a.Ssrc[gi + k];
    if (a.Rcap)
#pragma unroll
      for (int k = 0; k < L; ++k) a.Rcap[gi + k] = R[k];
    if (a.Rsub)
#pragma unroll
      for (int k = 0; k < L; ++k) R[k] -= a.Rsub[gi + k];
    eo_expand<L, Q>(R, u);
    st_pencil<Q>(sm.slot(s) + C::O_T + r * C::PQ, 1, u);
  }
  __syncthreads();
  for (int w = tid; w < C::EPB * C::NF * Q; w += NT) {
    const int s = w / (C::NF * Q), r = w - s * C::NF * Q, n = r / Q, j = r - n * Q, e = sm.eid[s];
    if (e < 0) continue;
    double v[L], u[Q];
    ld_pencil<L>(sm.slot(s) + C::O_T + n * L * C::PQ + j, C::PQ, v);
    eo_expand<L, Q>(v, u);
    double *dst = a.Fn + ((size_t)n * a.ne + e) * C::QD + j;
#pragma unroll
    for (int i = 0; i < Q; ++i) dst[i * Q] = u[i];
  }
}

// ---------------------------------------------------------------- Navier-Stokes
// ns2d_flux_kernel: the 2-D form of ns_flux_kernel (form3.cuh), EPB elements
// per CTA: state, lifted projected gradients, stresses, volume flux, its
// projected divergence (a.Pv, [e][n][L^2]) and the viscous normal-flux traces
// (a.V); stage2d_kernel then adds the face terms and advances the stage.
// Buffers [i][j] (rows of PQ): 0..3 the primitive state (density, velocity,
// internal energy), 4..9 the gradient work W; then 0..7 the fluxes (direction
// r, field n at 4 r + n).
template <class C>
struct NsFlux2 {
  static constexpr int BS = C::Q * C::PQ;
  static constexpr int O_W = 4 * BS, O_J = 10 * BS;               // J: jumps [c][f] lines, later face values
  static constexpr int FQ = C::Q % 2 == 0 ? C::Q + 1 : C::Q;      // [f][n] lines of Q
  static constexpr int SLOT = align_to(O_J + cmax(12 * C::PF, 12 * FQ), C::Q, 16);
  static constexpr size_t DATA = (size_t)C::EPB * SLOT * sizeof(double);
  static constexpr size_t SMEM = (DATA + 15) / 16 * 16 + 16 * C::EPB;   // elements and classes
  // flux constants of the right-hand side on GLL values, up to p = 5 (without
  // them 1.56, 1.86, 1.64, 1.31 and, at p = 7, 0.90 times the derivative-first
  // form's distance from a 64-bit evaluation)
  static constexpr bool SHIFT = C::L <= 6;
  static constexpr size_t SMEM_NODAL = SMEM + (SHIFT ? 8 * sizeof(double) * C::EPB : 0);
};

// One column's gradient pass along i: E_i v and P_i v.
template <class C, class T>
__device__ __forceinline__ void ns2_grad_i(const T (&v)[C::Q], T *de, T *pr) {
  constexpr int L = C::L, Q = C::Q;
  T s[(Q + 1) / 2], d[Q / 2], o[L];
  eo_fold<Q>(v, s, d);
  zero<L>(o);
  eo_project<L, Q, true>(s, d, o);
  st_pencil<L>(de, C::PQ, o);
  zero<L>(o);
  eo_project<L, Q, false>(s, d, o);
  st_pencil<L>(pr, C::PQ, o);
}
// Row a: projected derivatives along j and i with the lifted jumps (J: the
// component's four face lines, PF apart), then the chain rule, in z.
template <class C, class T>
__device__ __forceinline__ void ns2_grad_j(const T *de, const T *pr, const T *J, const double *met, int aa,
                                           T (&z)[2][C::L]) {
  constexpr int L = C::L, Q = C::Q, PF = C::PF;
  using K = coef_t<T>;
  T v[Q], s[(Q + 1) / 2], d[Q / 2];
  ld_pencil<Q>(de, 1, v);
  eo_fold<Q>(v, s, d);
  zero<L>(z[0]);
  eo_project<L, Q, false>(s, d, z[0]);
  ld_pencil<Q>(pr, 1, v);
  eo_fold<Q>(v, s, d);
  zero<L>(z[1]);
  eo_project<L, Q, true>(s, d, z[1]);
  const K e0 = end_value<K, L, Q>(0, aa), e1 = end_value<K, L, Q>(1, aa);
  const T j0 = J[aa], j2 = J[2 * PF + aa];
  const K m00 = K(met[0]), m01 = K(met[1]), m10 = K(met[3]), m11 = K(met[4]);
#pragma unroll
  for (int b = 0; b < L; ++b) {
    const T z0 = fma(e1, J[PF + b], fma(e0, J[3 * PF + b], z[0][b]));
    const T z1 = fma(cEnd<K, L, Q>[L + b], j2, fma(cEnd<K, L, Q>[b], j0, z[1][b]));
    z[0][b] = fma(m10, z1, fma(m00, z0, T(0)));
    z[1][b] = fma(m11, z1, fma(m01, z0, T(0)));
  }
}

template <class C, int PHYS, bool NODAL, bool F32>
__global__ void __launch_bounds__(C::NT, C::MINB) ns2d_flux_kernel(StageArgs a) {
  using N = NsFlux2<C>;
  constexpr int L = C::L, Q = C::Q, G = C::G, PQ = C::PQ, PF = C::PF, BS = N::BS, NT = C::NT, EPB = C::EPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *base = reinterpret_cast<double *>(smem_raw);
  int *eid = reinterpret_cast<int *>(smem_raw + (N::DATA + 15) / 16 * 16), *cls = eid + EPB;
  constexpr bool SHIFT = NODAL && N::SHIFT;
  double *cst = reinterpret_cast<double *>(smem_raw + N::SMEM);
  const int tid = threadIdx.x, e0 = (a.vtiles ? a.vtiles[blockIdx.x] : (int)blockIdx.x) * EPB;
  auto slot = [&](int s) { return base + (size_t)s * N::SLOT; };
  pdl_release();
  for (int s = tid; s < EPB; s += NT) {
    const int e = e0 + s, c = e < a.ne ? a.links[(size_t)e * 4].cls : -1;
    eid[s] = c >= 0 ? e : -1;
    cls[s] = c >= 0 ? c : 0;
  }
  pdl_wait();
  // (q_own + q_nbr)/2 - q_own of the primitive variables at the face points,
  // times the face's jump scale n J_side/J_el = jr tv metric[r]
  for (int w = tid; w < EPB * 4 * G; w += NT) {
    const int s = w / (4 * G), rem = w - s * 4 * G, f = rem / G, g = rem - f * G, e = e0 + s;
    if (e >= a.ne) continue;
    const FaceLink *lp = a.links + (size_t)e * 4;
    const int le = __ldg(&lp[f].elem), lf = __ldg(&lp[f].face), perm = __ldg(&lp[f].perm);
    const GeomClass *gc = a.classes + __ldg(&lp->cls);
    const double *to = a.Tin + ((size_t)e * 4 + f) * 4 * G + g;
    const double *tn = a.Tin + ((size_t)le * 4 + lf) * 4 * G + __ldg(a.perm + perm + g);
    double Uo[5], Un[5], qo[4], qn[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { Uo[k] = to[k * G]; Un[k] = tn[k * G]; }
    const int bt = (__ldg(&gc->bc) >> (4 * f)) & 15;
    if (bt) {
      const double on[3] = {__ldg(&gc->onrm[f][0]), __ldg(&gc->onrm[f][1]), 0.0};
      ghost_state<2, 4>(a.bckind[bt], a.bcpar[bt], Uo, on, true, Un);
    }
    primitive<2>(Uo, qo);
    primitive<2>(Un, qn);
    const double t = 0.5 * __ldg(&gc->tv[f]) * __ldg(&gc->jr[f]);
    double *J = slot(s) + N::O_J + f * PF + g;
    if constexpr (F32) {   // pairs (u, v), (e, 0)
      F2 *J2 = reinterpret_cast<F2 *>(J);
      J2[0] = F2(float(t * (qn[0] - qo[0])), float(t * (qn[1] - qo[1])));
      J2[4 * PF] = F2(float(t * (qn[2] - qo[2])), 0.0f);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) J[c * 4 * PF] = t * (qn[c] - qo[c]);
    }
  }
  if constexpr (NODAL) {
    for (int w = tid; w < EPB * 4 * Q * Q; w += NT) {
      const int s = w / (4 * Q * Q), r = w - s * 4 * Q * Q, n = r / (Q * Q), p = r - n * Q * Q, e = e0 + s;
      if (e < a.ne) slot(s)[n * BS + (p / Q) * PQ + p % Q] = a.Xn[((size_t)n * a.ne + e) * Q * Q + p];
    }
  } else {
    for (int w = tid; w < EPB * 4 * L; w += NT) {
      const int s = w / (4 * L), r = w - s * 4 * L, e = e0 + s;
      if (e >= a.ne) continue;
      double v[L], u[Q];
      ld_row<L>(a.X + ((size_t)e * 4 * L + r) * L, v);
      eo_expand<L, Q>(v, u);
      st_pencil<Q>(slot(s) + (r / L) * BS + (r % L) * PQ, 1, u);
    }
  }
  __syncthreads();
  if constexpr (!NODAL)
    for (int w = tid; w < EPB * 4 * Q; w += NT) {
      const int s = w / (4 * Q), r = w - s * 4 * Q;
      if (eid[s] < 0) continue;
      double *p = slot(s) + (r / Q) * BS + r % Q;
      double v[L], u[Q];
      ld_pencil<L>(p, PQ, v);
      eo_expand<L, Q>(v, u);
      st_pencil<Q>(p, PQ, u);
    }
  // projection of the jumps on their faces, in place
  constexpr int NJ = F32 ? 8 : 12;
  for (int w = NT - 1 - tid; w < EPB * NJ; w += NT) {
    const int s = w / NJ;
    if (eid[s] < 0) continue;
    auto line = [&](auto *p) {
      using T = std::remove_reference_t<decltype(*p)>;
      T v[G], z[L];
      ld_pencil<G>(p, 1, v);
#pragma unroll
      for (int b = 0; b < L; ++b) {
        T acc = T(0);
#pragma unroll
        for (int g = 0; g < G; ++g) acc = fma(cBwG<coef_t<T>, L, Q>[b * G + g], v[g], acc);
        z[b] = acc;
      }
      st_pencil<L>(p, 1, z);
    };
    double *p = slot(s) + N::O_J + (w - s * NJ) * PF;
    if constexpr (F32) line(reinterpret_cast<F2 *>(p)); else line(p);
  }
  __syncthreads();
  // density, velocity, internal energy in place
  for (int w = tid; w < EPB * Q * Q; w += NT) {
    const int s = w / (Q * Q), r = w - s * Q * Q;
    if (eid[s] < 0) continue;
    double *p = slot(s) + (r / Q) * PQ + r % Q;
    const double ir = 1.0 / p[0], u = p[BS] * ir, v = p[2 * BS] * ir;
    const double ei = fma(-0.5, fma(v, v, u * u), p[3 * BS] * ir);
    p[BS] = u; p[2 * BS] = v; p[3 * BS] = ei;
  }
  __syncthreads();
  // constants of the fluxes (pencil.cuh): the convective ones of the middle
  // point; stages leave the fluxes whole, as stage2d_kernel's
  if constexpr (SHIFT) for (int w = NT - 1 - tid; w < 2 * EPB; w += NT) {
    const int s = w / 2, d = w - 2 * s;
    if (eid[s] < 0) continue;
    const double *p = slot(s) + (Q / 2) * (PQ + 1), *m = a.classes[cls[s]].metric + 3 * d;
    const double rho = p[0], u = p[BS], v = p[2 * BS], ei = p[3 * BS];
    const double pr = (a.gamma - 1.0) * rho * ei, V = fma(m[1], v, m[0] * u), rV = rho * V;
    double *c = cst + 4 * w;
    c[0] = flux_constant(rV);
    c[1] = flux_constant(fma(rV, u, pr * m[0]));
    c[2] = flux_constant(fma(rV, v, pr * m[1]));
    c[3] = flux_constant(fma(rho, fma(0.5, fma(v, v, u * u), ei), pr) * V);
  }
  const double mu = a.vis, kap = a.gamma / a.Pr * a.vis;
  // gradients, then stresses (t11, t12, t22) and heat flux at the points
  if constexpr (F32) {
    for (int w = tid; w < EPB * 2 * Q; w += NT) {
      const int s = w / (2 * Q), r = w - s * 2 * Q, c = r / Q, j = r - c * Q;
      if (eid[s] < 0) continue;
      const double *p = slot(s) + (c == 0 ? BS : 3 * BS) + j;
      // differences from the middle point, as in ns_flux_kernel
      const double *mid = slot(s) + (c == 0 ? BS : 3 * BS) + (Q / 2) * (PQ + 1), r0 = mid[0], r1 = c == 0 ? mid[BS] : 0.0;
      F2 v[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i) v[i] = F2(float(p[i * PQ] - r0), c == 0 ? float(p[BS + i * PQ] - r1) : 0.0f);
      F2 *W = reinterpret_cast<F2 *>(slot(s) + N::O_W) + 2 * c * BS + j;
      ns2_grad_i<C>(v, W, W + BS);
    }
    __syncthreads();
    // rows: gradient of the pair, combined and expanded along j in place:
    // (u, v) -> (t11, t12), (t22, 0); (e, 0) -> (hx, hy)
    for (int w = tid; w < EPB * 2 * L; w += NT) {
      const int s = w / (2 * L), r = w - s * 2 * L, c = r / L, aa = r - c * L;
      if (eid[s] < 0) continue;
      F2 *W = reinterpret_cast<F2 *>(slot(s) + N::O_W) + 2 * c * BS + aa * PQ;
      const F2 *J = reinterpret_cast<const F2 *>(slot(s) + N::O_J) + c * 4 * PF;
      F2 z[2][L], u[Q];
      ns2_grad_j<C>(W, W + BS, J, a.classes[cls[s]].metric, aa, z);
      const float m = float(mu), k = float(kap);
#pragma unroll
      for (int b = 0; b < L; ++b) {
        const F2 gx = z[0][b], gy = z[1][b];
        if (c == 0) {
          const float g4[4] = {gx.x, gy.x, gx.y, gy.y};
          float t[3];
          viscous_stress<2, float>(g4, 1, m, t);
          z[0][b] = F2(t[0], t[1]);
          z[1][b] = F2(t[2], 0.0f);
        } else {
          z[0][b] = F2(k * gx.x, k * gy.x);
        }
      }
      eo_expand<L, Q>(z[0], u);
      st_pencil<Q>(W, 1, u);
      if (c == 0) {
        eo_expand<L, Q>(z[1], u);
        st_pencil<Q>(W + BS, 1, u);
      }
    }
    __syncthreads();
    for (int w = tid; w < EPB * 3 * Q; w += NT) {
      const int s = w / (3 * Q), r = w - s * 3 * Q;
      if (eid[s] < 0) continue;
      F2 *p = reinterpret_cast<F2 *>(slot(s) + N::O_W) + (r / Q) * BS + r % Q;
      F2 v[L], u[Q];
      ld_pencil<L>(p, PQ, v);
      eo_expand<L, Q>(v, u);
      st_pencil<Q>(p, PQ, u);
    }
  } else {
    for (int w = tid; w < EPB * 3 * Q; w += NT) {
      const int s = w / (3 * Q), r = w - s * 3 * Q, c = r / Q, j = r - c * Q;
      if (eid[s] < 0) continue;
      double v[Q];
      ld_pencil<Q>(slot(s) + (1 + c) * BS + j, PQ, v);
      double *W = slot(s) + N::O_W + 2 * c * BS + j;
      ns2_grad_i<C>(v, W, W + BS);
    }
    __syncthreads();
    for (int w = tid; w < EPB * 3 * L; w += NT) {
      const int s = w / (3 * L), r = w - s * 3 * L, c = r / L, aa = r - c * L;
      if (eid[s] < 0) continue;
      double *W = slot(s) + N::O_W + 2 * c * BS + aa * PQ;
      double z[2][L];
      ns2_grad_j<C>(W, W + BS, slot(s) + N::O_J + c * 4 * PF, a.classes[cls[s]].metric, aa, z);
      st_pencil<L>(W, 1, z[0]);
      st_pencil<L>(W + BS, 1, z[1]);
    }
    __syncthreads();
    // W: ux uy vx vy ex ey -> t11 (W0), t12 (W1), t22 (W3), hx (W4), hy (W5),
    // rows combined (linear in the gradient) and expanded along j
    for (int w = tid; w < EPB * 4 * L; w += NT) {
      const int s = w / (4 * L), r = w - s * 4 * L, k = r / L, aa = r - k * L;
      if (eid[s] < 0) continue;
      double *W = slot(s) + N::O_W + aa * PQ;
      double p[L], q[L], u[Q];
      if (k == 0) {
        ld_pencil<L>(W, 1, p);
        ld_pencil<L>(W + 3 * BS, 1, q);
#pragma unroll
        for (int b = 0; b < L; ++b) {
          const double ux = p[b], vy = q[b];
          p[b] = mu * ((2.0 / 3.0) * (2.0 * ux - vy));
          q[b] = mu * ((2.0 / 3.0) * (2.0 * vy - ux));
        }
        eo_expand<L, Q>(q, u);
        st_pencil<Q>(W + 3 * BS, 1, u);
        eo_expand<L, Q>(p, u);
        st_pencil<Q>(W, 1, u);
      } else if (k == 1) {
        ld_pencil<L>(W + BS, 1, p);
        ld_pencil<L>(W + 2 * BS, 1, q);
#pragma unroll
        for (int b = 0; b < L; ++b) p[b] = mu * (p[b] + q[b]);
        eo_expand<L, Q>(p, u);
        st_pencil<Q>(W + BS, 1, u);
      } else {
        W += (2 + k) * BS;
        ld_pencil<L>(W, 1, p);
#pragma unroll
        for (int b = 0; b < L; ++b) p[b] *= kap;
        eo_expand<L, Q>(p, u);
        st_pencil<Q>(W, 1, u);
      }
    }
    __syncthreads();
    for (int w = tid; w < EPB * 5 * Q; w += NT) {
      const int s = w / (5 * Q), r = w - s * 5 * Q, k = r / Q;
      if (eid[s] < 0) continue;
      double *p = slot(s) + N::O_W + (k < 2 ? k : k + 1) * BS + r % Q;
      double v[L], u[Q];
      ld_pencil<L>(p, PQ, v);
      eo_expand<L, Q>(v, u);
      st_pencil<Q>(p, PQ, u);
    }
  }
  __syncthreads();
  // contravariant flux G_r = metric[r] . (F(U) - g), and g . n on the faces
  for (int w = tid; w < EPB * Q * Q; w += NT) {
    const int s = w / (Q * Q), r = w - s * Q * Q, i = r / Q, j = r - i * Q;
    if (eid[s] < 0) continue;
    double *p = slot(s) + i * PQ + j;
    const GeomClass *gc = a.classes + cls[s];
    const double rho = p[0], u = p[BS], v = p[2 * BS], ei = p[3 * BS];
    double t11, t12, t22, hx, hy;
    if constexpr (F32) {
      const F2 *q = reinterpret_cast<const F2 *>(p + N::O_W);
      t11 = q[0].x; t12 = q[0].y; t22 = q[BS].x; hx = q[2 * BS].x; hy = q[2 * BS].y;
    } else {
      const double *q = p + N::O_W;
      t11 = q[0]; t12 = q[BS]; t22 = q[3 * BS]; hx = q[4 * BS]; hy = q[5 * BS];
    }
    const double qx = fma(t12, v, fma(t11, u, hx)), qy = fma(t22, v, fma(t12, u, hy));
    double pr, H;   // pressure, E + p
    if constexpr (SHIFT) {   // from the energy itself, as in ns_flux_kernel
      const double E = a.Xn[((size_t)3 * a.ne + eid[s]) * Q * Q + r];
      pr = (a.gamma - 1.0) * fma(-0.5 * rho, fma(v, v, u * u), E);
      H = E + pr;
    } else {
      pr = (a.gamma - 1.0) * rho * ei;
      H = fma(rho, fma(0.5, fma(v, v, u * u), ei), pr);
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const double m0 = __ldg(&gc->metric[3 * d]), m1 = __ldg(&gc->metric[3 * d + 1]);
      const double V = fma(m1, v, m0 * u), rV = rho * V;
      const double wx = fma(m1, t12, m0 * t11), wy = fma(m1, t22, m0 * t12), we = fma(m1, qy, m0 * qx);
      double *o = p + 4 * d * BS;
      const volatile double *c = cst + 4 * (2 * s + d);
      o[0] = SHIFT ? fma(rho, V, -c[0]) : rV;
      o[BS] = fma(rV, u, fma(pr, m0, -(SHIFT ? c[1] + wx : wx)));
      o[2 * BS] = fma(rV, v, fma(pr, m1, -(SHIFT ? c[2] + wy : wy)));
      o[3 * BS] = SHIFT ? fma(H, V, -c[3]) - we : fma(H, V, -we);
      const int idx = d == 0 ? i : j;
      if (idx == 0 || idx == Q - 1) {
        const int f = d == 0 ? (idx == 0 ? 3 : 1) : (idx == 0 ? 0 : 2);
        double *fv = slot(s) + N::O_J + f * 3 * N::FQ + (d == 0 ? j : i);
        const double sc = __ldg(&gc->tv[f]);
        fv[0] = sc * wx; fv[N::FQ] = sc * wy; fv[2 * N::FQ] = sc * we;
      }
    }
  }
  __syncthreads();
  for (int w = tid; w < EPB * 8 * Q; w += NT) {
    const int s = w / (8 * Q), r = w - s * 8 * Q, k = r / Q;
    if (eid[s] < 0) continue;
    double *p = slot(s) + k * BS + r % Q;
    double v[Q], sf[(Q + 1) / 2], df[Q / 2], o[L];
    ld_pencil<Q>(p, PQ, v);
    eo_fold<Q>(v, sf, df);
    zero<L>(o);
    if (k < 4) eo_project<L, Q, true>(sf, df, o); else eo_project<L, Q, false>(sf, df, o);
    st_pencil<L>(p, PQ, o);
  }
  for (int w = NT - 1 - tid; w < EPB * 12; w += NT) {   // face values -> Gauss points
    const int s = w / 12, fn = w - s * 12;
    if (eid[s] < 0) continue;
    double v[Q], u[G];
    ld_pencil<Q>(slot(s) + N::O_J + fn * N::FQ, 1, v);
#pragma unroll
    for (int h = 0; h < G; ++h) {
      double acc = 0.0;
#pragma unroll
      for (int x = 0; x < Q; ++x) acc = fma(cGL2G<double, L, Q>[h * Q + x], v[x], acc);
      u[h] = acc;
    }
    st_row<G>(a.V + ((size_t)eid[s] * 12 + fn) * G, u);
  }
  __syncthreads();
  for (int w = tid; w < EPB * 4 * L; w += NT) {
    const int s = w / (4 * L), r = w - s * 4 * L;
    if (eid[s] < 0) continue;
    const double *p = slot(s) + (r / L) * BS + (r % L) * PQ;
    double v[Q], sf[(Q + 1) / 2], df[Q / 2], R[L];
    zero<L>(R);
    ld_pencil<Q>(p, 1, v);
    eo_fold<Q>(v, sf, df);
    eo_project<L, Q, false>(sf, df, R);
    ld_pencil<Q>(p + 4 * BS, 1, v);
    eo_fold<Q>(v, sf, df);
    eo_project<L, Q, true>(sf, df, R);
    st_row<L>(a.Pv + ((size_t)eid[s] * 4 * L + r) * L, R);
  }
}

}  // namespace dgmx
