// In-place DG kernels for 3-D hexahedra (sm_100a): the third form.
//
// An element's data lives in shared memory as a row of equal buffers, one per
// scalar field, each large enough for the Q^3 GLL values.  A 1-D operator is
// applied to a pencil by the one thread that owns it: the pencil is read into
// registers, transformed and written back to the same place, whether the
// operator widens it (modal -> GLL, L to Q values) or narrows it (projection,
// Q to L).  So a pass needs no second buffer, every field of the element goes
// through the same pass together (a Navier-Stokes element has up to 15 fields
// in flight), and an interval between barriers holds hundreds of independent
// pencils.
//
//  * Operators.  P = B W (weighted basis) and E = B W D (weighted derivative)
//    project; B^T expands.  Their tables are symmetric or antisymmetric about
//    the middle of the GLL points, P[a][Q-1-i] = (-1)^a P[a][i] and
//    E[a][Q-1-i] = -(-1)^a E[a][i], so a pencil is folded into sums and
//    differences first and each output takes half the products (even-odd
//    decomposition, Solomonoff 1992): at L = 8, Q = 9 a pass takes 44
//    operations per pencil instead of 72.
//  * The projected divergence of fluxes G_r (contravariant, one per local
//    axis r) is R = P_k P_j (E_i G_0) + P_k E_j (P_i G_1) + E_k P_j (P_i G_2).
//  * Face terms are projected on their face (BwG x BwG) and enter as end
//    values of the face's normal axis, as in stage2.cuh.
//  * Navier-Stokes (BR1, src/Navier_Stokes3d.cpp:182-391): the gradient of an
//    element is needed by that element alone; its neighbours see only the
//    normal viscous flux on the faces.  So one kernel (ns_flux_kernel) forms
//    the state, the lifted projected gradients, the stresses and the complete
//    volume flux (convective minus viscous, before one projection), and a
//    second (ns_update_kernel) adds all face terms and advances the stage.
//    The gradient's lift of the jump along the normal n of a face uses
//    n J_side/J_el = +- metric[r] on affine elements, so the lift is added to
//    the derivative along the local axis r before the chain rule.
//
// Bank conflicts (8-byte values, 16 banks per half warp): rows of k have an
// odd pitch SJ, planes a pitch SI = Q (mod 16) so that the pencils (i, k) of
// a j pass read consecutive banks, and buffers a pitch BS = 8 (mod 16) so
// that two buffers' rows of a k pass fall on the two halves of the banks.
#pragma once

#include "stage2.cuh"

namespace dgmx {

constexpr int align_to(int v, int r, int m) { return v + ((r - v) % m + m) % m; }

template <int PHYS, int L_, int Q_, int NT_, int MINB_, bool MIXED_>
struct Cfg3 {
  static constexpr bool MIXED = MIXED_;
  static constexpr int PHYSICS = PHYS, DIM = 3;
  using R = std::conditional_t<MIXED_, float, double>;
  static constexpr int NF = 5, L = L_, Q = Q_, G = Q_ - 1, EPB = 1, NT = NT_;
  static constexpr int MINB = MINB_ > 0 ? MINB_ : 1, MINB_REQ = MINB_;
  static constexpr int NFACE = 6, GF = G * G, LD = L * L * L, QD = Q * Q * Q;
  static constexpr int BANKS = 128 / (int)sizeof(R);
  // buffer strides: [i][j][k] at i SI + j SJ + k, buffers BS apart
  static constexpr int SJ = Q % 2 == 0 ? Q + 1 : Q;
  static constexpr int SI = align_to(Q * SJ, Q, BANKS);
  static constexpr int BS = align_to((Q - 1) * SI + Q * SJ, 8, BANKS);
  // one (face, field) block of face terms, transformed in place: [g][h] ->
  // [a'][b'], odd row pitch
  static constexpr int MF = G > L ? G : L, PF = MF % 2 == 0 ? MF + 1 : MF, XLS = MF * PF;
  // one (face, component) block of face GLL values
  static constexpr int FVS = Q * SJ;
  static constexpr int PL = L % 2 == 0 ? L + 1 : L;
  static constexpr int FPS = L * PL;                    // end-reduced face plane, rows of PL
  static constexpr int S_XL = NFACE * NF * XLS, S_FP = NFACE * NF * FPS, S_W1 = NFACE * NF * G * PL;
  static constexpr int NG = 15;                         // flux buffers: direction r, field n at 5 r + n
};

// Links and geometry of the element a CTA works on, in shared memory.  The
// classes are read once, coalesced: a mesh whose vertex coordinates round
// differently has hundreds of them, more than the L1 left beside the tiles.
struct Geo3 {
  double metric[9];
  double tv[6];      // n = tv metric[r] on face f
  double jr[6];
  double nrm[6][3], onrm[6][3];
  double mean[5];    // a state of the element (Navier-Stokes: mean[0] a pressure)
  double c[15];      // FP64: constants of its fluxes (direction r, field n at 5 r + n);
                     // the mixed form: the reference state of its volume term
  int master, bc, cls;
  FaceLink lnk[6];
};

template <class C>
__device__ __forceinline__ void f3_load_links(Geo3 &g, const StageArgs &a, int e, int tid) {
  if (tid < 6) {
    const FaceLink lk = a.links[(size_t)e * 6 + tid];
    g.lnk[tid] = lk;
    if (tid == 0) g.cls = lk.cls >= 0 ? lk.cls : 0;
  }
}
// after a barrier
template <class C>
__device__ __forceinline__ void f3_load_geo(Geo3 &g, const StageArgs &a, int tid) {
  const GeomClass *gc = a.classes + g.cls;
  for (int w = tid; w < 58; w += C::NT) {
    if (w < 9) g.metric[w] = gc->metric[w];
    else if (w < 15) g.tv[w - 9] = gc->tv[w - 9];
    else if (w < 21) g.jr[w - 15] = gc->jr[w - 15];
    else if (w < 39) (&g.nrm[0][0])[w - 21] = (&gc->nrm[0][0])[w - 21];
    else if (w < 57) (&g.onrm[0][0])[w - 39] = (&gc->onrm[0][0])[w - 39];
    else { g.master = gc->master; g.bc = gc->bc; }
  }
}

// Asks `bytes` at p into L2 (hints: nothing is moved into the SM and nothing
// waits).
template <int NT>
__device__ __forceinline__ void prefetch_span(const void *p, int bytes, int tid) {
  for (int l = tid; l * 128 < bytes; l += NT) prefetch_l2_lines(p, bytes, l);
}
// The element that starts on this SM slot when this one ends: CTAs start in
// block order, so about (SMs x CTAs per SM) further on.
template <class C>
__device__ __forceinline__ int element_ahead(const StageArgs &a, int e) {
  unsigned nsm;
  asm("mov.u32 %0, %%nsmid;" : "=r"(nsm));
  const int n = e + (int)nsm * C::MINB;
  return n < a.ne ? n : -1;
}

// Asks the neighbours' face blocks of `vals` values per face (Tr: [e][face])
// into L2.
template <class C, class T>
__device__ __forceinline__ void prefetch_neighbours(const Geo3 &g, const T *Tr, int vals, int tid) {
  const int lines = (vals * (int)sizeof(T) + 127) / 128;
  for (int w = tid; w < 6 * lines; w += C::NT) {
    const FaceLink lk = g.lnk[w / lines];
    prefetch_l2_lines(Tr + ((size_t)lk.elem * 6 + lk.face) * vals, vals * (int)sizeof(T), w % lines);
  }
}

// Enumeration of pencils.  i pass: (buffer, j, k) with jk running over the
// padded rows (consecutive banks); j pass: (buffer, a, k); k pass: (a,
// buffer, b), b fastest.
template <class C, class Fn>
__device__ __forceinline__ void pencils_i(int nbuf, int tid, Fn fn) {
  constexpr int N = C::Q * C::SJ;
  for (int w = tid; w < nbuf * N; w += C::NT) {
    const int b = w / N, jk = w - b * N;
    if (C::SJ != C::Q && jk % C::SJ == C::Q) continue;
    fn(b, jk);
  }
}
template <class C, class Fn>
__device__ __forceinline__ void pencils_j(int nbuf, int tid, Fn fn) {
  constexpr int N = C::L * C::Q;
  for (int w = tid; w < nbuf * N; w += C::NT) {
    const int b = w / N, r = w - b * N, a = r / C::Q, k = r - a * C::Q;
    fn(b, a * C::SI + k, a, k);
  }
}
template <class C, class Fn>
__device__ __forceinline__ void pencils_k(int nbuf, int tid, Fn fn) {
  for (int w = tid; w < nbuf * C::L * C::L; w += C::NT) {
    const int b = w % C::L, r = w / C::L, f = r % nbuf, a = r / nbuf;
    fn(f, a * C::SI + b * C::SJ, a, b);
  }
}

// ---- modal -> GLL, in place ----------------------------------------------------
template <class C, class T>
__device__ __forceinline__ void f3_expand_j(T *buf, int nbuf, int tid) {
  pencils_j<C>(nbuf, tid, [&](int b, int o, int, int) {
    T *p = buf + b * C::BS + o;
    T v[C::L], u[C::Q];
    ld_pencil<C::L>(p, C::SJ, v);
    eo_expand<C::L, C::Q>(v, u);
    st_pencil<C::Q>(p, C::SJ, u);
  });
}
template <class C, class T>
__device__ __forceinline__ void f3_expand_i(T *buf, int nbuf, int tid) {
  pencils_i<C>(nbuf, tid, [&](int b, int jk) {
    T *p = buf + b * C::BS + jk;
    T v[C::L], u[C::Q];
    ld_pencil<C::L>(p, C::SI, v);
    eo_expand<C::L, C::Q>(v, u);
    st_pencil<C::Q>(p, C::SI, u);
  });
}
template <class C, class T>
__device__ __forceinline__ void f3_expand_k(T *buf, int nbuf, int tid) {
  pencils_k<C>(nbuf, tid, [&](int f, int o, int, int) {
    T *p = buf + f * C::BS + o;
    T v[C::L], u[C::Q];
    ld_pencil<C::L>(p, 1, v);
    eo_expand<C::L, C::Q>(v, u);
    st_pencil<C::Q>(p, 1, u);
  });
}
// k pass of the state from the modal rows in global memory.  The mixed form
// leaves the constant mode out: its value goes to mean[n].
template <class C>
__device__ __forceinline__ void f3_state_k(typename C::R *buf, double *mean, const StageArgs &a, int e, int tid) {
  using T = typename C::R;
  pencils_k<C>(C::NF, tid, [&](int n, int o, int aa, int b) {
    const int r = (n * C::L + aa) * C::L + b;
    double x[C::L];
    ld_row<C::L>(a.X + ((size_t)e * (C::NF * C::L * C::L) + r) * C::L, x);
    if constexpr (C::MIXED)
      if (aa == 0 && b == 0) {
        mean[n] = 0.35355339059327379 * x[0];   // 2^(-3/2)
        x[0] = 0.0;
      }
    T v[C::L], u[C::Q];
#pragma unroll
    for (int c = 0; c < C::L; ++c) v[c] = T(x[c]);
    eo_expand<C::L, C::Q>(v, u);
    st_pencil<C::Q>(buf + n * C::BS + o, 1, u);
  });
}
// GLL values of the state in Field layout [n][e][Q^3]; the middle point's go to
// mean[n].
template <class C>
__device__ __forceinline__ void f3_state_nodal(double *buf, double *mean, const StageArgs &a, int e, int tid) {
  constexpr int Q = C::Q, QD = C::QD;
  for (int w = tid; w < C::NF * QD; w += C::NT) {
    const int n = w / QD, p = w - n * QD, i = p / (Q * Q), jk = p - i * Q * Q, j = jk / Q, k = jk - j * Q;
    const double v = a.Xn[((size_t)n * a.ne + e) * QD + p];
    buf[n * C::BS + i * C::SI + j * C::SJ + k] = v;
    if (p == Q / 2 * (Q * Q + Q + 1)) mean[n] = v;
  }
}

// ---- projected divergence of the flux buffers ----------------------------------
template <class C, class T>
__device__ __forceinline__ void f3_div_i(T *G, int tid) {
  constexpr int L = C::L, Q = C::Q;
  pencils_i<C>(C::NG, tid, [&](int b, int jk) {
    T *p = G + b * C::BS + jk;
    T v[Q], s[(Q + 1) / 2], d[Q / 2], o[L];
    ld_pencil<Q>(p, C::SI, v);
    eo_fold<Q>(v, s, d);
    zero<L>(o);
    if (b < C::NF) eo_project<L, Q, true>(s, d, o); else eo_project<L, Q, false>(s, d, o);
    st_pencil<L>(p, C::SI, o);
  });
}
template <class C, class T>
__device__ __forceinline__ void f3_div_j(T *G, int tid) {
  constexpr int L = C::L, Q = C::Q;
  pencils_j<C>(C::NF, tid, [&](int n, int o, int, int) {
    T *p = G + n * C::BS + o;
    T v[Q], s[(Q + 1) / 2], d[Q / 2], y[L];
    zero<L>(y);
    ld_pencil<Q>(p, C::SJ, v);
    eo_fold<Q>(v, s, d);
    eo_project<L, Q, false>(s, d, y);
    ld_pencil<Q>(p + C::NF * C::BS, C::SJ, v);
    eo_fold<Q>(v, s, d);
    eo_project<L, Q, true>(s, d, y);
    st_pencil<L>(p, C::SJ, y);
    zero<L>(y);
    ld_pencil<Q>(p + 2 * C::NF * C::BS, C::SJ, v);
    eo_fold<Q>(v, s, d);
    eo_project<L, Q, false>(s, d, y);
    st_pencil<L>(p + 2 * C::NF * C::BS, C::SJ, y);
  });
}
// k pass of one row: R[c] = sum_k P[c][k] Y0[k] + E[c][k] Y2[k]
template <class C, class T>
__device__ __forceinline__ void f3_div_k_row(const T *G, int n, int o, T (&y)[C::L]) {
  constexpr int L = C::L, Q = C::Q;
  T v[Q], s[(Q + 1) / 2], d[Q / 2];
  zero<L>(y);
  ld_pencil<Q>(G + n * C::BS + o, 1, v);
  eo_fold<Q>(v, s, d);
  eo_project<L, Q, false>(s, d, y);
  ld_pencil<Q>(G + (2 * C::NF + n) * C::BS + o, 1, v);
  eo_fold<Q>(v, s, d);
  eo_project<L, Q, true>(s, d, y);
}

// ---- face terms ------------------------------------------------------------------
// Projection of nblk face blocks in place: rows h -> b', then columns g -> a'.
template <class C, class T>
__device__ __forceinline__ void f3_lift_rows(T *X, int nblk, int tid) {
  constexpr int L = C::L, G = C::G, Q = C::Q;
  for (int w = tid; w < nblk * G; w += C::NT) {
    T *p = X + (w / G) * C::XLS + (w % G) * C::PF;
    T v[G], z[L];
    ld_pencil<G>(p, 1, v);
#pragma unroll
    for (int b = 0; b < L; ++b) {
      T acc = T(0);
#pragma unroll
      for (int h = 0; h < G; ++h) acc = fma(cBwG<coef_t<T>, L, Q>[b * G + h], v[h], acc);
      z[b] = acc;
    }
    st_pencil<L>(p, 1, z);
  }
}
template <class C, class T>
__device__ __forceinline__ void f3_lift_cols(const T *X, T *Y, int nblk, int tid) {
  constexpr int L = C::L, G = C::G, Q = C::Q;
  for (int w = tid; w < nblk * L; w += C::NT) {
    const int o = (w / L) * C::XLS + w % L;
    T v[G], z[L];
    ld_pencil<G>(X + o, C::PF, v);
#pragma unroll
    for (int b = 0; b < L; ++b) {
      T acc = T(0);
#pragma unroll
      for (int g = 0; g < G; ++g) acc = fma(cBwG<coef_t<T>, L, Q>[b * G + g], v[g], acc);
      z[b] = acc;
    }
    st_pencil<L>(Y + o, C::PF, z);
  }
}

// The element's face terms E = (F^ - F(U_own)).n J_side/J_el at the side
// Gauss points into blocks [f][n] of XLS: the numerical flux against the
// neighbour's (or a boundary's ghost) state; Navier-Stokes adds the BR1
// viscous lift, whose central average leaves (V_own + V_nbr)/2 (zero on
// boundary sides, src/Navier_Stokes3d.cpp:377-390, :496-513).
template <class C, int PHYS>
__device__ __forceinline__ void f3_faces(typename C::R *X, const Geo3 &g, const RefState<typename C::R> *ref,
                                         const StageArgs &a, int e, int tid) {
  using T = typename C::R;
  constexpr int NF = C::NF, GF = C::GF, G = C::G;
  const T *Tin = trace_in<C>(a);
  for (int w = tid; w < 6 * GF; w += C::NT) {
    const int f = w / GF, q = w - f * GF;
    const FaceLink lk = g.lnk[f];
    const int gn = __ldg(a.perm + lk.perm + q);
    const T *to = Tin + ((size_t)e * 6 + f) * NF * GF + q;
    const T *tn = Tin + ((size_t)lk.elem * 6 + lk.face) * NF * GF + gn;
    const bool master = (g.master >> f) & 1;
    T Uo[5], Un[5], D[5];
#pragma unroll
    for (int k = 0; k < NF; ++k) { Uo[k] = to[k * GF]; Un[k] = tn[k * GF]; }
    T Va[4];
    if constexpr (is_ns(PHYS)) {
      const T *vo = a.V + ((size_t)e * 6 + f) * (NF - 1) * GF + q;
      const T *vn = a.V + ((size_t)lk.elem * 6 + lk.face) * (NF - 1) * GF + gn;
#pragma unroll
      for (int k = 0; k < 4; ++k) Va[k] = vo[k * GF] + vn[k * GF];
    }
    T *eo = X + f * NF * C::XLS + (q / G) * C::PF + q % G;
    const T jr = T(g.jr[f]);
    const T nm[3] = {T(g.nrm[f][0]), T(g.nrm[f][1]), T(g.nrm[f][2])};
    bool ok;
    if constexpr (C::MIXED) {
      T UL[5], UR[5], FR[5];
#pragma unroll
      for (int k = 0; k < NF; ++k) { UL[k] = master ? Uo[k] : Un[k]; UR[k] = master ? Un[k] : Uo[k]; }
      ok = face_flux_pert<PHYS, T>(*ref, UL, UR, nm, T(a.gamma), a.flux, D, FR, a.classes[g.cls].fr[f]);
#pragma unroll
      for (int k = 0; k < NF; ++k) eo[k * C::XLS] = (master ? D[k] : FR[k] - D[k]) * jr;
    } else {
      const int bt = (g.bc >> (4 * f)) & 15;
      if (bt) ghost_state<3, NF>(a.bckind[bt], a.bcpar[bt], Uo, nm, false, Un);
      T UL[5], UR[5];
#pragma unroll
      for (int k = 0; k < NF; ++k) { UL[k] = master ? Uo[k] : Un[k]; UR[k] = master ? Un[k] : Uo[k]; }
      ok = face_jump_vec3<T>(UL, UR, nm, T(a.gamma), a.flux, master, D);
      if constexpr (is_ns(PHYS)) {
        if (!bt)
#pragma unroll
          for (int k = 1; k < NF; ++k) D[k] = fma(0.5, Va[k - 1], D[k]);
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) eo[k * C::XLS] = D[k] * jr;
    }
    if (!ok) {
      atomicOr(a.err, 1);
      atomicMin(a.err + 1, e);
    }
  }
}

// Adds the projected face terms XL [f][n] to row (n, a, b) of the projected
// right-hand side: k faces 0 and 5 (plane (a, b)), j faces 1 and 3 (plane
// (a, c)), i faces 4 and 2 (plane (b, c)).
template <class C, class T>
__device__ __forceinline__ void f3_add_faces(const T *XL, int nblk, int n, int aa, int bb, T (&R)[C::L]) {
  constexpr int L = C::L, Q = C::Q, PF = C::PF;
  const int FB = nblk * C::XLS;
  const T *x = XL + n * C::XLS;
  const T xk0 = x[aa * PF + bb], xk1 = x[5 * FB + aa * PF + bb];
  const T *xj0 = x + FB + aa * PF, *xj1 = x + 3 * FB + aa * PF;
  const T *xi0 = x + 4 * FB + bb * PF, *xi1 = x + 2 * FB + bb * PF;
  const T eb0 = end_value<T, L, Q>(0, bb), eb1 = end_value<T, L, Q>(1, bb);
  const T ea0 = end_value<T, L, Q>(0, aa), ea1 = end_value<T, L, Q>(1, aa);
#pragma unroll
  for (int c = 0; c < L; ++c) {
    T acc = R[c];
    acc = fma(cEnd<T, L, Q>[c], xk0, acc);
    acc = fma(cEnd<T, L, Q>[L + c], xk1, acc);
    acc = fma(eb0, xj0[c], acc);
    acc = fma(eb1, xj1[c], acc);
    acc = fma(ea0, xi0[c], acc);
    acc = fma(ea1, xi1[c], acc);
    R[c] = acc;
  }
}

// ---- stage update -----------------------------------------------------------------
// One mode: the projected right-hand side q through stage kind `kind` from
// the evaluated state x, u = Ut (LSRK) or U (the other kinds) and acc = A
// (RK4); returns the next state and leaves what is stored in u and acc.
__device__ __forceinline__ double f3_stage_value(const StageArgs &a, double dt, double q, double x, double &u,
                                                 double &acc) {
  switch (a.kind) {
    case kLSRK: u = fma(-dt, q, a.c0 * u); return fma(a.c1, u, x);
    case kTVD0: return fma(-dt, q, x);
    case kTVD1:
    case kTVD2: return a.kind == kTVD1 ? fma(a.c0, u, a.c1 * fma(-dt, q, x)) : fma(a.c1, fma(-dt, q, x), a.c0 * u);
    case kRK40: acc = a.c1 * q; return fma(a.c0, q, x);
    case kRK41: acc = fma(a.c1, q, acc); return fma(a.c0, q, u);
    case kRK43: return fma(a.c0, fma(a.c1, q, acc), u);
    default: acc = q; return x;   // kRHS
  }
}

// The whole element: right-hand side rows in UB (field stride sn, planes sa,
// rows sb), plus the volume part `vol` in global memory when given; the next
// state, which the traces are taken of, replaces it.  Consecutive threads
// take consecutive modes, V at a time (2 where modal blocks are even): with a
// row per thread, 64 bytes apart, this interval took 18 k of the
// Navier-Stokes update kernel's 47 k cycles per element at p = 7, coalesced
// 11 k of 35 k (two groups of loads in flight per thread measured no faster).
template <class C>
__device__ __forceinline__ void f3_update_all(typename C::R *UB, int sn, int sa, int sb, const double *vol,
                                              const StageArgs &a, int e, int tid) {
  using T = typename C::R;
  constexpr int L = C::L, LD = C::LD, V = L % 2 == 0 ? 2 : 1, W = C::NF * LD / V;
  const double dt = a.dts ? a.dts[solve_of(a, e)] : a.dt;
  const size_t base = (size_t)e * C::NF * LD;
  const bool lsrk = a.kind == kLSRK;
  const bool need_u = a.kind != kTVD0 && a.kind != kRK40 && a.kind != kRHS;
  const bool need_a = a.kind == kRK41 || a.kind == kRK43;
  // where the next state and the accumulator go
  double *dst = (lsrk || a.kind == kTVD2 || a.kind == kRK43) ? a.U : (a.kind == kRHS ? nullptr : a.Ut);
  const bool put_a = a.kind == kRK40 || a.kind == kRK41 || a.kind == kRHS;
  for (int w = tid; w < W; w += C::NT) {
    const int m = w * V, n = m / LD, r = m - n * LD, ab = r / L, c = r - ab * L;
    T *p = UB + n * sn + (ab / L) * sa + (ab % L) * sb + c;
    const size_t gi = base + m;
    double x[V];
    T u[V];
    ld_row<V>(a.X + gi, x);
    if constexpr (C::MIXED) {
      const double ref0 = r == 0 ? a.uref[kUrefStride * solve_of(a, e) + 5 + n] : 0.0;
      if (lsrk) ld_row<V>(a.Utf + gi, u);
      double un[V];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const float q = p[k];
        if (lsrk) {
          u[k] = fmaf(-float(dt), q, float(a.c0) * u[k]);
          un[k] = fma(a.c1, double(u[k]), x[k]);
        } else {
          a.A[gi + k] = q;
          un[k] = x[k];
        }
        p[k] = float(k == 0 ? un[k] - ref0 : un[k]);
      }
      if (lsrk) { st_row<V>(a.Utf + gi, u); st_row<V>(a.U + gi, un); }
    } else {
      double acc[V], v[V], nx[V];
      if (need_u) ld_row<V>((lsrk ? a.Ut : a.U) + gi, u);
      if (vol) ld_row<V>(vol + gi, v);
      if (need_a) ld_row<V>(a.A + gi, acc);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const double q = vol ? p[k] + v[k] : p[k];
        if (a.R0 && r + k == 0) a.R0[(size_t)e * C::NF + n] = q;   // bulk-flow hold
        nx[k] = f3_stage_value(a, dt, q, x[k], u[k], acc[k]);
        p[k] = nx[k];
      }
      if (lsrk) st_row<V>(a.Ut + gi, u);
      if (dst) st_row<V>(dst + gi, nx);
      if (put_a) st_row<V>(a.A + gi, acc);
    }
  }
}

// ---- next traces --------------------------------------------------------------------
// End values of the next modal block (field stride sn, planes sa, rows sb)
// along a (faces 4, 2), b (1, 3) and c (0, 5) -> FP [f][n][a'][b'].
template <class C, class T>
__device__ __forceinline__ void f3_ends(const T *UB, int sn, int sa, int sb, T *FP, int tid) {
  constexpr int NF = C::NF, L = C::L, Q = C::Q, PL = C::PL, N = NF * L * L, PB = NF * C::FPS;
  for (int w = tid; w < 3 * N; w += C::NT) {
    const int ax = w / N, r = w - ax * N, n = r / (L * L), xy = r - n * L * L, x = xy / L, y = xy - x * L;
    const T *p = UB + n * sn + (ax == 0 ? x * sb + y : (ax == 1 ? x * sa + y : x * sa + y * sb));
    const int st = ax == 0 ? sa : (ax == 1 ? sb : 1);
    T lo = T(0), hi = T(0);
#pragma unroll
    for (int b = 0; b < L; ++b) {
      const T v = p[b * st];
      lo = fma(cEnd<T, L, Q>[b], v, lo);
      hi = fma(cEnd<T, L, Q>[L + b], v, hi);
    }
    T *fp = FP + n * C::FPS + x * PL + y;
    fp[(ax == 0 ? 4 : (ax == 1 ? 1 : 0)) * PB] = lo;
    fp[(ax == 0 ? 2 : (ax == 1 ? 3 : 5)) * PB] = hi;
  }
}
// W1[f][n][g][b'] = sum_a' Bg[a'][g] FP[f][n][a'][b'], then the trace rows.
template <class C, class T>
__device__ __forceinline__ void f3_traces_a(const T *FP, T *W1, int tid) {
  constexpr int L = C::L, Q = C::Q, G = C::G, PL = C::PL;
  for (int w = tid; w < C::NFACE * C::NF * L; w += C::NT) {
    const int fn = w / L, b = w - fn * L;
    T v[L];
    ld_pencil<L>(FP + fn * C::FPS + b, PL, v);
    T *dst = W1 + fn * G * PL + b;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      T acc = T(0);
#pragma unroll
      for (int aa = 0; aa < L; ++aa) acc = fma(cBg<T, L, Q>[aa * G + g], v[aa], acc);
      dst[g * PL] = acc;
    }
  }
}
template <class C, class T>
__device__ __forceinline__ void f3_traces_b(const T *W1, T *Tout, int e, int tid) {
  constexpr int L = C::L, Q = C::Q, G = C::G, PL = C::PL;
  for (int w = tid; w < C::NFACE * C::NF * G; w += C::NT) {
    T v[L], out[G];
    ld_pencil<L>(W1 + w * PL, 1, v);
#pragma unroll
    for (int h = 0; h < G; ++h) {
      T acc = T(0);
#pragma unroll
      for (int b = 0; b < L; ++b) acc = fma(cBg<T, L, Q>[b * G + h], v[b], acc);
      out[h] = acc;
    }
    st_row<G>(Tout + (size_t)e * C::NFACE * C::NF * C::GF + w * G, out);
  }
}
// GLL values from modal rows already expanded along k and j, to Field layout.
template <class C>
__device__ __forceinline__ void f3_store_nodal(const double *buf, const StageArgs &a, int e, int tid) {
  pencils_i<C>(C::NF, tid, [&](int n, int jk) {
    double v[C::L], u[C::Q];
    ld_pencil<C::L>(buf + n * C::BS + jk, C::SI, v);
    eo_expand<C::L, C::Q>(v, u);
    const int j = jk / C::SJ, k = jk - j * C::SJ;
    double *dst = a.Fn + ((size_t)n * a.ne + e) * C::QD + j * C::Q + k;
#pragma unroll
    for (int i = 0; i < C::Q; ++i) dst[i * C::Q * C::Q] = u[i];
  });
}

// ---------------------------------------------------------------------- Euler
// Contravariant fluxes G_r = metric[r] . F(U) at the points: state buffers
// 0..4 -> flux buffers 5 r + n, in place point by point; SHIFT: less the
// constants g.c.  The mixed form evaluates F(Ub + u') - F(Ub)
// (volume_flux_pert, kernels.cuh) about the element's mean.
template <class C, bool SHIFT>
__device__ __forceinline__ void f3_point_fluxes(typename C::R *G, const Geo3 &g, const StageArgs &a, int tid) {
  using T = typename C::R;
  constexpr int Q = C::Q, BS = C::BS;
  const T gm1 = T(a.gamma) - T(1.0);
  T m[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) m[k] = T(g.metric[k]);
  for (int w = tid; w < Q * Q * Q; w += C::NT) {
    const int i = w / (Q * Q), jk = w - i * Q * Q, j = jk / Q, k = jk - j * Q;
    T *p = G + i * C::SI + j * C::SJ + k;
    T U[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) U[n] = p[n * BS];
    if constexpr (C::MIXED) {
      const RefState<T> &b = *reinterpret_cast<const RefState<T> *>(g.c);
      const T ir = p_rcp(b.r + U[0]);
      const T mx = b.m[0] + U[1], my = b.m[1] + U[2], mz = b.m[2] + U[3];
      const T ux = (U[1] - b.u[0] * U[0]) * ir, uy = (U[2] - b.u[1] * U[0]) * ir, uz = (U[3] - b.u[2] * U[0]) * ir;
      T sd = T(0);
      sd = fma(U[1], b.u[0], sd); sd = fma(mx, ux, sd);
      sd = fma(U[2], b.u[1], sd); sd = fma(my, uy, sd);
      sd = fma(U[3], b.u[2], sd); sd = fma(mz, uz, sd);
      const T pp = gm1 * fma(T(-0.5), sd, U[4]);
      const T Hp = U[4] + pp, H = b.H + Hp;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T m0 = m[3 * r], m1 = m[3 * r + 1], m2 = m[3 * r + 2];
        const T Vb = m0 * b.u[0] + m1 * b.u[1] + m2 * b.u[2], Vp = m0 * ux + m1 * uy + m2 * uz;
        T *o = p + 5 * r * BS;
        o[0] = m0 * U[1] + m1 * U[2] + m2 * U[3];
        o[BS] = fma(U[1], Vb, fma(mx, Vp, pp * m0));
        o[2 * BS] = fma(U[2], Vb, fma(my, Vp, pp * m1));
        o[3 * BS] = fma(U[3], Vb, fma(mz, Vp, pp * m2));
        o[4 * BS] = fma(Hp, Vb, H * Vp);
      }
    } else {
      const T ir = T(1.0) / U[0];
      const T u = U[1] * ir, v = U[2] * ir, ww = U[3] * ir;
      const T pr = gm1 * fma(T(-0.5), fma(U[3], ww, fma(U[2], v, U[1] * u)), U[4]);
      const T Ep = U[4] + pr;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T m0 = m[3 * r], m1 = m[3 * r + 1], m2 = m[3 * r + 2];
        const T V = fma(m2, ww, fma(m1, v, m0 * u));
        T *o = p + 5 * r * BS;
        // a product, or the product less a constant (read each time: held in
        // registers the constants spill)
        auto mul = [&](T x, T y, int n) {
          return SHIFT ? fma(x, y, -*(const volatile double *)(g.c + 5 * r + n)) : x * y;
        };
        o[0] = mul(U[0], V, 0);
        o[BS] = fma(U[1], V, mul(pr, m0, 1));
        o[2 * BS] = fma(U[2], V, mul(pr, m1, 2));
        o[3 * BS] = fma(U[3], V, mul(pr, m2, 3));
        o[4 * BS] = mul(Ep, V, 4);
      }
    }
  }
}

// One fused stage (or, NODAL, one right-hand side on GLL values): 15 flux
// buffers and the face terms in shared memory.  The right-hand side rows go
// back to buffers 0..4, whose rows the k pass has just read; the end planes
// FP take the place of the face terms, the traces' first pass W1 buffers 5...
template <class C>
struct Stage3 {
  static constexpr int O_X = C::NG * C::BS;
  static constexpr size_t DATA = ((size_t)(O_X + C::S_XL) * sizeof(typename C::R) + 15) / 16 * 16;
  static constexpr size_t SMEM = DATA + (sizeof(Geo3) + 15) / 16 * 16 + (C::MIXED ? sizeof(RefState<float>) : 0);
  static_assert(C::S_FP <= C::S_XL && C::S_W1 <= 10 * C::BS, "end planes and trace rows fit the dead regions");
};
template <class C, int PHYS, bool NODAL>
__global__ void __launch_bounds__(C::NT, C::MINB) stage3_kernel(StageArgs a) {
  using T = typename C::R;
  using N = Stage3<C>;
  constexpr int L = C::L, BS = C::BS, SI = C::SI, SJ = C::SJ, GF = C::GF;
  // The constants of FP64 fluxes: on GLL values up to p = 4.  Above, this form
  // rounds no more than the derivative-first form without (1.31, 1.64, 1.2 times
  // its distance from a 64-bit evaluation at p = 2, 3, 4, with them 0.86; 1.03 and
  // 0.87 at p = 5 and 7), nor do stages, whose update of the state rounds more
  // than the operators (0.99)
  constexpr bool SHIFT = NODAL && L <= 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *U = reinterpret_cast<T *>(smem_raw), *X = U + N::O_X, *W1 = U + 5 * BS;
  Geo3 &g = *reinterpret_cast<Geo3 *>(smem_raw + N::DATA);
  RefState<T> *ref = reinterpret_cast<RefState<T> *>(smem_raw + N::DATA + (sizeof(Geo3) + 15) / 16 * 16);
  const int tid = threadIdx.x;
  pdl_release();
  const int ntile = a.tiles ? *a.ntiles : a.ne;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    const int e = a.tiles ? a.tiles[t] : t;
    if (t != (int)blockIdx.x) __syncthreads();
    f3_load_links<C>(g, a, e, tid);
    pdl_wait();
    if constexpr (C::MIXED) {
      if (tid == 0) *ref = *reinterpret_cast<const RefState<T> *>(a.uref + kUrefStride * solve_of(a, e) + 10);
    }
    if constexpr (NODAL) f3_state_nodal<C>(U, g.mean, a, e, tid); else f3_state_k<C>(U, g.mean, a, e, tid);
    if (const int n = element_ahead<C>(a, e); n >= 0 && !a.tiles) {
      if constexpr (!NODAL) prefetch_span<C::NT>(a.X + (size_t)n * 5 * C::LD, 5 * C::LD * 8, tid);
      prefetch_span<C::NT>(trace_in<C>(a) + (size_t)n * 30 * GF, 30 * GF * (int)sizeof(T), tid);
    }
    __syncthreads();
    f3_load_geo<C>(g, a, tid);
    prefetch_neighbours<C>(g, trace_in<C>(a), 5 * GF, tid);
    if constexpr (!NODAL) f3_expand_j<C>(U, 5, tid);
    __syncthreads();
    f3_faces<C, PHYS>(X, g, ref, a, e, tid);
    if constexpr (C::MIXED) {
      if (tid == C::NT - 1) {
        T m[5];
#pragma unroll
        for (int n = 0; n < 5; ++n) m[n] = T(g.mean[n]);
        *reinterpret_cast<RefState<T> *>(g.c) = element_reference<PHYS, T>(m, T(a.gamma));
      }
    } else if constexpr (NODAL) {
      const int k = tid - (C::NT - 15);
      if (SHIFT && k >= 0) g.c[k] = flux_constant<3>(g.mean, g.metric + k / 5 * 3, a.gamma, k % 5);
    }
    if constexpr (!NODAL) f3_expand_i<C>(U, 5, tid);
    __syncthreads();
    f3_lift_rows<C>(X, 30, tid);
    f3_point_fluxes<C, SHIFT>(U, g, a, tid);
    __syncthreads();
    f3_lift_cols<C>(X, X, 30, tid);
    f3_div_i<C>(U, tid);
    __syncthreads();
    f3_div_j<C>(U, tid);
    __syncthreads();
    pencils_k<C>(5, tid, [&](int n, int o, int aa, int bb) {
      T R[L];
      f3_div_k_row<C>(U, n, o, R);
      f3_add_faces<C>(X, 5, n, aa, bb, R);
      if constexpr (NODAL) {
        T v[C::Q];
        eo_expand<L, C::Q>(R, v);
        st_pencil<C::Q>(U + n * BS + o, 1, v);
      } else {
        st_pencil<L>(U + n * BS + o, 1, R);
      }
    });
    __syncthreads();
    if constexpr (NODAL) {
      f3_expand_j<C>(U, 5, tid);
      __syncthreads();
      f3_store_nodal<C>(U, a, e, tid);
    } else {
      f3_update_all<C>(U, BS, SI, SJ, nullptr, a, e, tid);
      __syncthreads();
      f3_ends<C>(U, BS, SI, SJ, X, tid);
      __syncthreads();
      f3_traces_a<C>(X, W1, tid);
      __syncthreads();
      f3_traces_b<C>(W1, trace_out<C>(a), e, tid);
    }
  }
}

// ------------------------------------------------------------------ Navier-Stokes
// Shared memory of ns_flux_kernel: 15 buffers, [0, 5) the primitive state
// (density, velocity, internal energy), [5, 15) the gradient work W; then all
// 15 are the flux buffers.  X holds the projected jumps of the gradients
// [c][f] (component-major, 4 x 6 blocks of XLS) and later the face GLL values
// of the viscous normal flux [f][n].
template <class C>
struct NsFlux {
  static constexpr int S_X = cmax(24 * C::XLS, 24 * C::FVS);
  static constexpr int O_W = 5 * C::BS, O_X = 15 * C::BS;
  static constexpr size_t DATA = (size_t)(15 * C::BS + S_X) * sizeof(double);
  static constexpr size_t SMEM = DATA + (sizeof(Geo3) + 15) / 16 * 16;
  // the energy gradient's first pass takes the part of X whose jumps
  // (velocity) are consumed by then as one more scratch buffer
  static_assert(18 * C::XLS >= (C::L - 1) * C::SI + C::Q * C::SJ, "scratch buffer of the energy gradient");
};

// (q_own + q_nbr)/2 - q_own of the primitive variables at the side Gauss
// points, times the face's jump scale, into blocks [c][f].
// FP32 form: formed in FP64, then rounded, components in pairs (u, v), (w, e)
// in blocks [pair][f].
template <class C, bool F32>
__device__ __forceinline__ void ns3_jumps(double *J, const Geo3 &g, const StageArgs &a, int e, int tid) {
  constexpr int NF = C::NF, GF = C::GF, G = C::G;
  for (int w = tid; w < 6 * GF; w += C::NT) {
    const int f = w / GF, q = w - f * GF;
    const FaceLink lk = g.lnk[f];
    const double *to = a.Tin + ((size_t)e * 6 + f) * NF * GF + q;
    const double *tn = a.Tin + ((size_t)lk.elem * 6 + lk.face) * NF * GF + __ldg(a.perm + lk.perm + q);
    double Uo[5], Un[5], qo[4], qn[4];
#pragma unroll
    for (int k = 0; k < NF; ++k) { Uo[k] = to[k * GF]; Un[k] = tn[k * GF]; }
    const int bt = (g.bc >> (4 * f)) & 15;
    if (bt) ghost_state<3, NF>(a.bckind[bt], a.bcpar[bt], Uo, g.onrm[f], true, Un);
    primitive<3>(Uo, qo);
    primitive<3>(Un, qn);
    const int o = f * C::XLS + (q / G) * C::PF + q % G;
    const double t = 0.5 * g.tv[f] * g.jr[f];
    if constexpr (F32) {
      F2 *J2 = reinterpret_cast<F2 *>(J) + o;
      J2[0] = F2(float(t * (qn[0] - qo[0])), float(t * (qn[1] - qo[1])));
      J2[6 * C::XLS] = F2(float(t * (qn[2] - qo[2])), float(t * (qn[3] - qo[3])));
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) J[o + c * 6 * C::XLS] = t * (qn[c] - qo[c]);
    }
  }
}

// Gradient passes of one scalar: i pass, v -> (E_i v, P_i v).
template <class C, class T>
__device__ __forceinline__ void ns3_grad_i(const T (&v)[C::Q], T *de, T *pr) {
  constexpr int L = C::L, Q = C::Q;
  T s[(Q + 1) / 2], d[Q / 2], o[L];
  eo_fold<Q>(v, s, d);
  zero<L>(o);
  eo_project<L, Q, true>(s, d, o);
  st_pencil<L>(de, C::SI, o);
  zero<L>(o);
  eo_project<L, Q, false>(s, d, o);
  st_pencil<L>(pr, C::SI, o);
}
// j pass: (E_i v, P_i v) -> (P_j E_i v, E_j P_i v, P_j P_i v)
template <class C, class T>
__device__ __forceinline__ void ns3_grad_j(const T *de, const T *pr, T *o0, T *o1, T *o2) {
  constexpr int L = C::L, Q = C::Q;
  T v[Q], s[(Q + 1) / 2], d[Q / 2], o[L];
  ld_pencil<Q>(de, C::SJ, v);
  eo_fold<Q>(v, s, d);
  zero<L>(o);
  eo_project<L, Q, false>(s, d, o);
  ld_pencil<Q>(pr, C::SJ, v);
  st_pencil<L>(o0, C::SJ, o);
  eo_fold<Q>(v, s, d);
  zero<L>(o);
  eo_project<L, Q, true>(s, d, o);
  st_pencil<L>(o1, C::SJ, o);
  zero<L>(o);
  eo_project<L, Q, false>(s, d, o);
  st_pencil<L>(o2, C::SJ, o);
}
// k pass of row (a, b): the projected derivatives along the local axes with
// the lifted jumps, then the chain rule: z[d] = sum_r metric[r][d] Z_r, in z.
template <class C, class T>
__device__ __forceinline__ void ns3_grad_k(const T *w0, const T *X, const double *met, int aa, int bb,
                                           T (&z)[3][C::L]) {
  constexpr int L = C::L, Q = C::Q, PF = C::PF, XLS = C::XLS;
  using K = coef_t<T>;
  T v[Q], s[(Q + 1) / 2], d[Q / 2];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    ld_pencil<Q>(w0 + r * C::BS, 1, v);
    eo_fold<Q>(v, s, d);
    zero<L>(z[r]);
    if (r == 2) eo_project<L, Q, true>(s, d, z[r]); else eo_project<L, Q, false>(s, d, z[r]);
  }
  const T xk0 = X[aa * PF + bb], xk1 = X[5 * XLS + aa * PF + bb];
  const T *xj0 = X + XLS + aa * PF, *xj1 = X + 3 * XLS + aa * PF;
  const T *xi0 = X + 4 * XLS + bb * PF, *xi1 = X + 2 * XLS + bb * PF;
  const K eb0 = end_value<K, L, Q>(0, bb), eb1 = end_value<K, L, Q>(1, bb);
  const K ea0 = end_value<K, L, Q>(0, aa), ea1 = end_value<K, L, Q>(1, aa);
  K m[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) m[k] = K(met[k]);
#pragma unroll
  for (int c = 0; c < L; ++c) {
    const T z0 = fma(ea1, xi1[c], fma(ea0, xi0[c], z[0][c]));
    const T z1 = fma(eb1, xj1[c], fma(eb0, xj0[c], z[1][c]));
    const T z2 = fma(cEnd<K, L, Q>[L + c], xk1, fma(cEnd<K, L, Q>[c], xk0, z[2][c]));
#pragma unroll
    for (int k = 0; k < 3; ++k) z[k][c] = fma(m[6 + k], z2, fma(m[3 + k], z1, fma(m[k], z0, T(0))));
  }
}

// Constants of the convective fluxes (pencil.cuh): those of the point at p
// (density, velocity, internal energy, buffers apart), one per thread k < 15,
// and its pressure.
template <class C>
__device__ __forceinline__ void ns3_flux_constants(const double *p, Geo3 &g, double gamma, int k) {
  const int r = k / 5, n = k - 5 * r;
  const float rho = float(p[0]), u = float(p[C::BS]), v = float(p[2 * C::BS]), w = float(p[3 * C::BS]);
  const float ei = float(p[4 * C::BS]);
  const float m0 = float(g.metric[3 * r]), m1 = float(g.metric[3 * r + 1]), m2 = float(g.metric[3 * r + 2]);
  const float V = fmaf(m2, w, fmaf(m1, v, m0 * u)), pr = (float(gamma) - 1.0f) * rho * ei;
  const float H = fmaf(rho, fmaf(0.5f, fmaf(w, w, fmaf(v, v, u * u)), ei), pr);
  const float x = n == 1 ? u : (n == 2 ? v : w), mn = n == 1 ? m0 : (n == 2 ? m1 : m2);
  g.c[k] = flux_constant(n == 0 ? rho * V : (n == 4 ? H * V : fmaf(rho * V, x, pr * mn)));
  if (k == 0) g.mean[0] = flux_constant(pr);
}

// One element: state, projected gradients, stresses, volume flux, its
// projected divergence (a.Pv, [e][n][L^3]) and the viscous normal-flux
// traces (a.V).  NODAL: the state comes from GLL values (a.Xn).  F32: the
// gradients and stresses in FP32 (precision = DGMX_MIXED); the primitive
// variables are formed in FP64 and rounded as their differences from the
// element's middle point (constants the gradient does not see: for the internal
// energy 1/(gamma (gamma-1) Ma^2) against variations of O(1)).
template <class C, int PHYS, bool NODAL, bool F32>
__global__ void __launch_bounds__(C::NT, C::MINB) ns_flux_kernel(StageArgs a) {
  using N = NsFlux<C>;
  constexpr int L = C::L, Q = C::Q, G = C::G, GF = C::GF, BS = C::BS, SI = C::SI, SJ = C::SJ, NT = C::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *U = reinterpret_cast<double *>(smem_raw), *W = U + N::O_W, *X = U + N::O_X;
  Geo3 &g = *reinterpret_cast<Geo3 *>(smem_raw + N::DATA);
  const int tid = threadIdx.x, e = a.vtiles ? a.vtiles[blockIdx.x] : (int)blockIdx.x;
  // links and geometry arrive behind the state's first passes
  pdl_release();
  f3_load_links<C>(g, a, e, tid);
  pdl_wait();
  if constexpr (NODAL) f3_state_nodal<C>(U, g.mean, a, e, tid); else f3_state_k<C>(U, nullptr, a, e, tid);
  if (const int n = element_ahead<C>(a, e); n >= 0) {
    if constexpr (!NODAL) prefetch_span<NT>(a.X + (size_t)n * 5 * C::LD, 5 * C::LD * 8, tid);
    prefetch_span<NT>(a.Tin + (size_t)n * 30 * GF, 30 * GF * 8, tid);
  }
  __syncthreads();
  f3_load_geo<C>(g, a, tid);
  prefetch_neighbours<C>(g, a.Tin, 5 * GF, tid);
  if constexpr (!NODAL) f3_expand_j<C>(U, 5, tid);
  __syncthreads();
  ns3_jumps<C, F32>(X, g, a, e, tid);
  if constexpr (!NODAL) f3_expand_i<C>(U, 5, tid);
  __syncthreads();
  if constexpr (F32) f3_lift_rows<C>(reinterpret_cast<F2 *>(X), 12, tid);
  else f3_lift_rows<C>(X, 24, tid);
  // density, velocity, internal energy in place
  for (int w = tid; w < Q * Q * Q; w += NT) {
    const int i = w / (Q * Q), jk = w - i * Q * Q, j = jk / Q, k = jk - j * Q;
    double *p = U + i * SI + j * SJ + k;
    double u[5], q[4];
#pragma unroll
    for (int n = 0; n < 5; ++n) u[n] = p[n * BS];
    const double ir = 1.0 / u[0];
    q[0] = u[1] * ir; q[1] = u[2] * ir; q[2] = u[3] * ir;
    q[3] = fma(-0.5, fma(q[2], q[2], fma(q[1], q[1], q[0] * q[0])), u[4] * ir);
#pragma unroll
    for (int n = 0; n < 4; ++n) p[(n + 1) * BS] = q[n];
  }
  __syncthreads();
  const double kap = a.gamma / a.Pr * a.vis;
  constexpr int MID = (Q / 2) * (SI + SJ + 1);
  if (tid >= NT - 15) ns3_flux_constants<C>(U + MID, g, a.gamma, tid - (NT - 15));
  if constexpr (F32) {
    F2 *W2 = reinterpret_cast<F2 *>(W), *X2 = reinterpret_cast<F2 *>(X);
    f3_lift_cols<C>(X2, X2, 12, tid);
    // gradient of the pairs (u, v) and (w, e), pair c in W2[3c .. 3c+2]
    pencils_i<C>(2, tid, [&](int c, int jk) {
      const double *f = U + (1 + 2 * c) * BS, r0 = f[MID], r1 = f[BS + MID];
      F2 v[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        const double *p = f + jk + i * SI;
        v[i] = F2(float(p[0] - r0), float(p[BS] - r1));
      }
      ns3_grad_i<C>(v, W2 + 3 * c * BS + jk, W2 + (3 * c + 1) * BS + jk);
    });
    __syncthreads();
    pencils_j<C>(2, tid, [&](int c, int o, int, int) {
      F2 *w = W2 + 3 * c * BS + o;
      ns3_grad_j<C>(w, w + BS, w, w + BS, w + 2 * BS);
    });
    __syncthreads();
    pencils_k<C>(2, tid, [&](int c, int o, int aa, int bb) {
      F2 *w = W2 + 3 * c * BS + o;
      F2 z[3][L];
      ns3_grad_k<C>(w, X2 + c * 6 * C::XLS, g.metric, aa, bb, z);
#pragma unroll
      for (int d = 0; d < 3; ++d) st_pencil<L>(w + d * BS, 1, z[d]);
    });
    __syncthreads();
    // stresses and heat flux (modal) as pairs (t11, t12), (t13, t22),
    // (t23, t33), (hx, hy), (hz, 0)
    for (int w = tid; w < L * L * L; w += NT) {
      const int i = w / (L * L), jk = w - i * L * L, j = jk / L, k = jk - j * L;
      F2 *p = W2 + i * SI + j * SJ + k;
      F2 q[6];
#pragma unroll
      for (int n = 0; n < 6; ++n) q[n] = p[n * BS];
      const float gr[9] = {q[0].x, q[1].x, q[2].x, q[0].y, q[1].y, q[2].y, q[3].x, q[4].x, q[5].x};
      const float kf = float(kap);
      float t[6];
      viscous_stress<3, float>(gr, 1, float(a.vis), t);
      p[0] = F2(t[0], t[1]); p[BS] = F2(t[2], t[3]); p[2 * BS] = F2(t[4], t[5]);
      p[3 * BS] = F2(kf * q[3].y, kf * q[4].y); p[4 * BS] = F2(kf * q[5].y, 0.0f);
    }
    __syncthreads();
    f3_expand_k<C>(W2, 5, tid);
    __syncthreads();
    f3_expand_j<C>(W2, 5, tid);
    __syncthreads();
    f3_expand_i<C>(W2, 5, tid);
    __syncthreads();
  } else {
    f3_lift_cols<C>(X, X, 24, tid);
    // velocity gradient: component c in W[3c .. 3c+2]
    pencils_i<C>(3, tid, [&](int c, int jk) {
      double v[Q];
      ld_pencil<Q>(U + (1 + c) * BS + jk, SI, v);
      ns3_grad_i<C>(v, W + 3 * c * BS + jk, W + (3 * c + 1) * BS + jk);
    });
    __syncthreads();
    pencils_j<C>(3, tid, [&](int c, int o, int, int) {
      double *w = W + 3 * c * BS + o;
      ns3_grad_j<C>(w, w + BS, w, w + BS, w + 2 * BS);
    });
    __syncthreads();
    pencils_k<C>(3, tid, [&](int c, int o, int aa, int bb) {
      double *w = W + 3 * c * BS + o;
      double z[3][L];
      ns3_grad_k<C>(w, X + c * 6 * C::XLS, g.metric, aa, bb, z);
#pragma unroll
      for (int d = 0; d < 3; ++d) st_pencil<L>(w + d * BS, 1, z[d]);
    });
    __syncthreads();
    // stresses (modal, linear in the gradient) into W[0..5]; the energy
    // gradient's i pass into W[9] and the velocity jumps' part of X
    double *A0 = X;
    for (int w = tid; w < L * L * L; w += NT) {
      const int i = w / (L * L), jk = w - i * L * L, j = jk / L, k = jk - j * L;
      double *p = W + i * SI + j * SJ + k;
      double t[6];
      viscous_stress<3, double>(p, BS, a.vis, t);
#pragma unroll
      for (int n = 0; n < 6; ++n) p[n * BS] = t[n];
    }
    pencils_i<C>(1, tid, [&](int, int jk) {
      double v[Q];
      ld_pencil<Q>(U + 4 * BS + jk, SI, v);
      ns3_grad_i<C>(v, W + 9 * BS + jk, A0 + jk);
    });
    __syncthreads();
    pencils_j<C>(1, tid, [&](int, int o, int, int) {
      double *w = W + 6 * BS + o;
      ns3_grad_j<C>(W + 9 * BS + o, A0 + o, w, w + BS, w + 2 * BS);
    });
    f3_expand_k<C>(W, 6, tid);
    __syncthreads();
    pencils_k<C>(1, tid, [&](int, int o, int aa, int bb) {
      double *w = W + 6 * BS + o;
      double z[3][L], u[Q];
      ns3_grad_k<C>(w, X + 18 * C::XLS, g.metric, aa, bb, z);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int c = 0; c < L; ++c) z[d][c] *= kap;
        eo_expand<L, Q>(z[d], u);
        st_pencil<Q>(w + d * BS, 1, u);
      }
    });
    f3_expand_j<C>(W, 6, tid);
    __syncthreads();
    f3_expand_j<C>(W + 6 * BS, 3, tid);
    f3_expand_i<C>(W, 6, tid);
    __syncthreads();
    f3_expand_i<C>(W + 6 * BS, 3, tid);
    __syncthreads();
  }
  // contravariant flux G_r = metric[r] . (F(U) - g) at the points, and the
  // viscous normal flux g . n on the face points
  {
    const double gm1 = a.gamma - 1.0;
    double m[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) m[k] = g.metric[k];
    for (int w = tid; w < Q * Q * Q; w += NT) {
      const int i = w / (Q * Q), jk = w - i * Q * Q, j = jk / Q, k = jk - j * Q;
      double *p = U + i * SI + j * SJ + k;
      const double rho = p[0], u = p[BS], v = p[2 * BS], ww = p[3 * BS], ei = p[4 * BS];
      double t[9];   // t11, t12, t13, t22, t23, t33, heat flux
      if constexpr (F32) {
        const F2 *q = reinterpret_cast<const F2 *>(p + 5 * BS);
#pragma unroll
        for (int n = 0; n < 5; ++n) {
          const F2 z = q[n * BS];
          t[2 * n] = z.x;
          if (n < 4) t[2 * n + 1] = z.y;
        }
      } else {
#pragma unroll
        for (int n = 0; n < 9; ++n) t[n] = p[(5 + n) * BS];
      }
      const double t11 = t[0], t12 = t[1], t13 = t[2], t22 = t[3], t23 = t[4], t33 = t[5];
      const double qx = fma(t13, ww, fma(t12, v, fma(t11, u, t[6])));
      const double qy = fma(t23, ww, fma(t22, v, fma(t12, u, t[7])));
      const double qz = fma(t33, ww, fma(t23, v, fma(t13, u, t[8])));
      // Less the element's constants (pencil.cuh): all of them on GLL values up
      // to p = 5; in stages, where the update of the state rounds more, those
      // that low Mach numbers make large (the pressure, which costs nothing,
      // and the energy flux)
      constexpr bool ALL = NODAL && L <= 6;
      const double gr = gm1 * rho, q2 = fma(ww, ww, fma(v, v, u * u));
      double pr, pd, H;   // pressure, pressure less the constant, E + p
      if constexpr (ALL) {
        // from the energy itself: by way of the internal energy it is rounded
        // three times more, on GLL values 1.25 times the error at p = 4
        const double E = a.Xn[((size_t)4 * a.ne + e) * C::QD + w];
        pr = pd = gm1 * fma(-0.5 * rho, q2, E);
        H = E + pr;
      } else {
        pr = gr * ei;
        pd = fma(gr, ei, -g.mean[0]);
        H = fma(rho, fma(0.5, q2, ei), pr);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double m0 = m[3 * r], m1 = m[3 * r + 1], m2 = m[3 * r + 2];
        const double V = fma(m2, ww, fma(m1, v, m0 * u)), rV = rho * V;
        const double wx = fma(m2, t13, fma(m1, t12, m0 * t11)), wy = fma(m2, t23, fma(m1, t22, m0 * t12));
        const double wz = fma(m2, t33, fma(m1, t23, m0 * t13)), we = fma(m2, qz, fma(m1, qy, m0 * qx));
        double *o = p + 5 * r * BS;
        const volatile double *c = g.c + 5 * r;
        o[0] = ALL ? fma(rho, V, -c[0]) : rV;
        o[BS] = fma(rV, u, fma(pd, m0, -(ALL ? c[1] + wx : wx)));
        o[2 * BS] = fma(rV, v, fma(pd, m1, -(ALL ? c[2] + wy : wy)));
        o[3 * BS] = fma(rV, ww, fma(pd, m2, -(ALL ? c[3] + wz : wz)));
        o[4 * BS] = fma(H, V, -c[4]) - we;
        const int idx = r == 0 ? i : (r == 1 ? j : k);
        if (idx == 0 || idx == Q - 1) {
          const int f = idx == 0 ? (r == 0 ? 4 : (r == 1 ? 1 : 0)) : (r == 0 ? 2 : (r == 1 ? 3 : 5));
          const int x = r == 0 ? j : i, y = r == 2 ? j : k;
          double *fv = X + f * 4 * C::FVS + x * SJ + y;
          const double s = g.tv[f];
          fv[0] = s * wx; fv[C::FVS] = s * wy; fv[2 * C::FVS] = s * wz; fv[3 * C::FVS] = s * we;
        }
      }
    }
  }
  __syncthreads();
  f3_div_i<C>(U, tid);
  for (int w = tid; w < 24 * Q; w += NT) {   // face values -> Gauss points along y
    double *p = X + (w / Q) * C::FVS + (w % Q) * SJ;
    double v[Q], u[G];
    ld_pencil<Q>(p, 1, v);
#pragma unroll
    for (int h = 0; h < G; ++h) {
      double acc = 0.0;
#pragma unroll
      for (int y = 0; y < Q; ++y) acc = fma(cGL2G<double, L, Q>[h * Q + y], v[y], acc);
      u[h] = acc;
    }
    st_pencil<G>(p, 1, u);
  }
  __syncthreads();
  f3_div_j<C>(U, tid);
  for (int w = tid; w < 24 * G; w += NT) {   // and along x, to global memory
    const int fn = w / G, h = w - fn * G;
    double v[Q];
    ld_pencil<Q>(X + fn * C::FVS + h, SJ, v);
    double *dst = a.V + ((size_t)e * 24 + fn) * GF + h;
#pragma unroll
    for (int q = 0; q < G; ++q) {
      double acc = 0.0;
#pragma unroll
      for (int x = 0; x < Q; ++x) acc = fma(cGL2G<double, L, Q>[q * Q + x], v[x], acc);
      dst[q * G] = acc;
    }
  }
  __syncthreads();
  pencils_k<C>(5, tid, [&](int n, int o, int aa, int bb) {
    double y[L];
    f3_div_k_row<C>(U, n, o, y);
    st_row<L>(a.Pv + ((((size_t)e * 5 + n) * L + aa) * L + bb) * L, y);
  });
}

// Face terms (inviscid and viscous) of one element, the stage update from
// the volume part ns_flux_kernel left in a.Pv, and the next traces.  NODAL:
// the projected right-hand side goes to GLL values (a.Fn) instead.
// Shared memory: the right-hand side and then the next state UB, whose place
// the traces' first pass W1 takes; the face terms XL, whose place the end
// planes FP take.
template <class C, bool NODAL>
struct NsUpdate {
  static constexpr int SB = NODAL ? C::SJ : C::PL, SA = NODAL ? C::SI : C::L * C::PL;
  static constexpr int SN = NODAL ? C::BS : C::L * C::L * C::PL;
  static constexpr int S_UB = cmax(5 * SN, C::S_W1), O_X = S_UB, S_X = cmax(C::S_XL, C::S_FP);
  static constexpr size_t DATA = (size_t)(O_X + S_X) * sizeof(double);
  static constexpr size_t SMEM = DATA + (sizeof(Geo3) + 15) / 16 * 16;
};
template <class C, int PHYS, bool NODAL>
__global__ void __launch_bounds__(C::NT, C::MINB) ns_update_kernel(StageArgs a) {
  using N = NsUpdate<C, NODAL>;
  constexpr int L = C::L, GF = C::GF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *UB = reinterpret_cast<double *>(smem_raw), *X = UB + N::O_X;
  Geo3 &g = *reinterpret_cast<Geo3 *>(smem_raw + N::DATA);
  const int tid = threadIdx.x;
  pdl_release();
  const int ntile = a.tiles ? *a.ntiles : a.ne;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    const int e = a.tiles ? a.tiles[t] : t;
    if (t != (int)blockIdx.x) __syncthreads();
    f3_load_links<C>(g, a, e, tid);
    pdl_wait();
    // read five intervals on
    prefetch_span<C::NT>(a.Pv + (size_t)e * 5 * C::LD, 5 * C::LD * 8, tid);
    if constexpr (!NODAL) {
      prefetch_span<C::NT>(a.X + (size_t)e * 5 * C::LD, 5 * C::LD * 8, tid);
      prefetch_span<C::NT>(a.Ut + (size_t)e * 5 * C::LD, 5 * C::LD * 8, tid);
    }
    __syncthreads();
    f3_load_geo<C>(g, a, tid);
    prefetch_neighbours<C>(g, a.Tin, 5 * GF, tid);
    prefetch_neighbours<C>(g, a.V, 4 * GF, tid);
    __syncthreads();
    f3_faces<C, PHYS>(X, g, nullptr, a, e, tid);
    __syncthreads();
    f3_lift_rows<C>(X, 30, tid);
    __syncthreads();
    f3_lift_cols<C>(X, X, 30, tid);
    __syncthreads();
    for (int w = tid; w < 5 * L * L; w += C::NT) {
      const int n = w / (L * L), ab = w - n * L * L, aa = ab / L, bb = ab - aa * L;
      double R[L];
      zero<L>(R);
      if constexpr (NODAL) ld_row<L>(a.Pv + ((size_t)e * 5 * L * L + w) * L, R);
      f3_add_faces<C>(X, 5, n, aa, bb, R);
      double *u = UB + n * N::SN + aa * N::SA + bb * N::SB;
      if constexpr (NODAL) {
        if (a.R0 && ab == 0) a.R0[(size_t)e * 5 + n] = R[0];
        double v[C::Q];
        eo_expand<L, C::Q>(R, v);
        st_pencil<C::Q>(u, 1, v);
      } else {
        st_pencil<L>(u, 1, R);
      }
    }
    __syncthreads();
    if constexpr (NODAL) {
      f3_expand_j<C>(UB, 5, tid);
      __syncthreads();
      f3_store_nodal<C>(UB, a, e, tid);
    } else {
      f3_update_all<C>(UB, N::SN, N::SA, N::SB, a.Pv, a, e, tid);
      __syncthreads();
      f3_ends<C>(UB, N::SN, N::SA, N::SB, X, tid);
      __syncthreads();
      f3_traces_a<C>(X, UB, tid);
      __syncthreads();
      f3_traces_b<C>(UB, a.Tout, e, tid);
    }
  }
}

}  // namespace dgmx
