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

// Geometry of the element a CTA works on, in shared memory.
struct Geo3 {
  double metric[9];
  double tj[6];      // jump scale of face f: J_side/J_el with the sign of n . metric[r]
  double tv[6];      // normal scale: n = tv metric[r]
  double jr[6];
  double nrm[6][3], onrm[6][3];
  int master, bc;
  FaceLink lnk[6];
};
__device__ __forceinline__ int face_ax(int f) { return (f == 0 || f == 5) ? 2 : ((f == 1 || f == 3) ? 1 : 0); }

template <class C>
__device__ __forceinline__ void f3_load_geo(Geo3 &g, const StageArgs &a, int e, int tid) {
  const int cl = a.gclass[e];
  const GeomClass *gc = a.classes + (cl >= 0 ? cl : 0);
  if (tid < 9) g.metric[tid] = gc->metric[tid];
  if (tid < 18) {
    g.nrm[tid / 3][tid % 3] = gc->nrm[tid / 3][tid % 3];
    g.onrm[tid / 3][tid % 3] = gc->onrm[tid / 3][tid % 3];
  }
  if (tid < 6) {
    const double *m = gc->metric + 3 * face_ax(tid), *n = gc->onrm[tid];
    const double t = (n[0] * m[0] + n[1] * m[1] + n[2] * m[2]) / (m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
    g.tv[tid] = t;
    g.tj[tid] = t * gc->jr[tid];
    g.jr[tid] = gc->jr[tid];
    g.lnk[tid] = a.links[(size_t)e * 6 + tid];
  }
  if (tid == 0) { g.master = gc->master; g.bc = gc->bc; }
}

// ---- pencil operators --------------------------------------------------------
// Even-odd folding of a pencil of N values: s[i] = v[i] + v[N-1-i] (and the
// middle value at N/2 when N is odd), d[i] = v[i] - v[N-1-i].
template <int N, class T>
__device__ __forceinline__ void eo_fold(const T (&v)[N], T (&s)[(N + 1) / 2], T (&d)[N / 2 > 0 ? N / 2 : 1]) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) { s[i] = v[i] + v[N - 1 - i]; d[i] = v[i] - v[N - 1 - i]; }
  if constexpr (N % 2 == 1) s[N / 2] = v[N / 2];
}
// acc[a] += sum_i P[a][i] v[i] (DER false) or E[a][i] v[i] (DER true) from the
// folded pencil.
template <int L, int Q, bool DER, class T>
__device__ __forceinline__ void eo_project(const T (&s)[(Q + 1) / 2], const T (&d)[Q / 2], T (&acc)[L]) {
#pragma unroll
  for (int a = 0; a < L; ++a) {
    const bool sym = (a % 2 == 0) != DER;
#pragma unroll
    for (int i = 0; i < (sym ? (Q + 1) / 2 : Q / 2); ++i)
      acc[a] = fma(DER ? cE2<T, L, Q>[a * Q + i] : cBw<T, L, Q>[a * Q + i], sym ? s[i] : d[i], acc[a]);
  }
}
// out[i] = sum_a B[a][i] v[a]
template <int L, int Q, class T>
__device__ __forceinline__ void eo_expand(const T (&v)[L], T (&out)[Q]) {
#pragma unroll
  for (int i = 0; i < (Q + 1) / 2; ++i) {
    T e = T(0), o = T(0);
#pragma unroll
    for (int a = 0; a < L; a += 2) e = fma(cB<T, L, Q>[a * Q + i], v[a], e);
    if (i == Q / 2) { out[i] = e; continue; }   // odd modes vanish in the middle
#pragma unroll
    for (int a = 1; a < L; a += 2) o = fma(cB<T, L, Q>[a * Q + i], v[a], o);
    out[i] = e + o;
    out[Q - 1 - i] = e - o;
  }
}
template <int N, class T>
__device__ __forceinline__ void ld_pencil(const T *p, int st, T (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = p[i * st];
}
template <int N, class T>
__device__ __forceinline__ void st_pencil(T *p, int st, const T (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) p[i * st] = v[i];
}
template <int N, class T>
__device__ __forceinline__ void zero(T (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = T(0);
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
// k pass of the state from the modal rows in global memory (the mixed form
// takes the solve's reference state out of the constant mode first).
template <class C>
__device__ __forceinline__ void f3_state_k(typename C::R *buf, const StageArgs &a, int e, int tid) {
  using T = typename C::R;
  pencils_k<C>(C::NF, tid, [&](int n, int o, int aa, int b) {
    const int r = (n * C::L + aa) * C::L + b;
    double x[C::L];
    ld_row<C::L>(a.X + ((size_t)e * (C::NF * C::L * C::L) + r) * C::L, x);
    if constexpr (C::MIXED)
      if (aa == 0 && b == 0) x[0] -= a.uref[kUrefStride * solve_of(a, e) + 5 + n];
    T v[C::L], u[C::Q];
#pragma unroll
    for (int c = 0; c < C::L; ++c) v[c] = T(x[c]);
    eo_expand<C::L, C::Q>(v, u);
    st_pencil<C::Q>(buf + n * C::BS + o, 1, u);
  });
}
// GLL values of the state in Field layout [n][e][Q^3].
template <class C>
__device__ __forceinline__ void f3_state_nodal(double *buf, const StageArgs &a, int e, int tid) {
  constexpr int Q = C::Q, QD = C::QD;
  for (int w = tid; w < C::NF * QD; w += C::NT) {
    const int n = w / QD, p = w - n * QD, i = p / (Q * Q), jk = p - i * Q * Q, j = jk / Q, k = jk - j * Q;
    buf[n * C::BS + i * C::SI + j * C::SJ + k] = a.Xn[((size_t)n * a.ne + e) * QD + p];
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
      for (int h = 0; h < G; ++h) acc = fma(cBwG<T, L, Q>[b * G + h], v[h], acc);
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
      for (int g = 0; g < G; ++g) acc = fma(cBwG<T, L, Q>[b * G + g], v[g], acc);
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
    T *eo = X + f * NF * C::XLS + (q / G) * C::PF + q % G;
    const T jr = T(g.jr[f]);
    const T nm[3] = {T(g.nrm[f][0]), T(g.nrm[f][1]), T(g.nrm[f][2])};
    bool ok;
    if constexpr (C::MIXED) {
      T UL[5], UR[5], FR[5];
#pragma unroll
      for (int k = 0; k < NF; ++k) { UL[k] = master ? Uo[k] : Un[k]; UR[k] = master ? Un[k] : Uo[k]; }
      const int cl = a.gclass[e];
      ok = face_flux_pert<PHYS, T>(*ref, UL, UR, nm, T(a.gamma), a.flux, D, FR, a.classes[cl >= 0 ? cl : 0].fr[f]);
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
        if (!bt) {
          const double *vo = a.V + ((size_t)e * 6 + f) * (NF - 1) * GF + q;
          const double *vn = a.V + ((size_t)lk.elem * 6 + lk.face) * (NF - 1) * GF + gn;
#pragma unroll
          for (int k = 1; k < NF; ++k) D[k] = fma(0.5, vo[(k - 1) * GF] + vn[(k - 1) * GF], D[k]);
        }
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

// ---- stage update of one modal row -----------------------------------------------
// Every stage kind; the row of the next state that the traces are taken of
// comes back in nx.
template <class C>
__device__ __forceinline__ void f3_update_row(const StageArgs &a, int e, int n, int ab, const typename C::R (&Rr)[C::L],
                                              typename C::R (&nx)[C::L]) {
  constexpr int L = C::L;
  const size_t gi = (((size_t)e * C::NF + n) * L * L + ab) * L;
  const double dt = a.dts ? a.dts[solve_of(a, e)] : a.dt;
  double x[L];
  ld_row<L>(a.X + gi, x);
  if constexpr (C::MIXED) {
    const double ref0 = ab == 0 ? a.uref[kUrefStride * solve_of(a, e) + 5 + n] : 0.0;
    if (a.kind == kRHS) {
#pragma unroll
      for (int c = 0; c < L; ++c) { a.A[gi + c] = Rr[c]; nx[c] = float(c == 0 ? x[c] - ref0 : x[c]); }
      return;
    }
    float ut[L];
    double u[L];
    ld_row<L>(a.Utf + gi, ut);
    const float c0 = float(a.c0), mdt = -float(dt);
#pragma unroll
    for (int c = 0; c < L; ++c) {
      ut[c] = fmaf(mdt, Rr[c], c0 * ut[c]);
      u[c] = fma(a.c1, double(ut[c]), x[c]);
      nx[c] = float(c == 0 ? u[c] - ref0 : u[c]);
    }
    st_row<L>(a.Utf + gi, ut);
    st_row<L>(a.U + gi, u);
  } else {
    if (a.R0 && ab == 0) a.R0[(size_t)e * C::NF + n] = Rr[0];   // bulk-flow hold
    if (a.kind == kLSRK) {
      double ut[L];
      ld_row<L>(a.Ut + gi, ut);
#pragma unroll
      for (int c = 0; c < L; ++c) {
        ut[c] = fma(-dt, Rr[c], a.c0 * ut[c]);
        nx[c] = fma(a.c1, ut[c], x[c]);
      }
      st_row<L>(a.Ut + gi, ut);
      st_row<L>(a.U + gi, nx);
      return;
    }
    double u[L], acc[L];
    switch (a.kind) {
      case kTVD0:
#pragma unroll
        for (int c = 0; c < L; ++c) nx[c] = fma(-dt, Rr[c], x[c]);
        st_row<L>(a.Ut + gi, nx);
        break;
      case kTVD1:
        ld_row<L>(a.U + gi, u);
#pragma unroll
        for (int c = 0; c < L; ++c) nx[c] = fma(a.c0, u[c], a.c1 * fma(-dt, Rr[c], x[c]));
        st_row<L>(a.Ut + gi, nx);
        break;
      case kTVD2:
        ld_row<L>(a.U + gi, u);
#pragma unroll
        for (int c = 0; c < L; ++c) nx[c] = fma(a.c1, fma(-dt, Rr[c], x[c]), a.c0 * u[c]);
        st_row<L>(a.U + gi, nx);
        break;
      case kRK40:
#pragma unroll
        for (int c = 0; c < L; ++c) { nx[c] = fma(a.c0, Rr[c], x[c]); acc[c] = a.c1 * Rr[c]; }
        st_row<L>(a.Ut + gi, nx);
        st_row<L>(a.A + gi, acc);
        break;
      case kRK41:
        ld_row<L>(a.U + gi, u);
        ld_row<L>(a.A + gi, acc);
#pragma unroll
        for (int c = 0; c < L; ++c) { nx[c] = fma(a.c0, Rr[c], u[c]); acc[c] = fma(a.c1, Rr[c], acc[c]); }
        st_row<L>(a.Ut + gi, nx);
        st_row<L>(a.A + gi, acc);
        break;
      case kRK43:
        ld_row<L>(a.U + gi, u);
        ld_row<L>(a.A + gi, acc);
#pragma unroll
        for (int c = 0; c < L; ++c) nx[c] = fma(a.c0, fma(a.c1, Rr[c], acc[c]), u[c]);
        st_row<L>(a.U + gi, nx);
        break;
      default:   // kRHS
#pragma unroll
        for (int c = 0; c < L; ++c) { acc[c] = Rr[c]; nx[c] = x[c]; }
        st_row<L>(a.A + gi, acc);
        break;
    }
  }
}

// ---- next traces --------------------------------------------------------------------
// The next modal rows sit in buffers UB (rows of pitch SJ, planes of SI);
// their end values along c were written by the update.  Ends along b (faces
// 1, 3) and a (faces 4, 2) -> FP [f][n][a'][b'], rows of PL.
template <class C, class T>
__device__ __forceinline__ void f3_ends(const T *UB, T *FP, int tid) {
  constexpr int NF = C::NF, L = C::L, Q = C::Q, PL = C::PL, N = NF * L * L, PB = NF * C::FPS;
  for (int w = tid; w < 2 * N; w += C::NT) {
    const int ax = w / N, r = w - ax * N, n = r / (L * L), xy = r - n * L * L, x = xy / L, y = xy - x * L;
    T lo = T(0), hi = T(0);
    const T *ub = UB + n * C::BS;
    T *fp = FP + n * C::FPS + x * PL + y;
    const T *p = ax == 0 ? ub + x * C::SI + y : ub + x * C::SJ + y;
    const int st = ax == 0 ? C::SJ : C::SI;
#pragma unroll
    for (int b = 0; b < L; ++b) {
      const T v = p[b * st];
      lo = fma(cEnd<T, L, Q>[b], v, lo);
      hi = fma(cEnd<T, L, Q>[L + b], v, hi);
    }
    fp[(ax == 0 ? 1 : 4) * PB] = lo;
    fp[(ax == 0 ? 3 : 2) * PB] = hi;
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
// End values along c of one next row: faces 0 and 5.
template <class C, class T>
__device__ __forceinline__ void f3_ends_c(const T (&nx)[C::L], T *FP, int n, int aa, int bb) {
  constexpr int L = C::L, Q = C::Q;
  T f0 = T(0), f5 = T(0);
#pragma unroll
  for (int c = 0; c < L; ++c) {
    f0 = fma(cEnd<T, L, Q>[c], nx[c], f0);
    f5 = fma(cEnd<T, L, Q>[L + c], nx[c], f5);
  }
  T *fp = FP + n * C::FPS + aa * C::PL + bb;
  fp[0] = f0;
  fp[5 * C::NF * C::FPS] = f5;
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
  static_assert(24 * C::XLS <= 10 * C::BS, "the jumps fit the work buffers");
  // the energy gradient's first pass takes the part of X whose jumps
  // (velocity) are consumed by then as one more scratch buffer
  static_assert(18 * C::XLS >= (C::L - 1) * C::SI + C::Q * C::SJ, "scratch buffer of the energy gradient");
};

// (q_own + q_nbr)/2 - q_own of the primitive variables at the side Gauss
// points, times the face's jump scale, into blocks [c][f].
template <class C>
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
    double *o = J + f * C::XLS + (q / G) * C::PF + q % G;
    const double t = 0.5 * g.tj[f];
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c * 6 * C::XLS] = t * (qn[c] - qo[c]);
  }
}

// Gradient passes of one scalar: i pass, v -> (E_i v, P_i v).
template <class C>
__device__ __forceinline__ void ns3_grad_i(const double *q, double *de, double *pr) {
  constexpr int L = C::L, Q = C::Q;
  double v[Q], s[(Q + 1) / 2], d[Q / 2], o[L];
  ld_pencil<Q>(q, C::SI, v);
  eo_fold<Q>(v, s, d);
  zero<L>(o);
  eo_project<L, Q, true>(s, d, o);
  st_pencil<L>(de, C::SI, o);
  zero<L>(o);
  eo_project<L, Q, false>(s, d, o);
  st_pencil<L>(pr, C::SI, o);
}
// j pass: (E_i v, P_i v) -> (P_j E_i v, E_j P_i v, P_j P_i v)
template <class C>
__device__ __forceinline__ void ns3_grad_j(const double *de, const double *pr, double *o0, double *o1, double *o2) {
  constexpr int L = C::L, Q = C::Q;
  double v[Q], s[(Q + 1) / 2], d[Q / 2], o[L];
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
template <class C>
__device__ __forceinline__ void ns3_grad_k(const double *w0, const double *X, const double *met, int aa, int bb,
                                           double (&z)[3][C::L]) {
  constexpr int L = C::L, Q = C::Q, PF = C::PF, XLS = C::XLS;
  double v[Q], s[(Q + 1) / 2], d[Q / 2];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    ld_pencil<Q>(w0 + r * C::BS, 1, v);
    eo_fold<Q>(v, s, d);
    zero<L>(z[r]);
    if (r == 2) eo_project<L, Q, true>(s, d, z[r]); else eo_project<L, Q, false>(s, d, z[r]);
  }
  const double xk0 = X[aa * PF + bb], xk1 = X[5 * XLS + aa * PF + bb];
  const double *xj0 = X + XLS + aa * PF, *xj1 = X + 3 * XLS + aa * PF;
  const double *xi0 = X + 4 * XLS + bb * PF, *xi1 = X + 2 * XLS + bb * PF;
  const double eb0 = end_value<double, L, Q>(0, bb), eb1 = end_value<double, L, Q>(1, bb);
  const double ea0 = end_value<double, L, Q>(0, aa), ea1 = end_value<double, L, Q>(1, aa);
#pragma unroll
  for (int c = 0; c < L; ++c) {
    const double z0 = fma(ea1, xi1[c], fma(ea0, xi0[c], z[0][c]));
    const double z1 = fma(eb1, xj1[c], fma(eb0, xj0[c], z[1][c]));
    const double z2 = fma(cEnd<double, L, Q>[L + c], xk1, fma(cEnd<double, L, Q>[c], xk0, z[2][c]));
#pragma unroll
    for (int k = 0; k < 3; ++k) z[k][c] = fma(met[6 + k], z2, fma(met[3 + k], z1, met[k] * z0));
  }
}

// One element: state, projected gradients, stresses, volume flux, its
// projected divergence (a.Pv, [e][n][L^3]) and the viscous normal-flux
// traces (a.V).  NODAL: the state comes from GLL values (a.Xn).
template <class C, int PHYS, bool NODAL>
__global__ void __launch_bounds__(C::NT, C::MINB) ns_flux_kernel(StageArgs a) {
  using N = NsFlux<C>;
  constexpr int L = C::L, Q = C::Q, G = C::G, GF = C::GF, BS = C::BS, SI = C::SI, SJ = C::SJ, NT = C::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *U = reinterpret_cast<double *>(smem_raw), *W = U + N::O_W, *X = U + N::O_X;
  Geo3 &g = *reinterpret_cast<Geo3 *>(smem_raw + N::DATA);
  const int tid = threadIdx.x, e = a.vtiles ? a.vtiles[blockIdx.x] : (int)blockIdx.x;
  f3_load_geo<C>(g, a, e, tid);
  __syncthreads();
  if constexpr (NODAL) f3_state_nodal<C>(U, a, e, tid); else f3_state_k<C>(U, a, e, tid);
  ns3_jumps<C>(W, g, a, e, tid);
  __syncthreads();
  if constexpr (!NODAL) f3_expand_j<C>(U, 5, tid);
  f3_lift_rows<C>(W, 24, tid);
  __syncthreads();
  if constexpr (!NODAL) f3_expand_i<C>(U, 5, tid);
  f3_lift_cols<C>(W, X, 24, tid);
  __syncthreads();
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
  // velocity gradient: component c in W[3c .. 3c+2]
  pencils_i<C>(3, tid, [&](int c, int jk) {
    ns3_grad_i<C>(U + (1 + c) * BS + jk, W + 3 * c * BS + jk, W + (3 * c + 1) * BS + jk);
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
  pencils_i<C>(1, tid, [&](int, int jk) { ns3_grad_i<C>(U + 4 * BS + jk, W + 9 * BS + jk, A0 + jk); });
  __syncthreads();
  pencils_j<C>(1, tid, [&](int, int o, int, int) {
    double *w = W + 6 * BS + o;
    ns3_grad_j<C>(W + 9 * BS + o, A0 + o, w, w + BS, w + 2 * BS);
  });
  f3_expand_k<C>(W, 6, tid);
  __syncthreads();
  const double kap = a.gamma / a.Pr * a.vis;
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
      const double *t = p + 5 * BS;
      const double t11 = t[0], t12 = t[BS], t13 = t[2 * BS], t22 = t[3 * BS], t23 = t[4 * BS], t33 = t[5 * BS];
      const double qx = fma(t13, ww, fma(t12, v, fma(t11, u, t[6 * BS])));
      const double qy = fma(t23, ww, fma(t22, v, fma(t12, u, t[7 * BS])));
      const double qz = fma(t33, ww, fma(t23, v, fma(t13, u, t[8 * BS])));
      const double pr = gm1 * rho * ei;
      const double H = fma(rho, fma(0.5, fma(ww, ww, fma(v, v, u * u)), ei), pr);   // E + p
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const double m0 = m[3 * r], m1 = m[3 * r + 1], m2 = m[3 * r + 2];
        const double V = fma(m2, ww, fma(m1, v, m0 * u)), rV = rho * V;
        const double wx = fma(m2, t13, fma(m1, t12, m0 * t11)), wy = fma(m2, t23, fma(m1, t22, m0 * t12));
        const double wz = fma(m2, t33, fma(m1, t23, m0 * t13)), we = fma(m2, qz, fma(m1, qy, m0 * qx));
        double *o = p + 5 * r * BS;
        o[0] = rV;
        o[BS] = fma(rV, u, fma(pr, m0, -wx));
        o[2 * BS] = fma(rV, v, fma(pr, m1, -wy));
        o[3 * BS] = fma(rV, ww, fma(pr, m2, -wz));
        o[4 * BS] = fma(H, V, -we);
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
template <class C>
struct NsUpdate {
  static constexpr int O_X = 5 * C::BS, S_X = cmax(C::S_XL, C::S_W1), O_FP = O_X + S_X;   // W1 follows XL
  static constexpr size_t DATA = (size_t)(O_FP + C::S_FP) * sizeof(double);
  static constexpr size_t SMEM = DATA + (sizeof(Geo3) + 15) / 16 * 16;
};
template <class C, int PHYS, bool NODAL>
__global__ void __launch_bounds__(C::NT, C::MINB) ns_update_kernel(StageArgs a) {
  using N = NsUpdate<C>;
  constexpr int L = C::L;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *UB = reinterpret_cast<double *>(smem_raw), *X = UB + N::O_X, *FP = UB + N::O_FP;
  Geo3 &g = *reinterpret_cast<Geo3 *>(smem_raw + N::DATA);
  const int tid = threadIdx.x;
  const int ntile = a.tiles ? *a.ntiles : (int)gridDim.x;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    const int e = a.tiles ? a.tiles[t] : t;
    if (t != (int)blockIdx.x) __syncthreads();
    f3_load_geo<C>(g, a, e, tid);
    __syncthreads();
    f3_faces<C, PHYS>(X, g, nullptr, a, e, tid);
    __syncthreads();
    f3_lift_rows<C>(X, 30, tid);
    __syncthreads();
    f3_lift_cols<C>(X, X, 30, tid);
    __syncthreads();
    pencils_k<C>(5, tid, [&](int n, int o, int aa, int bb) {
      double R[L], nx[L];
      ld_row<L>(a.Pv + ((((size_t)e * 5 + n) * L + aa) * L + bb) * L, R);
      f3_add_faces<C>(X, 5, n, aa, bb, R);
      if constexpr (NODAL) {
        if (a.R0 && aa == 0 && bb == 0) a.R0[(size_t)e * 5 + n] = R[0];
        double u[C::Q];
        eo_expand<L, C::Q>(R, u);
        st_pencil<C::Q>(UB + n * C::BS + o, 1, u);
      } else {
        f3_update_row<C>(a, e, n, aa * L + bb, R, nx);
        st_pencil<L>(UB + n * C::BS + o, 1, nx);
        f3_ends_c<C>(nx, FP, n, aa, bb);
      }
    });
    __syncthreads();
    if constexpr (NODAL) {
      f3_expand_j<C>(UB, 5, tid);
      __syncthreads();
      f3_store_nodal<C>(UB, a, e, tid);
    } else {
      f3_ends<C>(UB, FP, tid);
      __syncthreads();
      f3_traces_a<C>(FP, X, tid);
      __syncthreads();
      f3_traces_b<C>(X, a.Tout, e, tid);
    }
  }
}

}  // namespace dgmx
