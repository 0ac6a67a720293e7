// 1-D operators on a pencil held in registers, folded into even and odd parts
// (even-odd decomposition, Solomonoff 1992), and the tables of the weighted
// projections they use.
#pragma once

#include "stage.cuh"

namespace dgmx {

// Constant memory, per working type and (L, Q): the weighted derivative
// E = B W D and the lift projection BwG = B W G2GL (L rows each).
template <class T, int L, int Q> __constant__ T cE2[L * Q];          // E[a][j] = sum_i B[a][i] w_i D[i][j]
template <class T, int L, int Q> __constant__ T cBwG[L * (Q - 1)];   // BwG[a][g] = sum_i B[a][i] w_i G2GL[i][g]

// Two FP32 values that go through the same operator: a pair fills the slot of
// one FP64 value, so the FP32 viscous form keeps the FP64 layout (and its
// bank pattern) with half the buffers, loads and pencils.
struct F2 {
  float x, y;
  F2() = default;
  __device__ __forceinline__ F2(float v) : x(v), y(v) {}
  __device__ __forceinline__ F2(float a, float b) : x(a), y(b) {}
};
using ::fma;   // beside the overload for pairs
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ F2 fma(float c, F2 v, F2 a) { return F2(fmaf(c, v.x, a.x), fmaf(c, v.y, a.y)); }
template <class T> struct CoefOf { using type = T; };
template <> struct CoefOf<F2> { using type = float; };
template <class T> using coef_t = typename CoefOf<T>::type;

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
      acc[a] = fma(DER ? cE2<coef_t<T>, L, Q>[a * Q + i] : cBw<coef_t<T>, L, Q>[a * Q + i], sym ? s[i] : d[i], acc[a]);
  }
}
// out[i] = sum_a B[a][i] v[a]
template <int L, int Q, class T>
__device__ __forceinline__ void eo_expand(const T (&v)[L], T (&out)[Q]) {
#pragma unroll
  for (int i = 0; i < (Q + 1) / 2; ++i) {
    T e = T(0), o = T(0);
#pragma unroll
    for (int a = 0; a < L; a += 2) e = fma(cB<coef_t<T>, L, Q>[a * Q + i], v[a], e);
    if (i == Q / 2) { out[i] = e; continue; }   // odd modes vanish in the middle
#pragma unroll
    for (int a = 1; a < L; a += 2) o = fma(cB<coef_t<T>, L, Q>[a * Q + i], v[a], o);
    out[i] = e + o;
    out[Q - 1 - i] = e - o;
  }
}
// Constants taken out of an element's fluxes.  The projected divergence of a
// constant vanishes, but its rounding does not: P and E in place of the
// collocation derivative round the fluxes' mean about twice as much, the
// folding a tenth more (FP32, p = 2 to 7; with the flux of one state of the
// element taken out, a third to a tenth of the derivative-first form's error).
// Any finite constant is right; what is left of the mean is rounded as before.
template <class T>
__device__ __forceinline__ T flux_constant(T v) { return isfinite(v) ? v : T(0); }
// Contravariant flux metric[r] . F(U) of field n of an Euler state (m: the
// metric's row), one value per thread; FP32 will do for a constant.
template <int DIM>
__device__ __forceinline__ double flux_constant(const double *U, const double *m, double gamma, int n) {
  const float ir = __fdividef(1.0f, float(U[0]));
  float V = 0.0f, s = 0.0f, Un = float(U[0]), mn = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const float mom = float(U[1 + d]), u = mom * ir, md = float(m[d]);
    V = fmaf(md, u, V);
    s = fmaf(u, mom, s);
    if (n == 1 + d) { Un = mom; mn = md; }
  }
  const float E = float(U[DIM + 1]), p = (float(gamma) - 1.0f) * fmaf(-0.5f, s, E);
  if (n == DIM + 1) { Un = E; mn = V; }
  return double(flux_constant(fmaf(Un, V, p * mn)));
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

}  // namespace dgmx
