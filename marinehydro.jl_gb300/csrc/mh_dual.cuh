// mh_dual.cuh -- forward-mode dual numbers for the reverse (adjoint) kernels.
//
// Dn<M> carries a value and M partial derivatives.  The adjoint kernels evaluate
// the pair Green functions on Dn to obtain the exact derivatives of the code path
// the primal kernels run (the Wu polynomial/Struve fits, the Birk panel
// integral), the way the reference differentiates them with ForwardDiff / Enzyme
// (ad_rules.jl:79-294).  Derivatives of the special functions:
//   d j0 = -j1, d j1 = j0 - j1/x, d y0 = -y1, d y1 = y0 - y1/x.
#pragma once

#include <cuda_runtime.h>

#include "mh_bessel01.cuh"

namespace mh {

template <int M>
struct Dn {
  double v;
  double d[M];
  __device__ Dn() : v(0.0) {
#pragma unroll
    for (int q = 0; q < M; ++q) d[q] = 0.0;
  }
  __device__ Dn(double x) : v(x) {
#pragma unroll
    for (int q = 0; q < M; ++q) d[q] = 0.0;
  }
  __device__ static Dn var(double x, int slot) {
    Dn r(x);
    if (slot >= 0 && slot < M) r.d[slot] = 1.0;
    return r;
  }
};

template <int M> __device__ __forceinline__ double val(const Dn<M>& a) { return a.v; }
__device__ __forceinline__ double val(double a) { return a; }

// double overloads, so that unqualified calls inside namespace mh keep finding the CUDA math
// functions
__device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
__device__ __forceinline__ double log(double x) { return ::log(x); }
__device__ __forceinline__ double exp(double x) { return ::exp(x); }
__device__ __forceinline__ double hypot(double x, double y) { return ::hypot(x, y); }

// chain: r = f(a) with f'(a) = s
template <int M> __device__ __forceinline__ Dn<M> chain1(const Dn<M>& a, double fv, double s) {
  Dn<M> r(fv);
#pragma unroll
  for (int q = 0; q < M; ++q) r.d[q] = s * a.d[q];
  return r;
}

template <int M> __device__ __forceinline__ Dn<M> operator+(const Dn<M>& a, const Dn<M>& b) {
  Dn<M> r(a.v + b.v);
#pragma unroll
  for (int q = 0; q < M; ++q) r.d[q] = a.d[q] + b.d[q];
  return r;
}
template <int M> __device__ __forceinline__ Dn<M> operator-(const Dn<M>& a, const Dn<M>& b) {
  Dn<M> r(a.v - b.v);
#pragma unroll
  for (int q = 0; q < M; ++q) r.d[q] = a.d[q] - b.d[q];
  return r;
}
template <int M> __device__ __forceinline__ Dn<M> operator-(const Dn<M>& a) { return chain1(a, -a.v, -1.0); }
template <int M> __device__ __forceinline__ Dn<M> operator*(const Dn<M>& a, const Dn<M>& b) {
  Dn<M> r(a.v * b.v);
#pragma unroll
  for (int q = 0; q < M; ++q) r.d[q] = a.d[q] * b.v + a.v * b.d[q];
  return r;
}
// Divisions, square roots, exponentials and logarithms of the wave terms run on the integer pipe
// (mh_fixpoint.cuh; every divisor and argument there is positive, every exponent <= 0), within
// an ulp or two.  The panel frames' (birk_geometry_t) divisors take either sign: pos_recip.
static __device__ __noinline__ double pos_recip(double x) { return x > 0.0 ? fx::recip(x) : 1.0 / x; }
template <int M> __device__ __forceinline__ Dn<M> operator/(const Dn<M>& a, const Dn<M>& b) {
  const double inv = pos_recip(b.v), rv = a.v * inv;
  Dn<M> r(rv);
#pragma unroll
  for (int q = 0; q < M; ++q) r.d[q] = (a.d[q] - rv * b.d[q]) * inv;
  return r;
}
template <int M> __device__ __forceinline__ Dn<M> operator+(const Dn<M>& a, double b) { return chain1(a, a.v + b, 1.0); }
template <int M> __device__ __forceinline__ Dn<M> operator+(double b, const Dn<M>& a) { return chain1(a, b + a.v, 1.0); }
template <int M> __device__ __forceinline__ Dn<M> operator-(const Dn<M>& a, double b) { return chain1(a, a.v - b, 1.0); }
template <int M> __device__ __forceinline__ Dn<M> operator-(double b, const Dn<M>& a) { return chain1(a, b - a.v, -1.0); }
template <int M> __device__ __forceinline__ Dn<M> operator*(const Dn<M>& a, double b) { return chain1(a, a.v * b, b); }
template <int M> __device__ __forceinline__ Dn<M> operator*(double b, const Dn<M>& a) { return chain1(a, b * a.v, b); }
template <int M> __device__ __forceinline__ Dn<M> operator/(const Dn<M>& a, double b) {
  const double inv = 1.0 / b;
  return chain1(a, a.v * inv, inv);
}
template <int M> __device__ __forceinline__ Dn<M> operator/(double b, const Dn<M>& a) {
  const double inv = pos_recip(a.v), rv = b * inv;
  return chain1(a, rv, -rv * inv);
}
template <int M> __device__ __forceinline__ Dn<M>& operator+=(Dn<M>& a, const Dn<M>& b) { a = a + b; return a; }
template <int M> __device__ __forceinline__ Dn<M>& operator-=(Dn<M>& a, const Dn<M>& b) { a = a - b; return a; }

template <int M> __device__ __forceinline__ Dn<M> sqrt(const Dn<M>& a) {
  const double s = fx::sqrt_pos(a.v);
  return chain1(a, s, s > 0.0 ? 0.5 * fx::recip(s) : 0.0);
}
template <int M> __device__ __forceinline__ Dn<M> log(const Dn<M>& a) {
  return chain1(a, fx::log_pos(a.v), fx::recip(a.v));
}
template <int M> __device__ __forceinline__ Dn<M> exp(const Dn<M>& a) {  // a <= 0
  const double e = fx::exp_nonpos(a.v);
  return chain1(a, e, e);
}
}  // namespace mh
