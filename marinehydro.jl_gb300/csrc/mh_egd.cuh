// mh_egd.cuh -- the exact Guevel-Delhommeau wave term and its r-derivative, one thread per pair.
//
// _dimless_wave_term and _d_dimless_wave_term_dr (exact_Guevel_Delhommeau.jl:15-46) are the
// integrals over theta of e^zeta (E1(zeta)/pi + i), zeta = z + i r cos(theta).  With
// e^zeta E1(zeta) = int_0^inf e^-u / (u + zeta) du the theta integral is elementary, and with
// Y = -z (Newman, "Algorithms for the free-surface Green function", J. Eng. Math. 19, 1985;
// DLMF 11.5.2 for H0 - Y0):
//     Re G = -e^-Y [ pi (H0(r) + Y0(r)) + 2 I ],   I = int_0^Y e^t / sqrt(t^2 + r^2) dt,
//     Im G = 2 pi e^-Y J0(r),   Im dG/dr = -2 pi e^-Y J1(r),
// and dG/dr the r-derivative of the first line.  What is left is one finite smooth integral, so
// the adaptive Gauss-Kronrod quadrature of a complex exponential integral (one warp per pair,
// some 5000 FP64 instructions for each) becomes one thread per pair with at most ~550 FP64
// instructions, its exponentials, square roots, logarithms and Bessel polynomials on the integer
// pipe (mh_fixpoint.cuh).  The kernels stay bound by the FP64 pipe (two lanes per SM and clock).  S and
// D of a 900-panel hemisphere into device buffers: 44.8 ms with the quadrature, 0.37 ms so.
//
// * I over [a, Y] by Gauss-Legendre: e^(t - Y) makes everything below Y - 38 vanish, so the
//   interval is at most 38 long; 18 nodes up to a length of 22, 24 above (the integrand's
//   singularities t = +-i r stay at least 3, or half the interval, from where e^(t - Y) counts;
//   measured against 40-digit references over r in [1e-6, 500], Y in [1e-5, 300]: 1.1e-15
//   relative to |G| + 2/d).
// * Where r < 3 and r < Y/2 the part over [0, a], a = min(Y, 3), is summed as the power series
//   of e^t with M_m = int_0^a t^m / sqrt(t^2 + r^2) dt from their recurrence (stable for r < a),
//   q_m = M_m / m!:  q_m = (a^(m-1)/(m-1)! d_a - r^2 q_(m-2)) / m^2,  d_a = sqrt(a^2 + r^2).  The
//   logarithm M_0 = asinh(a/r) joins Y0's: 2 asinh(a/r) + 2 lam J0 =
//   2 log((a + d_a)/2) + 2 gamma + 2 lam (J0 - 1), lam = log(r/2) + gamma, and likewise for the
//   1/r poles of the derivative, so no term grows as r -> 0.
// * J0, J1 and the entire parts F0, F1 of pi (H0 + Y0), pi (H0' + Y0') from half-unit tables
//   below r = 8 (namespace egdq); above, Hankel's forms and H - Y as polynomials in (8/r)^2.
//
// Points above the surface (z > 0) and the surface's own r = z = 0 take the adaptive quadrature at
// the caller's tolerances, which the closed form undercuts everywhere else.  It runs one warp per
// point (egd_warp): the kernels go over their points twice, thread by thread for the closed form
// and warp by warp for the others, few or none as a rule.  (One thread per point with a refinement
// stack of its own made 8192 points above the surface 295 ms instead of 15.7, and reserved 300 MB of
// local memory for every kernel of the exact term.)
#pragma once

#include <cuda_runtime.h>

#include "mh_greens.cuh"

namespace mh {

constexpr double kEulerGamma = 0.57721566490153286061;

// sums over the nodes of a Gauss-Legendre rule on [Y - h, Y], without the factor h:
// A = sum w e^(t - Y) / sqrt(t^2 + r^2), B = sum w e^(t - Y) (t^2 + r^2)^(-3/2)
template <int N>
__device__ __forceinline__ void egd_gauss(const double (&rule)[N][2], double Y, double h, double r2, double& A,
                                          double& B) {
#pragma unroll 2
  for (int i = 0; i < N; ++i) {
    const double hc = h * rule[i][0];
    const double t = Y - hc;
    const double rs = fx::rsqrt_pos(fma(t, t, r2));
    const double w = rule[i][1] * fx::exp_nonpos(-hc) * rs;
    A += w;
    B = fma(w, rs * rs, B);
  }
}

constexpr double kDoubleMax = 1.7976931348623157e308;

// finite points that the closed form does not cover
__device__ __forceinline__ bool egd_takes_quadrature(double r, double z) {
  if (z <= 0.0 && r >= 0.0 && r - z > 1e-140) return false;
  return fabs(r) <= kDoubleMax && fabs(z) <= kDoubleMax;
}

// G and dG/dr at a point (r, z) of that kind for a pair of panels, by the whole warp (the same r and
// z on every lane; sw: 8 kGKWarpStack doubles of shared memory of this warp).  Vertically stacked
// centres: the integrand does not depend on theta (zeta = z), so 4 times its integral over
// [0, pi/2] is 2 pi times its value; the r-derivative is not needed (the horizontal gradient
// vanishes for r <= 1e-6).
__device__ static __noinline__ void egd_pair_quadrature(double r, double z, double rtol, double atol, double* sw,
                                                        double2* G, double2* Gr) {
  if (r == 0.0) {
    double f[4];
    egd_integrands(0.0, 0.0, z, f);
    *G = make_double2(2.0 * kPi * f[0], 2.0 * kPi * f[1]);
    *Gr = make_double2(0.0, 0.0);
    return;
  }
  egd_warp(r, z, rtol, atol, sw, *G, *Gr);
}

// work(q) by the whole warp for those q of [0, m) with need(q); the warps of the grid's x direction
// share the range, at most 32 neighbours per warp and turn
template <typename Need, typename Work>
__device__ __forceinline__ void for_items_by_warp(int64_t m, Need need, Work work) {
  const int lane = threadIdx.x & 31;
  const int64_t per_cta = blockDim.x >> 5, warps = gridDim.x * per_cta;
  const int64_t each = (m + warps - 1) / warps, group = each < 32 ? each : 32;
  for (int64_t q0 = (blockIdx.x * per_cta + (threadIdx.x >> 5)) * group; q0 < m; q0 += warps * group) {
    unsigned todo = __ballot_sync(0xffffffffu, lane < group && q0 + lane < m && need(q0 + lane));
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      work(q0 + src);
      __syncwarp();
    }
  }
}

__device__ __forceinline__ bool egd_pair_takes_quadrature(const double* x, const double* xi, double k) {
  double r, z;
  reduced_coords(x, xi, k, r, z);
  return egd_takes_quadrature(r, z);
}

// false where no pair of the mesh takes the quadrature, as a rule: every centre below kBelowSurface
__device__ __forceinline__ bool egd_any_quadrature(const AssemblyParams& p, double k) {
  return !p.above || *p.above != 0 || !(k > 1e-100);
}

// G and dG/dr in closed form (NaN where r or z is not finite); for every point but those of
// egd_takes_quadrature
__device__ inline void egd_values(double r, double z, double2& G, double2& Gr) {
  const double Y = -z;
  if (!(fabs(r) + fabs(z) <= kDoubleMax)) {
    const double nan = __longlong_as_double(0x7FF8000000000000LL);
    G = Gr = make_double2(nan, nan);
    return;
  }
  const double r2 = r * r;
  const double e = fx::exp_nonpos(z);
  const bool near = r < 3.0 && 2.0 * r < Y;
  const double a = near ? fmin(Y, 3.0) : 0.0;
  const double h = fmin(Y - a, 38.0);
  double A = 0.0, B = 0.0;
  if (h > 0.0) {
    if (h <= 22.0) egd_gauss(egdq::kGl18, Y, h, r2, A, B);
    else egd_gauss(egdq::kGl24, Y, h, r2, A, B);
    A *= h;
    B *= h * r;
  }
  double J0, J1, S0, S1;  // S0 = pi (H0 + Y0), S1 = pi (H0' + Y0'), with the [0, a] part where near
  if (r < 8.0) {
    const long long X = fx::to_q(r, 60);
    const int q = (int)(X >> 59);
    const long long zq = (X - (((long long)q << 59) + (1ll << 58))) << 5;
    const int row = q * bes::kLowTerms;
    J0 = fx::to_double(fx::horner_s_ld<bes::kLowTerms>(besq::kJ0 + row, zq), besq::kFrac);
    J1 = fx::to_double(fx::horner_s_ld<bes::kLowTerms>(besq::kJ1 + row, zq), besq::kFrac);
    const double F0 = fx::to_double(fx::horner_s_ld<bes::kLowTerms>(egdq::kF0 + row, zq), egdq::kFrac);
    const double F1 = fx::to_double(fx::horner_s_ld<bes::kLowTerms>(egdq::kF1 + row, zq), egdq::kFrac);
    const double rp = fmax(r, 1e-290);
    const double lr = fx::log_pos(0.5 * rp);
    const double lam = lr + kEulerGamma;
    if (near) {
      const double da = fx::sqrt_pos(fma(a, a, r2));
      const double la = fx::log_pos(0.5 * (a + da));
      double q2 = la - lr, q1 = da - r, y = a;  // q_(m-2), q_(m-1), a^(m-1)/(m-1)!
      double sa = q1, sb = fma(q1, 1.0 / 3.0, 0.5 * q2), sy = 0.0;
      for (int m = 2; m < 48 && y > 1e-18; ++m) {
        const double im = kInvN.v[m];
        sy = fma(y, im, sy);
        const double qm = fma(-r2, q2, y * da) * (im * im);
        y *= a * im;
        q2 = q1;
        q1 = qm;
        sa += qm;
        sb = fma(qm, kInvN.v[m + 2], sb);
      }
      S0 = F0 + 2.0 * (la + kEulerGamma + lam * (J0 - 1.0) + sa);
      S1 = F1 + 2.0 * (fma(r * fx::recip(da), 1.0 + sy + fx::recip(a + da), -lam * J1) - r * sb);
    } else {
      S0 = fma(2.0 * lam, J0, F0);
      S1 = F1 + 2.0 * (1.0 + fx::recip(rp) - lam * J1);
    }
  } else {
    double Y0, Y1;
    bessel01(r, J0, J1, Y0, Y1);
    const double ir = fx::recip(r), s = 8.0 * ir;
    const long long zq = fx::to_q(fmin(fma(s, s, -0.5), 0.49999999999999989), 64);
    S0 = 2.0 * fma(kPi, Y0, ir * fx::to_double(fx::horner_s(egdq::kS0, zq), egdq::kFrac));
    S1 = fma(-2.0 * kPi, Y1, fx::to_double(fx::horner_s(egdq::kS1, zq), egdq::kFrac));
  }
  const double pe = 2.0 * kPi * e;
  G = make_double2(-fma(e, S0, 2.0 * A), pe * J0);
  Gr = make_double2(fma(-e, S1, 2.0 * B), -pe * J1);
}

}  // namespace mh
