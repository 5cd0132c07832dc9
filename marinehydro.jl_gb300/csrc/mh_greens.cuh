// mh_greens.cuh -- device Green-function kernels of the MarineHydro.jl hot path (FP64).
//
// Each function restates the reference function cited beside it (paths within the
// MarineHydro.jl tree).  Elementary functions are CUDA's (exp, log, atan2, sqrt, hypot,
// sincos), except in the Wu term, whose exp, log and reciprocals run on the integer pipe
// (mh_fixpoint.cuh); the Bessel functions J0, J1, Y0, Y1 (mh_bessel01.cuh, Chebyshev and Hankel
// forms), the complex exponential integral and the Gauss-Kronrod rule are written from
// published methods (DLMF 10.17.3, 6.6.2, 6.9.1; Kronrod's 15-point nodes, QUADPACK qk15).
#pragma once

#include <cuda_runtime.h>

#include "mh_bessel01.cuh"
#include "mh_fixpoint.cuh"
#include "mh_internal.cuh"

namespace mh {

// ------------------------------- complex ------------------------------------
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
__device__ __forceinline__ double2 zexp(double2 a) {
  double s, c;
  sincos(a.y, &s, &c);
  double e = exp(a.x);
  return make_double2(e * c, e * s);
}

// ------------------------------- Birk Rankine -------------------------------
constexpr double kBirkZTol = 1e-14;   // rankine_vectorized.jl:24
constexpr double kBirkDkTol = 1e-14;  // rankine_vectorized.jl:25

// _abs_ad (rankine_vectorized.jl:30): -0.0 stays -0.0
__device__ __forceinline__ double abs_ad(double x) { return x < 0.0 ? -x : x; }

// birk_phi_and_velocity (rankine_vectorized.jl:241-267); lc = 4 local corners (x, y),
// edge = their 4 edge lengths (per panel, precomputed; the same hypot of the corner offsets).
// Square roots, reciprocals, logarithms and arc tangents run on the integer pipe
// (mh_fixpoint.cuh), and an edge's two arc tangents (den >= 0, so each lies in [-pi/2, pi/2])
// are taken as one: the argument of the product of one complex number with the other's
// conjugate is their difference.  About 170 FP64 instructions are left of some 700.
__device__ inline void birk_phi_and_velocity(double x, double y, double z, const double* lc, const double* edge,
                                             double& phi, double v[3]) {
  double sx[4], sy[4], r[4], e[4], h[4];
  const double z2 = z * z;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    sx[k] = x - lc[2 * k];
    sy[k] = y - lc[2 * k + 1];
    e[k] = sx[k] * sx[k] + z2;
    r[k] = fx::sqrt_pos(sy[k] * sy[k] + e[k]);
    h[k] = sx[k] * sy[k];
  }
  const bool inplane = fabs(z) <= kBirkZTol;  // _inplane_atan (:49-54)
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int kn = (k + 1) & 3;
    const double dk = edge[k];
    if (dk <= kBirkDkTol) continue;
    const double dx = lc[2 * kn] - lc[2 * k];
    const double dy = lc[2 * kn + 1] - lc[2 * k + 1];
    const double rsum = r[k] + r[kn];
    const double num = rsum - dk;
    const double w = num * fx::recip(rsum + dk);
    // on the edge itself num vanishes or rounds below zero: log's own answer
    const double log_term = num > 0.0 ? fx::log_pos(w) : log(w);
    const double lt_dk = log_term * fx::recip(dk);
    if (!inplane) {
      const double dxz = dx * z;
      double n1 = dy * e[k] - dx * h[k], d1 = dxz * r[k];
      double n2 = dy * e[kn] - dx * h[kn], d2 = dxz * r[kn];
      if (d1 < 0.0) { n1 = -n1; d1 = -d1; }  // _atan_ratio (:42-45): den's sign moved to num
      if (d2 < 0.0) { n2 = -n2; d2 = -d2; }
      s3 += fx::atan2_int(n1 * d2 - n2 * d1, d1 * d2 + n1 * n2);
    }
    s0 += (sx[k] * dy - sy[k] * dx) * lt_dk;
    s1 += dy * lt_dk;
    s2 -= dx * lt_dk;
  }
  s0 += z * s3;
  // a point or panel that is not finite (a collapsed panel's frame among them) shows in z; the integer
  // functions give a number whatever they are given
  if ((__double2hiint(z) & 0x7FF00000) == 0x7FF00000) s0 = s1 = s2 = s3 = z - z;
  phi = kMinusInv4Pi * s0;
  v[0] = kMinusInv4Pi * s1;
  v[1] = kMinusInv4Pi * s2;
  v[2] = kMinusInv4Pi * s3;
}

// the near-field form of vrankine_from_geom (pt within 7 radii of the panel's centre)
__device__ inline void vrankine_near(const double pt[3], const PanelRec& P, double& phi, double g[3]) {
  double d0 = pt[0] - P.qgc[0], d1 = pt[1] - P.qgc[1], d2 = pt[2] - P.qgc[2];
  double fx_ = P.T[0] * d0 + P.T[1] * d1 + P.T[2] * d2;
  double fy_ = P.T[3] * d0 + P.T[4] * d1 + P.T[5] * d2;
  double fz_ = P.T[6] * d0 + P.T[7] * d1 + P.T[8] * d2;
  double phb, vl[3];
  birk_phi_and_velocity(fx_, fy_, fz_, P.lc, P.edge, phb, vl);
#pragma unroll
  for (int i = 0; i < 3; ++i) g[i] = kFourPi * (P.T[i] * vl[0] + P.T[3 + i] * vl[1] + P.T[6 + i] * vl[2]);
  phi = -kFourPi * phb;
}

// _vrankine_from_geom (rankine_vectorized.jl:273-287): integral of 1/r over panel P
// seen from `pt`, and its gradient with respect to the source.
__device__ inline void vrankine_from_geom(const double pt[3], const PanelRec& P, double& phi, double g[3]) {
  double rb0 = pt[0] - P.c[0], rb1 = pt[1] - P.c[1], rb2 = pt[2] - P.c[2];
  double r = sqrt(rb0 * rb0 + rb1 * rb1 + rb2 * rb2);
  if (r > 7 * P.radius) {
    // a/r and a r_vec/r^3 from one FP64 division (within an ulp or two of the quotients)
    const double inv_r = 1.0 / r;
    const double s = P.area * inv_r * inv_r * inv_r;
    phi = P.area * inv_r;
    g[0] = rb0 * s;
    g[1] = rb1 * s;
    g[2] = rb2 * s;
    return;
  }
  vrankine_near(pt, P, phi, g);
}

// ---------------------------- Delhommeau Rankine ----------------------------
__device__ __forceinline__ double sign_ad(double x) { return x < 0.0 ? -1.0 : 1.0; }

// integral(::DelhommeauRankine) (rankine.jl:33-71) and the gradient of
// both_integral_and_integral_gradient (rankine.jl:73-131); v12: 4 raw corners.
__device__ inline void delhommeau_rankine(const double pt[3], const PanelRec& P, const double* v12, int wrt_first,
                                          double& integral, double g[3]) {
  double rb[3] = {pt[0] - P.c[0], pt[1] - P.c[1], pt[2] - P.c[2]};
  double r = sqrt(rb[0] * rb[0] + rb[1] * rb[1] + rb[2] * rb[2]);
  const double* nrm = P.n;
  if (r > 7 * P.radius) {
    double r3 = r * r * r;
    integral = P.area / r;
    for (int c = 0; c < 3; ++c) g[c] = (1 / r3 * rb[c]) * P.area;
  } else {
    integral = 0.0;
    g[0] = g[1] = g[2] = 0.0;
    double GZ = rb[0] * nrm[0] + rb[1] * nrm[1] + rb[2] * nrm[2];
    double RR[4], DRX[4][3];
    for (int i = 0; i < 4; ++i) {
      double d[3] = {pt[0] - v12[3 * i], pt[1] - v12[3 * i + 1], pt[2] - v12[3 * i + 2]};
      RR[i] = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
      for (int c = 0; c < 3; ++c) DRX[i][c] = d[c] / RR[i];
    }
    for (int iv = 0; iv < 4; ++iv) {
      int in = (iv + 1) & 3;
      double ctn[3] = {v12[3 * in] - v12[3 * iv], v12[3 * in + 1] - v12[3 * iv + 1], v12[3 * in + 2] - v12[3 * iv + 2]};
      double seg = sqrt(ctn[0] * ctn[0] + ctn[1] * ctn[1] + ctn[2] * ctn[2]);
      if (!(seg >= 1e-3 * P.radius)) continue;
      double u[3] = {ctn[0] / seg, ctn[1] / seg, ctn[2] / seg};
      double GYX[3] = {nrm[1] * u[2] - nrm[2] * u[1], nrm[2] * u[0] - nrm[0] * u[2], nrm[0] * u[1] - nrm[1] * u[0]};
      double pv[3] = {pt[0] - v12[3 * iv], pt[1] - v12[3 * iv + 1], pt[2] - v12[3 * iv + 2]};
      double GY = pv[0] * GYX[0] + pv[1] * GYX[1] + pv[2] * GYX[2];
      double ANT = 2 * GY * seg;
      double rs = RR[in] + RR[iv];
      double DNT = rs * rs - seg * seg + 2 * abs_ad(GZ) * rs;
      double ANL = rs + seg, DNL = rs - seg;
      double ALDEN = log(ANL / DNL);
      double AT = fabs(GZ) >= 1e-4 * P.radius ? atan2(ANT, DNT) : 0.0;  // _delhommeau_atan
      integral -= 2 * abs_ad(GZ) * AT;
      if (fabs(GY) > 1e-5) integral += GY * ALDEN;
      double q1 = GY * (DNL - ANL), q2 = 2 * abs_ad(GZ), den2 = ANT * ANT + DNT * DNT;
      for (int c = 0; c < 3; ++c) {
        double ANLX = DRX[in][c] + DRX[iv][c];
        double ANTX = 2 * seg * GYX[c];
        double DNTX = 2 * (rs + abs_ad(GZ)) * ANLX + 2 * sign_ad(GZ) * rs * nrm[c];
        double term = ALDEN * GYX[c] - 2 * sign_ad(GZ) * AT * nrm[c] + q1 / (ANL * DNL) * ANLX -
                      q2 * (ANTX * DNT - DNTX * ANT) / den2;
        g[c] = g[c] - term;
      }
    }
  }
  if (wrt_first) { g[0] = -g[0]; g[1] = -g[1]; g[2] = -g[2]; }
}

// ------------------------------------ Wu -----------------------------------
// Polynomial fits A-D and dA-dC of Liang, Wu & Noblesse (wu.jl:131-197, 235-329), lowest
// degree first, all seven at one rho in [0, 1), in 64-bit fixed point on the integer pipe
// (mh_fixpoint.cuh): coefficients and partial sums are integers v 2^-44 (the partial sums
// stay below 2^18 on [0, 1)), so each Horner step truncates at 5.7e-14 absolute where FP64
// rounds partial sums up to 2e5 at 2.9e-11 (worst error of a fit 4e-13 here, up to 3e-11 in
// the reference's FP64 order); the coefficients are the FP64 values of the literals, as in
// the reference, exactly.
struct WuFits {
  double A, B, C, D, dA, dB, dC;
};

constexpr int kWuFrac = 44;
// A, B, C, D, dA, dB, dC, with zeros above their degrees
static __device__ __constant__ const long long kWuFit[7][10] = {
    {fx::q(1.21, kWuFrac), fx::q(-13.328, kWuFrac), fx::q(215.896, kWuFrac), fx::q(-1763.96, kWuFrac),
     fx::q(8418.94, kWuFrac), fx::q(-24314.21, kWuFrac), fx::q(42002.57, kWuFrac), fx::q(-41592.9, kWuFrac),
     fx::q(21859.0, kWuFrac), fx::q(-4838.6, kWuFrac)},
    {fx::q(0.938, kWuFrac), fx::q(5.737, kWuFrac), fx::q(-67.92, kWuFrac), fx::q(796.534, kWuFrac),
     fx::q(-4780.77, kWuFrac), fx::q(17137.74, kWuFrac), fx::q(-36618.81, kWuFrac), fx::q(44894.06, kWuFrac),
     fx::q(-29030.24, kWuFrac), fx::q(7671.22, kWuFrac)},
    {fx::q(1.268, kWuFrac), fx::q(-9.747, kWuFrac), fx::q(209.653, kWuFrac), fx::q(-1397.89, kWuFrac),
     fx::q(5155.67, kWuFrac), fx::q(-9844.35, kWuFrac), fx::q(9136.4, kWuFrac), fx::q(-3272.62, kWuFrac), 0,
     0},
    {fx::q(0.632, kWuFrac), fx::q(-40.97, kWuFrac), fx::q(667.16, kWuFrac), fx::q(-6072.07, kWuFrac),
     fx::q(31127.39, kWuFrac), fx::q(-96293.05, kWuFrac), fx::q(181856.75, kWuFrac), fx::q(-205690.43,
     kWuFrac), fx::q(128170.2, kWuFrac), fx::q(-33744.6, kWuFrac)},
    {fx::q(2.948, kWuFrac), fx::q(-24.53, kWuFrac), fx::q(249.69, kWuFrac), fx::q(-754.85, kWuFrac),
     fx::q(-1187.71, kWuFrac), fx::q(16370.75, kWuFrac), fx::q(-48811.41, kWuFrac), fx::q(68220.87, kWuFrac),
     fx::q(-46688.0, kWuFrac), fx::q(12622.25, kWuFrac)},
    {fx::q(1.11, kWuFrac), fx::q(2.894, kWuFrac), fx::q(-76.765, kWuFrac), fx::q(1565.35, kWuFrac),
     fx::q(-11336.19, kWuFrac), fx::q(44270.15, kWuFrac), fx::q(-97014.11, kWuFrac), fx::q(118879.26,
     kWuFrac), fx::q(-76209.82, kWuFrac), fx::q(19923.28, kWuFrac)},
    {fx::q(14.19, kWuFrac), fx::q(-148.24, kWuFrac), fx::q(847.8, kWuFrac), fx::q(-2318.58, kWuFrac),
     fx::q(3168.35, kWuFrac), fx::q(-1590.27, kWuFrac), 0, 0, 0, 0}};

// one function, called: inlined seven times the fits are 800 instructions, which the warps of an
// SM fetch more slowly than they run (wave_kernel)
static __device__ __noinline__ double wu_fit(int which, unsigned long long t) {
  long long v = kWuFit[which][9];
#pragma unroll
  for (int i = 8; i >= 0; --i) v = kWuFit[which][i] + fx::mulhi_su(v, t);
  return fx::to_double(v, kWuFrac);
}

__device__ __forceinline__ void wu_fits(double rho, WuFits& f) {
  const unsigned long long t = fx::unit_q64(rho);
  f.A = wu_fit(0, t);
  f.B = wu_fit(1, t);
  f.C = wu_fit(2, t);
  f.D = wu_fit(3, t);
  f.dA = wu_fit(4, t);
  f.dB = wu_fit(5, t);
  f.dC = wu_fit(6, t);
}

// StruveH0 and StruveH1 fits (wu.jl:368-435); also returns J0/J1.  The four Bessel
// functions of the argument come from one joint evaluation (mh_bessel01.cuh).  The
// polynomials in yy in [0, 1] run in fixed point (v 2^-59 below 3, 2^-55 above, variable
// yy / 2, so coefficient i carries 2^i); the rational fits' quotients stay FP64.
// inv_xx = 1 / xx (used above 3).
__device__ inline void struve_bessel(double xx, double inv_xx, double& H0, double& H1, double& J0, double& J1) {
  double Y0, Y1;
  bessel01(xx, J0, J1, Y0, Y1);
  constexpr int F = 59;
  if (xx <= 3.0) {
    const double x3 = xx * (1.0 / 3.0);
    const unsigned long long t = fx::unit_q63(x3 * x3);
    constexpr long long kH0[6] = {fx::q(1.909859164, F), fx::q(-1.909855001, F + 1), fx::q(0.687514637, F + 2),
                                  fx::q(-0.126164557, F + 3), fx::q(0.013828813, F + 4),
                                  fx::q(-0.000876918, F + 5)};
    // H1 = yy (1.909859286 + ...): the factor yy as one more Horner step with c = 0
    constexpr long long kH1[7] = {0, fx::q(1.909859286, F + 1), fx::q(-1.145914713, F + 2),
                                  fx::q(0.294656958, F + 3), fx::q(-0.042070508, F + 4),
                                  fx::q(0.003785727, F + 5), fx::q(-0.000207183, F + 6)};
    H0 = fx::to_double(fx::horner_u(kH0, t), F) * x3;
    H1 = fx::to_double(fx::horner_u(kH1, t), F);
  } else {
    constexpr int G = 55;  // partial sums up to 2^7
    const double t3 = 3.0 * inv_xx;
    const unsigned long long t = fx::unit_q63(t3 * t3);
    constexpr long long kC1[4] = {fx::q(0.99999906, G + 1), fx::q(4.77228920, G + 2), fx::q(3.85542044, G + 3),
                                  fx::q(0.32303607, G + 4)};  // 2 (a0 + a1 yy + ...)
    constexpr long long kC2[4] = {fx::q(1.0, G), fx::q(4.88331068, G + 1), fx::q(4.28957333, G + 2),
                                  fx::q(0.52120508, G + 3)};
    constexpr long long kD1[4] = {fx::q(1.00000004, G + 1), fx::q(3.92205313, G + 2), fx::q(2.64893033, G + 3),
                                  fx::q(0.27450895, G + 4)};
    constexpr long long kD2[4] = {fx::q(1.0, G), fx::q(3.81095112, G + 1), fx::q(2.26216956, G + 2),
                                  fx::q(0.10885141, G + 3)};
    const double c1 = fx::to_double(fx::horner_u(kC1, t), G);
    const double c2 = kPi * xx * fx::to_double(fx::horner_u(kC2, t), G);
    const double d1 = fx::to_double(fx::horner_u(kD1, t), G);
    const double d2 = kPi * fx::to_double(fx::horner_u(kD2, t), G);
    const double inv = fx::recip_call(c2 * d2);
    H0 = c1 * d2 * inv + Y0;
    H1 = d1 * c2 * inv + Y1;
  }
}

// _wu_wave_term_and_derivs (wu.jl:28-37) with GF_Func_L0/Lp/W/Ls/Lsp/Wh (wu.jl:201-366)
// FP64 division is a multi-instruction sequence on GB300's FP64 pipe, which bounds this
// kernel; 1/dd, 1/(dd - vv), 1/(1 + dd^3) and 1/hh come from one reciprocal of their
// product, taken on the integer pipe (fx::recip, within an ulp) like the other reciprocals
// and the square roots of the term, and are multiplied out (rho gets one residual
// correction on top: an ulp of rho moves the fits A-D by up to 1e-13).  inv_hh: 1/hh for hh > 1e-6 (the only pairs
// whose horizontal gradient factor k^2/hh is used, wu.jl:118-121), else 0.
// `step` is called three times, by every thread: the wave assembly passes a CTA barrier that
// keeps its warps on the same instructions.
struct NoStep { __device__ __forceinline__ void operator()() const {} };
struct CtaStep {
  __device__ __forceinline__ void operator()() const { asm volatile("bar.sync 0;" ::: "memory"); }
};
template <typename Step = NoStep>
__device__ __forceinline__ void wu_wave_term_and_derivs(double hh, double vv, double2& GF, double2& dGh, double2& dGv,
                                                        double* inv_hh = nullptr, Step step = Step()) {
  double dd = fx::sqrt_pos(hh * hh + vv * vv);
  double dd2 = dd * dd, dd3 = dd * dd * dd;
  // 1/dd, 1/(dd - vv), 1/(1 + dd^3) and 1/hh from one division of their product (all
  // factors are positive, dd - vv >= dd >= hh with vv <= 0, and moderate: below 1e6 in the
  // reduced coordinates, so the product stays far inside the FP64 range)
  const double dmv = dd - vv, opd3 = 1.0 + dd3;
  const bool has_h = fabs(hh) > 1e-6;
  const double hf = has_h ? hh : 1.0;
  const double prod3 = dd * dmv * opd3;
  const double inv_all = fx::recip_call(prod3 * hf);
  const double inv_all3 = inv_all * hf;  // 1 / (dd dmv opd3)
  const double inv_dd = dmv * opd3 * inv_all3;
  const double inv_dmv = dd * opd3 * inv_all3;
  const double inv_1dd3 = dd * dmv * inv_all3;
  const double inv_h = has_h ? prod3 * inv_all : 0.0;
  if (inv_hh) *inv_hh = inv_h;
  double alpha = -vv * inv_dd;
  double beta = hh * inv_dd;
  // rho = dd / (1 + dd): the integer-pipe reciprocal and one residual correction, which
  // leaves rho within a rounding of the correctly rounded quotient
  const double opdd = 1 + dd;
  const double r1 = fx::recip_call(opdd);
  double rho = dd * r1;
  rho = fma(fma(-rho, opdd, dd), r1, rho);
  double omr = 1.0 - rho;
  double omr3 = omr * omr * omr;
  double ev = fx::exp_nonpos(vv);
  double H0, H1, J0, J1;
  step();
  struve_bessel(hh, inv_h, H0, H1, J0, J1);
  // GF_Func_Lp
  WuFits fit;
  step();
  wu_fits(rho, fit);
  step();
  double RR = (1.0 - beta) * fit.A;
  RR -= beta * fit.B;
  RR -= alpha * fit.C * fx::recip_call(1.0 + 6.0 * alpha * rho * (1.0 - rho));
  RR += beta * (1.0 - beta) * fit.D;
  double Lp = rho * omr3 * RR;
  // GF_Func_L0
  const double gama = 0.5772156649;
  double PP = fx::log_pos(0.5 * (dd - vv)) + gama - 2.0 * dd2;
  PP = ev * PP;
  PP = PP + dd2 - vv;
  double L0 = 2.0 * PP * inv_1dd3 + 2.0 * Lp;
  const double twopi = 2 * kPi;
  GF = make_double2(-L0 - (twopi * H0) * ev, -((twopi * -J0) * ev));
  // GF_Func_Lsp
  double RS = beta * fit.dA;
  RS -= (1.0 - alpha) * fit.dB;
  RS += beta * (1.0 - beta) * rho * (1.0 - 2.0 * rho) * fit.dC;
  double Lsp = rho * omr3 * RS;
  // GF_Func_Ls
  double PS = (beta + hh) * inv_dmv;
  PS = PS - 2.0 * beta + 2.0 * ev * dd - hh;
  double QS = fx::exp_nonpos(-dd) * (1.0 - beta);
  QS = QS * (1.0 + dd * inv_1dd3);
  double Ls = 2.0 * PS * inv_1dd3 - 4.0 * QS + 2.0 * Lsp;
  dGh = make_double2(-Ls - (twopi * (2 / kPi - H1)) * ev, -((twopi * J1) * ev));
  dGv = make_double2(GF.x + 2 * inv_dd, GF.y);
}

// _wu_reduced_hh_vv (wu.jl:7-18) == with_reduced_coordinates (abstract_greens_function.jl:117-138)
__device__ __forceinline__ void reduced_coords(const double x[3], const double xi[3], double k, double& hh,
                                               double& vv) {
  double d2 = (x[0] - xi[0]) * (x[0] - xi[0]) + (x[1] - xi[1]) * (x[1] - xi[1]);
  const double purt = 1e-18;
  double dis = (d2 == 0) ? sqrt(d2 + purt * purt) - purt : fx::sqrt_pos(d2);
  hh = k * dis;
  vv = k * (x[2] + xi[2]);
}

// ------------------------- exact Guevel-Delhommeau --------------------------
// 1/n for the power series of E1 (every entry the correctly rounded quotient, as 1.0 / n)
struct InvN {
  double v[400];
};
__constant__ static const InvN kInvN = [] {
  InvN t{};
  for (int n = 1; n < 400; ++n) t.v[n] = 1.0 / (double)n;
  return t;
}();

// a / b for a real numerator: a conj(b) / |b|^2, one division (|b| stays far inside the
// FP64 range in the continued fraction below: its terms are b_i = z + 2i + 1 and their
// quotients)
__device__ __forceinline__ double2 rdivz(double a, double2 b) {
  const double s = a / (b.x * b.x + b.y * b.y);
  return make_double2(b.x * s, -b.y * s);
}

// e^z E1(z): power series of E1 (DLMF 6.6.2) where its cancellation loss
// exp(|z| + Re z) is below e^4, else the even continued fraction of DLMF 6.9.1
// by the modified Lentz method.  Iteration counts are bounded.  `ez` = e^z (the
// integrands have it already).  Convergence and underflow tests compare squared
// magnitudes (no hypot in the loops); 1/n comes from a table.
__device__ inline double2 exp_e1(double2 z, double2 ez) {
  const double az = hypot(z.x, z.y);
  if (az + z.x < 4.0) {
    double2 term = make_double2(1.0, 0.0), sum = make_double2(0.0, 0.0);
    const double2 mz = make_double2(-z.x, -z.y);
    for (int n = 1; n < 400; ++n) {
      const double inv = kInvN.v[n];
      term = zscale(inv, zmul(term, mz));
      const double2 add = zscale(inv, term);
      sum = zadd(sum, add);
      if (add.x * add.x + add.y * add.y <= 1e-34 * (sum.x * sum.x + sum.y * sum.y)) break;
    }
    const double euler_gamma = 0.57721566490153286061;
    const double2 lz = make_double2(log(az), atan2(z.y, z.x));
    const double2 e1 = make_double2(-euler_gamma - lz.x - sum.x, -lz.y - sum.y);
    return zmul(ez, e1);
  }
  const double tiny = 1e-300;
  double2 b = make_double2(z.x + 1.0, z.y);
  double2 f = b;
  double2 C = f, D = make_double2(0.0, 0.0);
  for (int i = 1; i < 400; ++i) {
    const double a = -(double)i * (double)i;
    b.x += 2.0;
    D = make_double2(b.x + a * D.x, b.y + a * D.y);
    if (fabs(D.x) + fabs(D.y) < tiny) D = make_double2(tiny, 0.0);
    const double2 q = rdivz(a, C);
    C = make_double2(b.x + q.x, b.y + q.y);
    if (fabs(C.x) + fabs(C.y) < tiny) C = make_double2(tiny, 0.0);
    D = rdivz(1.0, D);
    const double2 delta = zmul(C, D);
    f = zmul(f, delta);
    const double dx = delta.x - 1.0;
    if (dx * dx + delta.y * delta.y < 1e-32) break;
  }
  return rdivz(1.0, f);
}

__constant__ static const double kGKx[8] = {0.991455371120812639206854697526329, 0.949107912342758524526189684047851,
                                           0.864864423359769072789712788640926, 0.741531185599394439863864773280788,
                                           0.586087235467691130294144845693013, 0.405845151377397166906606412076961,
                                           0.207784955007898467600689403773245, 0.0};
__constant__ static const double kGKwk[8] = {0.022935322010529224963732008058970, 0.063092092629978553290700663189204,
                                            0.104790010322250183839876322541518, 0.140653259715525918745189590510238,
                                            0.169004726639267902826583426598550, 0.190350578064785409913256402421014,
                                            0.204432940075298892414161999234649, 0.209482141084727828012999174891714};
__constant__ static const double kGKwg[4] = {0.129484966168869693270611432679082, 0.279705391489276667901467771423780,
                                            0.381830050505118944950369775488975, 0.417959183673469387755102040816327};

// Adaptive GK(7,15) over [0, pi/2], times 4 (exact_Guevel_Delhommeau.jl:8-13, 25, 45), by a whole
// warp: the 15 Kronrod nodes of two segments run on 30 lanes, G and dG/dr come from the same
// exp(zeta), E1(zeta) evaluation at each node, and the depth-first refinement stack lives in
// shared memory, written by lane 0 and read by the whole warp.
constexpr int kGKWarpStack = 48;   // entries of 8 doubles: a, b, G (2), dG/dr (2), err G, err dG/dr
constexpr int kGKMaxEvals = 8192;  // evaluations of two segments, a hard bound

// both integrands at theta (exact_Guevel_Delhommeau.jl:16-23, 36-43), from one E1
__device__ __forceinline__ void egd_integrands(double theta, double r, double z, double f[4]) {
  const double ct = cos(theta);
  const double2 zeta = make_double2(z, r * ct);
  const double2 ez = zexp(zeta);
  const double2 g = exp_e1(zeta, ez);
  const double inv_pi = 1.0 / kPi;
  // j = e^zeta (E1(zeta)/pi + i) = g/pi + i e^zeta
  const double2 j = make_double2(g.x * inv_pi - ez.y, g.y * inv_pi + ez.x);
  f[0] = j.x;
  f[1] = ez.x;
  const double2 inv = rdivz(inv_pi, zeta);  // 1 / (pi zeta); |zeta| >= -z > 0 below the free surface
  const double2 w = make_double2(j.x - inv.x, j.y - inv.y);
  // Re(i ct w) = -ct Im(w); Re(i ct e^zeta) = -ct Im(e^zeta)
  f[2] = -ct * w.y;
  f[3] = -ct * ez.y;
}

// Kronrod node, Kronrod weight and Gauss weight of this lane (lanes 15 and 31 idle)
__device__ __forceinline__ void gk_lane_node(int lane, double& t, double& wk, double& wg) {
  const int j = lane & 15;
  t = 0.0; wk = 0.0; wg = 0.0;
  if (j == 15) return;
  if (j < 7) {
    t = -kGKx[j]; wk = kGKwk[j]; wg = (j & 1) ? kGKwg[j >> 1] : 0.0;
  } else if (j == 7) {
    wk = kGKwk[7]; wg = kGKwg[3];
  } else {
    const int m = 14 - j;
    t = kGKx[m]; wk = kGKwk[m]; wg = (m & 1) ? kGKwg[m >> 1] : 0.0;
  }
}

// GK(7,15) of both integrands over [aA, bA] (lanes 0-15) and [aB, bB] (lanes 16-31);
// every lane returns both results
__device__ __forceinline__ void gk15_pair_warp(double aA, double bA, double aB, double bB, double r, double z,
                                               double vA[4], double& eGA, double& eRA, double vB[4], double& eGB,
                                               double& eRB) {
  const int lane = threadIdx.x & 31;
  double t, wk, wg;
  gk_lane_node(lane, t, wk, wg);
  const double a = lane < 16 ? aA : aB, b = lane < 16 ? bA : bB;
  const double c = 0.5 * (a + b), h = 0.5 * (b - a);
  double f[4];
  egd_integrands(c + h * t, r, z, f);
  double K[4], Gs[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) { K[q] = wk * f[q]; Gs[q] = wg * f[q]; }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      K[q] += __shfl_xor_sync(0xffffffffu, K[q], off);
      Gs[q] += __shfl_xor_sync(0xffffffffu, Gs[q], off);
    }
  }
  double KA[4], GA[4], KB[4], GB[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    KA[q] = __shfl_sync(0xffffffffu, K[q], 0);
    GA[q] = __shfl_sync(0xffffffffu, Gs[q], 0);
    KB[q] = __shfl_sync(0xffffffffu, K[q], 16);
    GB[q] = __shfl_sync(0xffffffffu, Gs[q], 16);
  }
  const double hA = 0.5 * (bA - aA), hB = 0.5 * (bB - aB);
#pragma unroll
  for (int q = 0; q < 4; ++q) { vA[q] = hA * KA[q]; vB[q] = hB * KB[q]; }
  eGA = hypot(hA * (KA[0] - GA[0]), hA * (KA[1] - GA[1]));
  eRA = hypot(hA * (KA[2] - GA[2]), hA * (KA[3] - GA[3]));
  eGB = hypot(hB * (KB[0] - GB[0]), hB * (KB[1] - GB[1]));
  eRB = hypot(hB * (KB[2] - GB[2]), hB * (KB[3] - GB[3]));
}

// G = _dimless_wave_term(r, z) and dG/dr = _d_dimless_wave_term_dr(r, z) by the whole warp
// (all 32 lanes call it with the same r, z; `sw` is this warp's 8 * kGKWarpStack doubles of
// shared memory), to a total error estimate <= max(atol, rtol |I|) of each integral.  The phase
// r cos(theta) of the integrand turns through r radians over the interval, so the interval is
// first cut into ceil(r / 4) equal segments (at most 1024, about 2/3 of an oscillation each); each
// is then refined depth-first by bisection until both error estimates are below its share of the
// tolerances, tol * length / (pi/2), with tol from a first pass over the initial segments.  Large r
// costs time, not memory.
__device__ inline void egd_warp(double r, double z, double rtol, double atol, double* sw, double2& G, double2& Gr) {
  const int lane = threadIdx.x & 31;
  const double L = kPi / 2;
  const int m0 = (int)fmin(1024.0, fmax(1.0, ceil(r / 4.0)));
  const double h0 = L / m0;
  // first pass: the integrals over the initial segments and the tolerances they imply
  double cg[4] = {0.0, 0.0, 0.0, 0.0};
  double v1[4] = {0.0, 0.0, 0.0, 0.0}, e1G = 0.0, e1R = 0.0;
  int evals = 0;
  for (int s = 0; s < m0; s += 2) {
    const int s2 = s + 1 < m0 ? s + 1 : s;
    double vA[4], vB[4], eGA, eRA, eGB, eRB;
    gk15_pair_warp(s * h0, s == m0 - 1 ? L : (s + 1) * h0, s2 * h0, s2 == m0 - 1 ? L : (s2 + 1) * h0, r, z, vA, eGA,
                   eRA, vB, eGB, eRB);
    ++evals;
#pragma unroll
    for (int q = 0; q < 4; ++q) cg[q] += vA[q] + (s2 != s ? vB[q] : 0.0);
    if (s == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v1[q] = vA[q];
      e1G = eGA;
      e1R = eRA;
    }
  }
  const double tolG = fmax(atol, rtol * hypot(cg[0], cg[1]));
  const double tolR = fmax(atol, rtol * hypot(cg[2], cg[3]));
  double tot[4] = {0.0, 0.0, 0.0, 0.0};
  int top = 0;
  auto push = [&](double a, double b, const double v[4], double eG, double eR) {
    if (lane == 0) {
      double* e = sw + 8 * top;
      e[0] = a; e[1] = b; e[2] = v[0]; e[3] = v[1]; e[4] = v[2]; e[5] = v[3]; e[6] = eG; e[7] = eR;
    }
    ++top;
  };
  for (int s = 0; s < m0; s += 2) {
    const int s2 = s + 1 < m0 ? s + 1 : s;
    if (m0 == 1) {
      push(0.0, L, v1, e1G, e1R);
    } else {
      double vA[4], vB[4], eGA, eRA, eGB, eRB;
      const double aA = s * h0, bA = s == m0 - 1 ? L : (s + 1) * h0;
      const double aB = s2 * h0, bB = s2 == m0 - 1 ? L : (s2 + 1) * h0;
      gk15_pair_warp(aA, bA, aB, bB, r, z, vA, eGA, eRA, vB, eGB, eRB);
      ++evals;
      if (s2 != s) push(aB, bB, vB, eGB, eRB);
      push(aA, bA, vA, eGA, eRA);
    }
    __syncwarp();
    while (top > 0) {
      --top;
      const double* e = sw + 8 * top;
      const double a = e[0], b = e[1], eG = e[6], eR = e[7];
      const double v[4] = {e[2], e[3], e[4], e[5]};
      __syncwarp();  // every lane has read the entry before it can be overwritten
      const double frac = (b - a) / L;
      if ((eG <= tolG * frac && eR <= tolR * frac) || top + 2 > kGKWarpStack || evals + 1 > kGKMaxEvals) {
#pragma unroll
        for (int q = 0; q < 4; ++q) tot[q] += v[q];
        continue;
      }
      const double mid = 0.5 * (a + b);
      double vA[4], vB[4], eGA, eRA, eGB, eRB;
      gk15_pair_warp(a, mid, mid, b, r, z, vA, eGA, eRA, vB, eGB, eRB);
      ++evals;
      push(mid, b, vB, eGB, eRB);
      push(a, mid, vA, eGA, eRA);  // the left half is refined first
      __syncwarp();
    }
  }
  G = make_double2(4.0 * tot[0], 4.0 * tot[1]);
  Gr = make_double2(4.0 * tot[2], 4.0 * tot[3]);
}

}  // namespace mh
