// mh_adjoint.cu -- reverse (adjoint) kernels of the assembly: gradient of a
// real objective with respect to every panel's centre, normal, area and corner
// vertices, recomputing the Green-function derivatives pair by pair instead of
// storing them (the reference differentiates the assembly loops with Enzyme /
// ForwardDiff, matrix_assembly.jl:341-342, with the Birk kernel rules of
// ad_rules.jl:79-294).
//
// Objective weights.  With J = sum Re(W^S_ij dS_ij + W^D_ij dD_ij) over pairs,
// the caller supplies, per wavenumber, the weight factors as vectors
//   W^S_ij = c sum_h lS_h[i] rS_h[j],   W^D_ij = -c sum_h lD_h[i] rD_h[j]
// (rank-nh outer products, never formed), and for the wavenumber-independent
// Rankine part the real, frequency-summed matrices RS = Re sum W^S, RD = Re sum W^D.
// Direct BEM (phi = D^-1 S b, lam = D^-T w for the force weights w): lS = lD = lam,
// rS = b, rD = phi.  Indirect BEM (sigma = K^-1 b, phi = S sigma, lam = K^-T S^T w):
// lS = w, rS = rD = sigma, lD = lam -- the _mulvec and _linearsolve rules
// (ad_rules.jl:300-414) applied to the two formulations of solve (matrix_assembly.jl:436-449).
// The pair kernels are templated on the formulation: the indirect D differentiates the
// field point and carries the field panel's normal.
//
// Per-panel gradient accumulators (device, FP64, atomically summed):
//   gc[n][3] centre, gn[n][3] normal, ga[n] area, gv[n][12] Birk corner vertices.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "mh_dual.cuh"
#include "mh_egd.cuh"
#include "mh_internal.cuh"

namespace mh {

namespace {

constexpr int kRows = 128;
constexpr int kCols = 8;
constexpr int kMaxH = 4;  // right-hand sides per frequency in the adjoint weights

struct GradPtrs {
  double* gc;
  double* gn;
  double* ga;
  double* gv;
};

template <typename R> struct CR { R x, y; };

// ---------------------------------------------------------------------------
// Wu wave term on a generic scalar (the same operations as wu_wave_term_and_derivs)
// ---------------------------------------------------------------------------
// The seven fits (wu.jl:131-197, 235-329) and their derivatives in rho.  The terms from rho^2 up run
// in 64-bit fixed point (mh_fixpoint.cuh) with the fraction bits that the largest partial sum on
// [0, 1] leaves, the last two steps in FP64.  The differentiated coefficients are integer
// multiples of the fixed-point ones: as doubles (7 * 205690.43 ..) they would round by up to
// 1e-10, the same way in every pair, and the added mass' frequency derivative would be off by
// 2e-14 instead of 8e-15.
constexpr double kWuCoef[7][10] = {
    {1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6},        // A
    {0.938, 5.737, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22},        // B
    {1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62},                             // C
    {0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2, -33744.6},   // D
    {2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25},       // dA
    {1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82, 19923.28},     // dB
    {14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27}};                                               // dC
struct WuDualTable {
  long long c[14][8];  // the seven fits', then their derivatives', coefficients from rho^2 up
  double low[14][2];
  int frac[14];
};
constexpr WuDualTable make_wu_dual_table() {
  constexpr int degree[7] = {9, 9, 7, 9, 9, 9, 5};
  constexpr int frac[14] = {47, 47, 49, 45, 46, 46, 51, 44, 44, 47, 42, 44, 43, 49};
  WuDualTable t{};
  for (int w = 0; w < 14; ++w) {
    const int der = w >= 7, top = degree[w % 7] - 2 - der;
    const double* c = kWuCoef[w % 7];
    t.frac[w] = frac[w];
    t.low[w][0] = c[der];
    t.low[w][1] = (1 + der) * c[1 + der];
    for (int i = 0; i <= top; ++i) t.c[w][i] = (der ? i + 3 : 1) * fx::q(c[i + 2 + der], frac[w]);
    // a shorter fit starts from zeros: what wu_dual_fit's half units add to them (every odd
    // coefficient) is taken off again
    for (int i = top < 7 ? top : 7; i < 7; ++i)
      if (i & 1) t.c[w][i] -= 1;
  }
  return t;
}
static __device__ __constant__ const WuDualTable kWuDual = make_wu_dual_table();

// Horner's scheme without the bias of fx::horner_u: every step rounds down by half a unit on average,
// which every other coefficient makes up for with one unit.  A sum over many pairs would not
// average the bias out, as it does the rounding itself.  Called fourteen times (inlined, the fits
// outgrow the instruction caches; see wu_fit in mh_greens.cuh).
static __device__ __noinline__ double wu_dual_fit(int which, double rho, unsigned long long t) {
  long long v = kWuDual.c[which][7];
#pragma unroll
  for (int i = 6; i >= 0; --i) v = kWuDual.c[which][i] + (i & 1) + fx::mulhi_su(v, t);
  return fma(fma(fx::to_double(v, kWuDual.frac[which]), rho, kWuDual.low[which][1]), rho, kWuDual.low[which][0]);
}
__device__ __forceinline__ void wu_fits_and_derivatives(double rho, WuFits& f, WuFits& d) {
  const unsigned long long t = fx::unit_q64(rho);
  f.A = wu_dual_fit(0, rho, t);
  f.B = wu_dual_fit(1, rho, t);
  f.C = wu_dual_fit(2, rho, t);
  f.D = wu_dual_fit(3, rho, t);
  f.dA = wu_dual_fit(4, rho, t);
  f.dB = wu_dual_fit(5, rho, t);
  f.dC = wu_dual_fit(6, rho, t);
  d.A = wu_dual_fit(7, rho, t);
  d.B = wu_dual_fit(8, rho, t);
  d.C = wu_dual_fit(9, rho, t);
  d.D = wu_dual_fit(10, rho, t);
  d.dA = wu_dual_fit(11, rho, t);
  d.dB = wu_dual_fit(12, rho, t);
  d.dC = wu_dual_fit(13, rho, t);
}

// sum c_i t^i, its derivative, and the derivative of t times it
template <int N>
__device__ __forceinline__ double poly(const double (&c)[N], double t) {
  double v = c[N - 1];
#pragma unroll
  for (int i = N - 2; i >= 0; --i) v = fma(v, t, c[i]);
  return v;
}
template <int N>
__device__ __forceinline__ double poly_d(const double (&c)[N], double t) {
  double v = (N - 1) * c[N - 1];
#pragma unroll
  for (int i = N - 2; i >= 1; --i) v = fma(v, t, i * c[i]);
  return v;
}
template <int N>
__device__ __forceinline__ double poly_td(const double (&c)[N], double t) {
  double v = N * c[N - 1];
#pragma unroll
  for (int i = N - 2; i >= 0; --i) v = fma(v, t, (i + 1) * c[i]);
  return v;
}

// StruveH0 and StruveH1 fits (wu.jl:368-435) and J0, J1 of one argument: the values and the
// derivatives as plain numbers, the dual's directions multiplied on at the end (J0' = -J1, J1' =
// J0 - J1/x, Y0' = -Y1, Y1' = Y0 - Y1/x)
template <typename R>
__device__ __forceinline__ void struve_bessel_t(const R& hh, R& H0, R& H1, R& J0, R& J1) {
  const double x = val(hh);
  double j0, j1, y0, y1;
  bessel01(x, j0, j1, y0, y1);
  const double inv_x = x != 0.0 ? fx::recip_call(x) : 0.0;
  J0 = chain1(hh, j0, -j1);
  J1 = chain1(hh, j1, x != 0.0 ? fma(-j1, inv_x, j0) : 0.5);
  if (x <= 3.0) {
    constexpr double kP[6] = {1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918};
    constexpr double kQ[6] = {1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183};
    const double x3 = x * (1.0 / 3.0), yy = x3 * x3;
    const double p = poly(kP, yy), dp = poly_d(kP, yy), q = poly(kQ, yy);
    H0 = chain1(hh, p * x3, fma(2.0 * yy, dp, p) * (1.0 / 3.0));
    H1 = chain1(hh, q * yy, poly_td(kQ, yy) * (2.0 / 3.0) * x3);
  } else {
    constexpr double kA[4] = {0.99999906, 4.77228920, 3.85542044, 0.32303607};
    constexpr double kB[3] = {4.88331068, 4.28957333, 0.52120508};  // after 1
    constexpr double kC[4] = {1.00000004, 3.92205313, 2.64893033, 0.27450895};
    constexpr double kD[3] = {3.81095112, 2.26216956, 0.10885141};
    const double t3 = 3.0 * inv_x, yy = t3 * t3, dy = -2.0 * yy * inv_x;
    const double c1 = 2.0 * poly(kA, yy), dc1 = 2.0 * poly_d(kA, yy) * dy;
    const double e2 = kPi * fma(poly(kB, yy), yy, 1.0), de2 = kPi * poly_td(kB, yy) * dy;
    const double d1 = 2.0 * poly(kC, yy), dd1 = 2.0 * poly_d(kC, yy) * dy;
    const double d2 = kPi * fma(poly(kD, yy), yy, 1.0), dd2 = kPi * poly_td(kD, yy) * dy;
    // c2 = x e2
    const double inv_c2 = fx::recip_call(e2) * inv_x, inv_d2 = fx::recip_call(d2);
    const double r = c1 * inv_c2, s = d1 * inv_d2;
    H0 = chain1(hh, r + y0, fma(dc1 - r * fma(x, de2, e2), inv_c2, -y1));
    H1 = chain1(hh, s + y1, fma(dd1 - s * dd2, inv_d2, fma(-y1, inv_x, y0)));
  }
}

// `step` is called twice, by every thread: a CTA barrier keeps the warps on the same instructions
// (wave_kernel, mh_assembly.cu).
template <typename R, typename Step = NoStep>
__device__ __forceinline__ void wu_terms_t(R hh, R vv, CR<R>& GF, CR<R>& Gh, CR<R>& Gv, Step step = Step()) {
  R dd = sqrt(hh * hh + vv * vv);
  const R inv_dd = 1.0 / dd;
  R alpha = -vv * inv_dd;
  R beta = hh * inv_dd;
  // rho = dd / (1 + dd), with one residual correction as in the primal: an ulp of rho moves the
  // fits by up to 1e-13
  const double opdd = 1.0 + val(dd), r1 = pos_recip(opdd);
  double rv = val(dd) * r1;
  rv = fma(fma(-rv, opdd, val(dd)), r1, rv);
  const R rho = chain1(dd, rv, r1 * r1);
  R dd2 = dd * dd, dd3 = dd * dd * dd;
  R omr = 1.0 - rho;
  R omr3 = omr * omr * omr;
  R ev = exp(vv);
  R J0, J1, H0, H1;
  step();
  struve_bessel_t(hh, H0, H1, J0, J1);
  step();
  WuFits fit, der;
  wu_fits_and_derivatives(val(rho), fit, der);
  R RR = (1.0 - beta) * chain1(rho, fit.A, der.A);
  RR -= beta * chain1(rho, fit.B, der.B);
  RR -= alpha * chain1(rho, fit.C, der.C) / (1.0 + 6.0 * alpha * rho * (1.0 - rho));
  RR += beta * (1.0 - beta) * chain1(rho, fit.D, der.D);
  R Lp = rho * omr3 * RR;
  const double gama = 0.5772156649;
  R PP = log(0.5 * (dd - vv)) + gama - 2.0 * dd2;
  PP = ev * PP;
  PP = PP + dd2 - vv;
  const R inv_1dd3 = 1.0 / (1.0 + dd3);
  R L0 = 2.0 * PP * inv_1dd3 + 2.0 * Lp;
  const double twopi = 2 * kPi;
  GF.x = -L0 - (twopi * H0) * ev;
  GF.y = -((twopi * -J0) * ev);
  R RS = beta * chain1(rho, fit.dA, der.dA);
  RS -= (1.0 - alpha) * chain1(rho, fit.dB, der.dB);
  RS += beta * (1.0 - beta) * rho * (1.0 - 2.0 * rho) * chain1(rho, fit.dC, der.dC);
  R Lsp = rho * omr3 * RS;
  R PS = (beta + hh) / (dd - vv);
  PS = PS - 2.0 * beta + 2.0 * ev * dd - hh;
  R QS = exp(-dd) * (1.0 - beta);
  QS = QS * (1.0 + dd * inv_1dd3);
  R Ls = 2.0 * PS * inv_1dd3 - 4.0 * QS + 2.0 * Lsp;
  Gh.x = -Ls - (twopi * (2 / kPi - H1)) * ev;
  Gh.y = -((twopi * J1) * ev);
  Gv.x = GF.x + 2.0 * inv_dd;
  Gv.y = GF.y;
}

// ---------------------------------------------------------------------------
// Birk panel frame on a generic scalar: T (s, t, n), area centroid and local corners from the
// panel's 4 corners (rankine_vectorized.jl:79-137), as panel_geometry_kernel computes them
// ---------------------------------------------------------------------------
template <typename R>
__device__ void birk_geometry_t(const R v[12], R T[9], R qgc[3], R lc[8]) {
  R mid[4][3], mgc[3], s[3], tt[3], nn[3], t[3];
  for (int i = 0; i < 4; ++i) {
    int ip = (i + 1) & 3;
    for (int c = 0; c < 3; ++c) mid[i][c] = (v[3 * i + c] + v[3 * ip + c]) / 2.0;
  }
  for (int c = 0; c < 3; ++c) {
    mgc[c] = (mid[1][c] + mid[3][c]) / 2.0;
    s[c] = mid[1][c] - mid[3][c];
    tt[c] = mid[2][c] - mid[0][c];
  }
  R ns = sqrt(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
  for (int c = 0; c < 3; ++c) s[c] = s[c] / ns;
  nn[0] = s[1] * tt[2] - s[2] * tt[1];
  nn[1] = s[2] * tt[0] - s[0] * tt[2];
  nn[2] = s[0] * tt[1] - s[1] * tt[0];
  R nl = sqrt(nn[0] * nn[0] + nn[1] * nn[1] + nn[2] * nn[2]);
  for (int c = 0; c < 3; ++c) nn[c] = nn[c] / nl;
  t[0] = nn[1] * s[2] - nn[2] * s[1];
  t[1] = nn[2] * s[0] - nn[0] * s[2];
  t[2] = nn[0] * s[1] - nn[1] * s[0];
  R tl = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
  for (int c = 0; c < 3; ++c) t[c] = t[c] / tl;
  R tc[4][2];
  for (int k = 0; k < 4; ++k) {
    R d0 = v[3 * k] - mgc[0], d1 = v[3 * k + 1] - mgc[1], d2 = v[3 * k + 2] - mgc[2];
    tc[k][0] = d0 * s[0] + d1 * s[1] + d2 * s[2];
    tc[k][1] = d0 * t[0] + d1 * t[1] + d2 * t[2];
  }
  R Ar(0.0), Mx(0.0), My(0.0);
  for (int k = 0; k < 4; ++k) {
    int kn = (k + 1) & 3;
    R xk = tc[k][0], yk = tc[k][1], xk1 = tc[kn][0], yk1 = tc[kn][1];
    Ar = Ar + (yk1 - yk) * (xk + xk1) / 2.0;
    Mx = Mx + (xk1 - xk) * (yk * yk + yk * yk1 + yk1 * yk1) / 6.0;
    My = My + (yk1 - yk) * (xk * xk + xk * xk1 + xk1 * xk1) / 6.0;
  }
  R clx = My / Ar, cly = -Mx / Ar;
  for (int c = 0; c < 3; ++c) qgc[c] = mgc[c] + clx * s[c] + cly * t[c];
  for (int k = 0; k < 4; ++k) {
    lc[2 * k] = tc[k][0] - clx;
    lc[2 * k + 1] = tc[k][1] - cly;
  }
  for (int c = 0; c < 3; ++c) {
    T[c] = s[c];
    T[3 + c] = t[c];
    T[6 + c] = nn[c];
  }
}

constexpr int kGeo = 20;  // a panel's geometry in the near-field adjoint: T (9), qgc (3), lc (8)

// d/d corners from d/d (T, qgc, lc), once per panel: three forward sweeps of four corner
// coordinates each
__global__ void __launch_bounds__(64) birk_geometry_adjoint_kernel(int64_t n, const double* __restrict__ V,
                                                                   const double* __restrict__ geo,
                                                                   double* __restrict__ gv) {
  const int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 3;
  const int chunk = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) % 3);
  if (j >= n) return;
  Dn<4> v[12], T[9], q[3], lc[8];
  for (int e = 0; e < 12; ++e) v[e] = Dn<4>::var(V[12 * j + e], e - 4 * chunk);
  birk_geometry_t(v, T, q, lc);
  const double* g = geo + kGeo * j;
  for (int e = 0; e < 4; ++e) {
    double a = 0.0;
    for (int c = 0; c < 9; ++c) a = fma(g[c], T[c].d[e], a);
    for (int c = 0; c < 3; ++c) a = fma(g[9 + c], q[c].d[e], a);
    for (int c = 0; c < 8; ++c) a = fma(g[12 + c], lc[c].d[e], a);
    gv[12 * j + 4 * chunk + e] += a;
  }
}

// Reverse mode through birk_phi_and_velocity (mh_greens.cuh): L = A0 s0 + B1 s1 + B2 s2 + B3 s3 of
// the edge sums s0 (4 pi times the potential) and s1..s3 (the velocity) at the local point
// (x, y, z).  Returns s1..s3, and the derivatives of L in the point (gp) and the local corners
// (gl; the edge lengths are functions of them).  In the panel's plane (|z| <= tol) the arc-tangent
// terms are 0 as in the primal, with the tangent the reference keeps (_zero_primal_keep_tangent,
// rankine_vectorized.jl:36-37): each moves only with z, at the rate d(vz)/dz of the Birk
// Hessian (hzz = lambda rsum / (rk rk1 rho), velocity_hessian, rankine_vectorized.jl:200-235),
// which stays finite where the arc tangent is 0/0 (field point on the line of an edge).
__device__ inline void birk_reverse(double x, double y, double z, const double* lc, const double* edge, double A0,
                                    double B1, double B2, double B3, double sum[3], double gp[3], double gl[8]) {
  double sx[4], sy[4], r[4], e[4], h[4];
  double gsx[4], gsy[4], gr[4], ge[4], gh[4];
  const double z2 = z * z;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    sx[k] = x - lc[2 * k];
    sy[k] = y - lc[2 * k + 1];
    e[k] = sx[k] * sx[k] + z2;
    r[k] = fx::sqrt_pos(sy[k] * sy[k] + e[k]);
    h[k] = sx[k] * sy[k];
    gsx[k] = gsy[k] = gr[k] = ge[k] = gh[k] = 0.0;
    gl[2 * k] = gl[2 * k + 1] = 0.0;
  }
  const bool inplane = fabs(z) <= kBirkZTol;
  const double W = fma(A0, z, B3);  // adjoint of every arc-tangent term (s0 holds z s3)
  double s1 = 0.0, s2 = 0.0, s3 = 0.0, gz = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int kn = (k + 1) & 3;
    const double dk = edge[k];
    if (dk <= kBirkDkTol) continue;
    const double dx = lc[2 * kn] - lc[2 * k], dy = lc[2 * kn + 1] - lc[2 * k + 1];
    const double rs = r[k] + r[kn], num = rs - dk, inv_sum = fx::recip(rs + dk), inv_d = fx::recip(dk);
    const double w = num * inv_sum;
    const double lt = (num > 0.0 ? fx::log_pos(w) : log(w)) * inv_d;
    const double inv_num = num > 0.0 ? fx::recip(num) : 1.0 / num;
    const double cl = fma(A0, sx[k] * dy - sy[k] * dx, fma(B1, dy, -(B2 * dx)));  // adjoint of lt
    s1 = fma(dy, lt, s1);
    s2 = fma(-dx, lt, s2);
    gsx[k] = fma(A0 * dy, lt, gsx[k]);
    gsy[k] = fma(-(A0 * dx), lt, gsy[k]);
    double gdx = -lt * fma(A0, sy[k], B2), gdy = lt * fma(A0, sx[k], B1);
    // lt = log((rs - d) / (rs + d)) / d
    const double den2 = 2.0 * inv_num * inv_sum;
    gr[k] = fma(cl, den2, gr[k]);
    gr[kn] = fma(cl, den2, gr[kn]);
    const double gd = -(cl * inv_d * inv_d) * fma(rs, den2, lt);
    gdx = fma(gd, dx, gdx);
    gdy = fma(gd, dy, gdy);
    if (!inplane) {
      const double dxz = dx * z;
      const double N1 = dy * e[k] - dx * h[k], D1 = dxz * r[k];
      const double N2 = dy * e[kn] - dx * h[kn], D2 = dxz * r[kn];
      const double n1 = D1 < 0.0 ? -N1 : N1, d1 = fabs(D1), n2 = D2 < 0.0 ? -N2 : N2, d2 = fabs(D2);
      s3 += fx::atan2_int(n1 * d2 - n2 * d1, d1 * d2 + n1 * n2);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int q = c ? kn : k;
        const double N = c ? N2 : N1, D = c ? D2 : D1;
        const double m2 = fma(N, N, D * D);
        const double f = m2 > 0.0 ? (c ? -W : W) * fx::recip(m2) : 0.0;
        const double gN = f * D, gD = -f * N;
        gdy = fma(gN, e[q], gdy);
        ge[q] = fma(gN, dy, ge[q]);
        gh[q] = fma(-gN, dx, gh[q]);
        gdx = fma(gD * z, r[q], fma(-gN, h[q], gdx));
        gz = fma(gD * dx, r[q], gz);
        gr[q] = fma(gD, dxz, gr[q]);
      }
    } else {
      const double lam = sx[k] * sy[kn] - sx[kn] * sy[k];
      const double rr = r[k] * r[kn], rho = rr + sx[k] * sx[kn] + sy[k] * sy[kn] + z2;
      if (rho > 0.0) gz = fma(W, lam * rs / (rr * rho), gz);
    }
    gl[2 * kn] += gdx;
    gl[2 * k] -= gdx;
    gl[2 * kn + 1] += gdy;
    gl[2 * k + 1] -= gdy;
  }
  gz = fma(A0, s3, gz);
  double gx = 0.0, gy = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double t = r[k] > 0.0 ? gr[k] * fx::recip(r[k]) : 0.0;
    const double u = fma(2.0, ge[k], t);
    const double a = fma(gh[k], sy[k], fma(u, sx[k], gsx[k])), b = fma(gh[k], sx[k], fma(t, sy[k], gsy[k]));
    gz = fma(u, z, gz);
    gx += a;
    gy += b;
    gl[2 * k] -= a;
    gl[2 * k + 1] -= b;
  }
  sum[0] = s1;
  sum[1] = s2;
  sum[2] = s3;
  gp[0] = gx;
  gp[1] = gy;
  gp[2] = gz;
}

// ---------------------------------------------------------------------------
// static (Rankine + image, Birk) adjoint, real weights.  Direct: D = a (n_j . g) with g the
// source gradient of the panel integral at the field point (or its image).  Indirect: the
// field-point gradient of the same integral, -M g (M = diag(1, 1, -1) for the image point),
// with the field panel's normal: D = a (nv . g), nv = -M n_i.
//
// A CTA takes 128 rows by kCols columns.  Far terms (beyond 7 radii) go thread by thread, their
// column sums through a tile in shared memory.  Near terms are listed column by column and
// taken densely, 128 at a time, in reverse mode: the derivative of one scalar in the 23
// quantities of the panel's frame, centroid, local corners and normal, about 600 FP64
// instructions.  The corners follow from the frame once per panel
// (birk_geometry_adjoint_kernel).  Forward duals per pair (15 inputs in four sweeps of the whole
// geometry, some 14000 FP64 instructions paid by every warp that holds one near pair) took
// 21.6 ms for 1400 panels; now 0.5 ms.  Bound: the FP64 pipe.
// ---------------------------------------------------------------------------
constexpr int kNearVals = kGeo + 3;      // geometry and source normal
constexpr int kTileLd = kRows + 1;       // odd: the column sums read down a column
constexpr int kStaticAdjSmem = 8 * kTileLd * (7 * kCols > kNearVals ? 7 * kCols : kNearVals);

template <bool DIRECT>
__global__ void __launch_bounds__(kRows) static_adjoint_kernel(AssemblyParams p, const double* __restrict__ RS,
                                                               const double* __restrict__ RD, GradPtrs gp,
                                                               double* __restrict__ geo) {
  extern __shared__ double tile[];       // far: [7 kCols][kTileLd]; near: [kNearVals][kTileLd]
  __shared__ PanelRec sp[kCols];
  __shared__ double near2[kCols][2];     // (7 radius)^2 less / more four roundings
  __shared__ unsigned short todo[2 * kCols * kRows];  // image << 10 | column << 7 | row, by column
  __shared__ int cnt[2 * kCols][kRows / 32];          // near terms per (column, image) and warp, then offsets
  __shared__ int cstart[kCols + 1];
  const int64_t n = p.n;
  const int64_t i0 = blockIdx.x * (int64_t)kRows;
  const int64_t i = i0 + threadIdx.x;
  const int64_t j0 = blockIdx.y * (int64_t)kCols;
  const int ncol = (int)((n - j0) < kCols ? (n - j0) : kCols);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    const double2* src = reinterpret_cast<const double2*>(p.P + j0);
    double2* dst = reinterpret_cast<double2*>(sp);
    for (int q = threadIdx.x; q < ncol * 16; q += blockDim.x) dst[q] = src[q];
  }
  __syncthreads();
  if (threadIdx.x < ncol) {
    const double t = 7 * sp[threadIdx.x].radius, t2 = t * t;
    near2[threadIdx.x][0] = t2 * (1.0 - 0x1p-50);
    near2[threadIdx.x][1] = t2 * (1.0 + 0x1p-50);
  }
  __syncthreads();
  const bool active = i < n;
  double ci[3] = {0, 0, 0}, ni[3] = {0, 0, 0};
  if (active)
    for (int c = 0; c < 3; ++c) { ci[c] = p.P[i].c[c]; ni[c] = p.P[i].n[c]; }
  const bool need[2] = {(p.gfs & MH_GF_RANKINE) != 0,
                        (p.gfs & (MH_GF_RANKINE_REFLECTED | MH_GF_RANKINE_REFLECTED_NEGATIVE)) != 0};
  const double image_sign = ((p.gfs & MH_GF_RANKINE_REFLECTED) ? 1.0 : 0.0) -
                            ((p.gfs & MH_GF_RANKINE_REFLECTED_NEGATIVE) ? 1.0 : 0.0);
  double gci[3] = {0, 0, 0}, gni[3] = {0, 0, 0};
  unsigned near_mask = 0;  // bit 2 column + image
  for (int jj = 0; jj < ncol; ++jj) {
    const PanelRec& Pj = sp[jj];
    // column terms: gc_j (3), gn_j (3), ga_j (1)
    double col[7] = {0, 0, 0, 0, 0, 0, 0};
    if (active) {
      const double ws = RS[i + (j0 + jj) * n], wd = RD[i + (j0 + jj) * n];
      const double rx = ci[0] - Pj.c[0], ry = ci[1] - Pj.c[1], h2 = rx * rx + ry * ry;
#pragma unroll
      for (int img = 0; img < 2; ++img) {
        if (!need[img]) continue;
        const double zf = img ? -1.0 : 1.0;  // d pt / d ci_z
        const double rz = (img ? -ci[2] : ci[2]) - Pj.c[2];
        const double r2 = h2 + rz * rz;
        bool far = r2 > near2[jj][1];
        if (!far && r2 >= near2[jj][0]) far = sqrt(r2) > 7 * Pj.radius;
        if (!far) {
          near_mask |= 1u << (2 * jj + img);
          continue;
        }
        const double a = img ? kMinusInv4Pi * image_sign : kMinusInv4Pi;
        double nv[3];
        if (DIRECT) { nv[0] = Pj.n[0]; nv[1] = Pj.n[1]; nv[2] = Pj.n[2]; }
        else { nv[0] = -ni[0]; nv[1] = -ni[1]; nv[2] = img ? ni[2] : -ni[2]; }
        // S = a A / r, D = a A (nv . rb) / r^3
        const double rb[3] = {rx, ry, rz};
        const double ir = fx::rsqrt_pos(r2), ir2 = ir * ir, q = a * Pj.area * ir * ir2;
        const double nr = (nv[0] * rx + nv[1] * ry + nv[2] * rz) * ir2;
        const double f = fma(3.0 * wd, nr, ws);
        for (int c = 0; c < 3; ++c) {
          const double gtot = q * (wd * nv[c] - f * rb[c]);  // d/d pt_c
          gci[c] += (c == 2 ? zf : 1.0) * gtot;
          col[c] -= gtot;
        }
        col[6] += a * ir * fma(wd, nr, ws);  // d/d A_j
        const double wq = wd * q;
        for (int c = 0; c < 3; ++c) {
          if (DIRECT) col[3 + c] += wq * rb[c];
          else gni[c] -= wq * (c == 2 ? zf : 1.0) * rb[c];
        }
      }
    }
    for (int c = 0; c < 7; ++c) tile[(7 * jj + c) * kTileLd + threadIdx.x] = col[c];
  }
  // near terms per column, image and warp
  for (int b = 0; b < 2 * kCols; ++b) {
    const unsigned m = __ballot_sync(0xffffffffu, (near_mask >> b) & 1u);
    if (lane == 0) cnt[b][warp] = __popc(m);
  }
  __syncthreads();
  // column sums of the far terms, two threads each
  for (int t = threadIdx.x; t < 2 * 7 * ncol; t += kRows) {
    const int v = t >> 1;
    const double* src = tile + v * kTileLd + (t & 1) * (kRows / 2);
    double a = 0.0, b = 0.0;
    for (int q = 0; q < kRows / 2; q += 2) {
      a += src[q];
      b += src[q + 1];
    }
    a += b;
    const int64_t j = j0 + v / 7;
    const int c = v % 7;
    atomicAdd(c < 3 ? gp.gc + 3 * j + c : (c < 6 ? gp.gn + 3 * j + c - 3 : gp.ga + j), a);
  }
  if (threadIdx.x == 0) {
    int base = 0;
    for (int b = 0; b < 2 * kCols; ++b) {
      if ((b & 1) == 0) cstart[b >> 1] = base;
      for (int w = 0; w < kRows / 32; ++w) {
        const int c = cnt[b][w];
        cnt[b][w] = base;
        base += c;
      }
    }
    cstart[kCols] = base;
  }
  __syncthreads();
  for (int b = 0; b < 2 * kCols; ++b) {
    const bool mine = (near_mask >> b) & 1u;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (mine)
      todo[cnt[b][warp] + __popc(m & ((1u << lane) - 1u))] =
          (unsigned short)((b & 1) << 10 | (b >> 1) << 7 | (int)threadIdx.x);
  }
  __syncthreads();
  const int total = cstart[kCols];
  for (int base = 0; base < total; base += kRows) {
    const int q = base + threadIdx.x;
    if (q < total) {
      const int ent = todo[q], img = ent >> 10, jj = (ent >> 7) & 7, row = ent & 127;
      const PanelRec& Pj = sp[jj];
      const PanelRec& Pi = p.P[i0 + row];
      const int64_t idx = i0 + row + (j0 + jj) * n;
      const double zf = img ? -1.0 : 1.0, a = img ? kMinusInv4Pi * image_sign : kMinusInv4Pi;
      const double ws = a * RS[idx], wd = a * RD[idx];
      double nv[3];
      for (int c = 0; c < 3; ++c) nv[c] = DIRECT ? Pj.n[c] : -(c == 2 ? zf : 1.0) * __ldg(&Pi.n[c]);
      const double d[3] = {__ldg(&Pi.c[0]) - Pj.qgc[0], __ldg(&Pi.c[1]) - Pj.qgc[1],
                           zf * __ldg(&Pi.c[2]) - Pj.qgc[2]};
      const double* T = Pj.T;
      double loc[3], nl[3];
      for (int c = 0; c < 3; ++c) {
        loc[c] = T[3 * c] * d[0] + T[3 * c + 1] * d[1] + T[3 * c + 2] * d[2];
        nl[c] = T[3 * c] * nv[0] + T[3 * c + 1] * nv[1] + T[3 * c + 2] * nv[2];
      }
      // S = a s0, D = a (nv . g) with g = -(s s1 + t s2 + n s3)
      double sum[3], gl3[3], gl[8];
      birk_reverse(loc[0], loc[1], loc[2], Pj.lc, Pj.edge, ws, -wd * nl[0], -wd * nl[1], -wd * nl[2], sum, gl3, gl);
      double* out = tile + threadIdx.x;
      for (int c = 0; c < 3; ++c)
        for (int x = 0; x < 3; ++x) out[(3 * c + x) * kTileLd] = fma(gl3[c], d[x], -(wd * sum[c]) * nv[x]);
      for (int x = 0; x < 3; ++x) {
        const double gx = T[x] * gl3[0] + T[3 + x] * gl3[1] + T[6 + x] * gl3[2];  // d/d pt
        const double wg = -wd * (T[x] * sum[0] + T[3 + x] * sum[1] + T[6 + x] * sum[2]);  // d/d nv
        out[(9 + x) * kTileLd] = -gx;
        out[(kGeo + x) * kTileLd] = DIRECT ? wg : 0.0;
        atomicAdd(gp.gc + 3 * (i0 + row) + x, x == 2 ? zf * gx : gx);
        if (!DIRECT) atomicAdd(gp.gn + 3 * (i0 + row) + x, -(x == 2 ? zf : 1.0) * wg);
      }
      for (int c = 0; c < 8; ++c) out[(12 + c) * kTileLd] = gl[c];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kNearVals * ncol; t += kRows) {
      const int v = t % kNearVals, jj = t / kNearVals;
      const int q0 = max(cstart[jj], base) - base, q1 = min(cstart[jj + 1], base + kRows) - base;
      if (q0 >= q1 || (!DIRECT && v >= kGeo)) continue;
      double s0 = 0.0, s1 = 0.0;
      for (int e = q0; e < q1; ++e) {
        if (e & 1) s1 += tile[v * kTileLd + e];
        else s0 += tile[v * kTileLd + e];
      }
      const int64_t j = j0 + jj;
      atomicAdd(v < kGeo ? geo + kGeo * j + v : gp.gn + 3 * j + v - kGeo, s0 + s1);
    }
    __syncthreads();
  }
  if (active)
    for (int c = 0; c < 3; ++c) {
      atomicAdd(gp.gc + 3 * i + c, gci[c]);
      if (!DIRECT) atomicAdd(gp.gn + 3 * i + c, gni[c]);
    }
}

// ---------------------------------------------------------------------------
// wave adjoint (Wu or exact Delhommeau), one wavenumber, complex rank-nh weights
// ---------------------------------------------------------------------------
struct WaveWeights {
  const double2* lS;  // n x nh:  W^S_ij = c sum_h lS_h[i] rS_h[j]
  const double2* rS;
  const double2* lD;  //          W^D_ij = -c sum_h lD_h[i] rD_h[j]
  const double2* rD;
  int nh;
  double2 c;          // objective factor of this frequency
};

__device__ __forceinline__ double2 cmulz(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// c + a b
__device__ __forceinline__ double2 cmadd(double2 c, double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}

constexpr int kWaveWu = 1, kWaveExact = 2;

// index of the unordered pair i <= j in the packed upper triangle
__device__ __forceinline__ int64_t packed_pair(int64_t i, int64_t j) { return j * (j + 1) / 2 + i; }

// The exact term and its first and second derivatives in (r, z) = (hh, vv) as duals, from
// G and dG/dr at the pair: dG/dz = G + 2/d (d = |(r, z)|, the relation the primal uses,
// exact_Guevel_Delhommeau.jl:52-59), so G_zz = G_z - 2 z/d^3 and G_rz = G_r - 2 r/d^3; the
// wave term is harmonic below the free surface, so G_rr = -G_r/r - G_zz.  For r <= 1e-6
// (where the primal zeroes every horizontal term) G_rr only ever meets zero weights and is
// set to 0.
__device__ void egd_terms_from_values(double2 G, double2 Gr, double r, double z, CR<Dn<2>>& GF, CR<Dn<2>>& Gh,
                                      CR<Dn<2>>& Gv) {
  const double d = hypot(r, z);
  const double id3 = 1.0 / (d * d * d);
  const double2 Gz = make_double2(G.x + 2 / d, G.y);
  const double2 Gzz = make_double2(Gz.x - 2.0 * z * id3, Gz.y);
  const double2 Grz = make_double2(Gr.x - 2.0 * r * id3, Gr.y);
  const double2 Grr = fabs(r) > 1e-6 ? make_double2(-Gr.x / r - Gzz.x, -Gr.y / r - Gzz.y) : make_double2(0.0, 0.0);
  GF.x.v = G.x;   GF.x.d[0] = Gr.x;  GF.x.d[1] = Gz.x;
  GF.y.v = G.y;   GF.y.d[0] = Gr.y;  GF.y.d[1] = Gz.y;
  Gh.x.v = Gr.x;  Gh.x.d[0] = Grr.x; Gh.x.d[1] = Grz.x;
  Gh.y.v = Gr.y;  Gh.y.d[0] = Grr.y; Gh.y.d[1] = Grz.y;
  Gv.x.v = Gz.x;  Gv.x.d[0] = Grz.x; Gv.x.d[1] = Gzz.x;
  Gv.y.v = Gz.y;  Gv.y.d[0] = Grz.y; Gv.y.d[1] = Gzz.y;
}

// contribution of one oriented pair (field f, source s) to the gradient:
// S = sc k a_s GF, D = sc a_s k^2 (u Gh + n3 Gv) with u = (n1 dx + n2 dy)/dis,
// (dx, dy) = source - field horizontal offset.
struct PairGrad {
  double gcf[3], gcs[3], gns[3], gas;
};

__device__ __forceinline__ void wave_pair_grad(double k, double ux, double uy, double inv_dis, double as,
                                               const double ns[3], const CR<Dn<2>>& GF, const CR<Dn<2>>& Gh,
                                               const CR<Dn<2>>& Gv, double2 WS, double2 WD, PairGrad& o) {
  // the weights' real products with GF, Gh, Gv and their derivatives first; everything after is
  // real: sa = sc k a_s, and A, B the derivatives in hh and vv
  auto re = [](double2 w, double x, double y) { return fma(w.x, x, -(w.y * y)); };
  const double sck = kMinusInv4Pi * k, sa = sck * as, sak = sa * k;
  const double F = re(WS, GF.x.v, GF.y.v), Fh = re(WS, GF.x.d[0], GF.y.d[0]), Fv = re(WS, GF.x.d[1], GF.y.d[1]);
  const double H = re(WD, Gh.x.v, Gh.y.v), Hh = re(WD, Gh.x.d[0], Gh.y.d[0]), Hv = re(WD, Gh.x.d[1], Gh.y.d[1]);
  const double V = re(WD, Gv.x.v, Gv.y.v), Vh = re(WD, Gv.x.d[0], Gv.y.d[0]), Vv = re(WD, Gv.x.d[1], Gv.y.d[1]);
  const double u = fma(ns[0], ux, ns[1] * uy);
  const double A = fma(sak, fma(u, Hh, ns[2] * Vh), sa * Fh);
  const double B = fma(sak, fma(u, Hv, ns[2] * Vv), sa * Fv);
  o.gas = sck * fma(k, fma(u, H, ns[2] * V), F);
  const double sH = sak * H;
  o.gns[0] = sH * ux;
  o.gns[1] = sH * uy;
  o.gns[2] = sak * V;
  // hh = k |(dx, dy)| and u = n . (dx, dy) / |(dx, dy)|: (ux, uy) and inv_dis are 0 where the primal
  // treats the pair as vertically aligned (hh <= 1e-6, which also catches centres whose
  // horizontal offset is rounding noise): no direction is preferred there and the derivative is
  // taken as 0, the central difference of the kink.
  const double kA = k * A, sHd = sH * inv_dis;
  const double gdx = fma(sHd, fma(-u, ux, ns[0]), kA * ux), gdy = fma(sHd, fma(-u, uy, ns[1]), kA * uy);
  o.gcs[0] = gdx; o.gcs[1] = gdy; o.gcs[2] = k * B;  // vv = k (z_f + z_s)
  o.gcf[0] = -gdx; o.gcf[1] = -gdy; o.gcf[2] = o.gcs[2];
}

// The sums over the warp of eight numbers per lane in nine additions (a butterfly for each would take
// 40 of the FP64 pipe's slots): every step halves the numbers a lane carries.  Lane 4 q holds
// number q's (bits 4, 3 and 2 of the lane are q's bits 2, 1 and 0).
__device__ __forceinline__ double warp_sum8(const double (&x)[8], int lane) {
  double a[4], b[2];
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double got = __shfl_xor_sync(0xffffffffu, h4 ? x[q] : x[q + 4], 16);
    a[q] = (h4 ? x[q + 4] : x[q]) + got;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const double got = __shfl_xor_sync(0xffffffffu, h3 ? a[q] : a[q + 2], 8);
    b[q] = (h3 ? a[q + 2] : a[q]) + got;
  }
  double c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  return c + __shfl_xor_sync(0xffffffffu, c, 1);
}

// One thread per unordered pair (i <= j), both orientations.  DIRECT: the pair (field f,
// source s) enters D through the source normal and the offset s - f; indirect: through the
// field normal and the offset f - s.  WAVE: the Wu fits on duals, or the exact term from the
// packed values gv[2q] = G, gv[2q + 1] = dG/dr of pair q.
// Bound: the FP64 pipe (82 % busy at 660 warp instructions per pair).  The weights are therefore
// contracted with the term before anything else, so that both orientations' chains are real, the
// Struve and Bessel values are differentiated as plain numbers, the objective's factor is on the
// weights, and a column's sums take 9 additions per warp instead of 35: 1400 panels 1.67 -> 1.23 ms
// per frequency.
template <bool DIRECT, int WAVE>
__global__ void __launch_bounds__(kRows) wave_adjoint_kernel(AssemblyParams p, double k, WaveWeights w,
                                                             const double2* __restrict__ gv, GradPtrs gp) {
  __shared__ PanelRec sp[kCols];
  __shared__ double2 slS[kCols][kMaxH], srS[kCols][kMaxH], slD[kCols][kMaxH], srD[kCols][kMaxH];
  __shared__ double red[2][8][kRows / 32];
  const int64_t n = p.n;
  const int64_t i0 = blockIdx.x * (int64_t)kRows;
  const int64_t j0 = blockIdx.y * (int64_t)kCols;
  if (i0 > j0 + kCols - 1) return;  // strictly below the diagonal
  const int64_t i = i0 + threadIdx.x;
  const int ncol = (int)((n - j0) < kCols ? (n - j0) : kCols);
  {
    const double2* src = reinterpret_cast<const double2*>(p.P + j0);
    double2* dst = reinterpret_cast<double2*>(sp);
    for (int q = threadIdx.x; q < ncol * 16; q += blockDim.x) dst[q] = src[q];
    for (int q = threadIdx.x; q < ncol * w.nh; q += blockDim.x) {
      int jj = q % ncol, h = q / ncol;
      slS[jj][h] = cmulz(w.c, w.lS[(j0 + jj) + h * n]);  // the objective's factor c, and -c for D
      srS[jj][h] = w.rS[(j0 + jj) + h * n];
      slD[jj][h] = cmulz(make_double2(-w.c.x, -w.c.y), w.lD[(j0 + jj) + h * n]);
      srD[jj][h] = w.rD[(j0 + jj) + h * n];
    }
  }
  __syncthreads();
  const bool active = i < n;
  double ci[3] = {0, 0, 0}, ni[3] = {0, 0, 0}, ai = 0.0;
  double2 lSi[kMaxH], rSi[kMaxH], lDi[kMaxH], rDi[kMaxH];
  if (active) {
    for (int c = 0; c < 3; ++c) { ci[c] = p.P[i].c[c]; ni[c] = p.P[i].n[c]; }
    ai = p.P[i].area;
    for (int h = 0; h < w.nh; ++h) {
      lSi[h] = cmulz(w.c, w.lS[i + h * n]); rSi[h] = w.rS[i + h * n];
      lDi[h] = cmulz(make_double2(-w.c.x, -w.c.y), w.lD[i + h * n]); rDi[h] = w.rD[i + h * n];
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t first = i - lane;  // the warp's first row
  using Step = typename std::conditional<WAVE == kWaveWu, CtaStep, NoStep>::type;
  double gci[3] = {0, 0, 0}, gni[3] = {0, 0, 0}, gai = 0.0;
  for (int jj = 0; jj < ncol; ++jj) {
    const int64_t j = j0 + jj;
    const PanelRec& Pj = sp[jj];
    double col[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // gc_j (3), gn_j (3), ga_j
    // whole warps walk through the term (rows past n at the origin of a panel, discarded)
    if (first > j || first >= n) {
      Step()();
      Step()();
    } else {
      double hh, vv;
      reduced_coords(ci, Pj.c, k, hh, vv);
      CR<Dn<2>> GF, Gh, Gv;
      if (WAVE == kWaveWu) {
        wu_terms_t(Dn<2>::var(hh, 0), Dn<2>::var(vv, 1), GF, Gh, Gv, Step());
      } else if (active && i <= j) {
        const int64_t q = packed_pair(i, j);
        egd_terms_from_values(gv[2 * q], gv[2 * q + 1], hh, vv, GF, Gh, Gv);
      }
      if (active && i <= j) {
        const double dx = Pj.c[0] - ci[0], dy = Pj.c[1] - ci[1];
        const double dis = fx::sqrt_pos(dx * dx + dy * dy);
        const double inv_dis = k * dis > 1e-6 ? fx::recip_call(dis) : 0.0;
        const double ux = dx * inv_dis, uy = dy * inv_dis;
        // weights of (i, j) and (j, i)
        double2 WSij = make_double2(0, 0), WDij = WSij, WSji = WSij, WDji = WSij;
        for (int h = 0; h < w.nh; ++h) {
          WSij = cmadd(WSij, lSi[h], srS[jj][h]);
          WDij = cmadd(WDij, lDi[h], srD[jj][h]);
          WSji = cmadd(WSji, slS[jj][h], rSi[h]);
          WDji = cmadd(WDji, slD[jj][h], rDi[h]);
        }
        PairGrad g1;  // field i, source j
        if (DIRECT) {
          wave_pair_grad(k, ux, uy, inv_dis, Pj.area, Pj.n, GF, Gh, Gv, WSij, WDij, g1);
          for (int c = 0; c < 3; ++c) { gci[c] += g1.gcf[c]; col[c] += g1.gcs[c]; col[3 + c] += g1.gns[c]; }
        } else {
          wave_pair_grad(k, -ux, -uy, inv_dis, Pj.area, ni, GF, Gh, Gv, WSij, WDij, g1);
          for (int c = 0; c < 3; ++c) { gci[c] += g1.gcs[c]; col[c] += g1.gcf[c]; gni[c] += g1.gns[c]; }
        }
        col[6] += g1.gas;
        if (i != j) {
          PairGrad g2;  // field j, source i
          if (DIRECT) {
            wave_pair_grad(k, -ux, -uy, inv_dis, ai, ni, GF, Gh, Gv, WSji, WDji, g2);
            for (int c = 0; c < 3; ++c) { col[c] += g2.gcf[c]; gci[c] += g2.gcs[c]; gni[c] += g2.gns[c]; }
          } else {
            wave_pair_grad(k, ux, uy, inv_dis, ai, Pj.n, GF, Gh, Gv, WSji, WDji, g2);
            for (int c = 0; c < 3; ++c) { col[c] += g2.gcs[c]; gci[c] += g2.gcf[c]; col[3 + c] += g2.gns[c]; }
          }
          gai += g2.gas;
        }
      }
    }
    const double sum = warp_sum8(col, lane);
    if ((lane & 3) == 0) red[jj & 1][lane >> 2][warp] = sum;
    __syncthreads();
    if (threadIdx.x < 7) {  // a number each; the other buffer is written before the next barrier
      const double* r = red[jj & 1][threadIdx.x];
      double* to = threadIdx.x < 3 ? gp.gc + 3 * j + threadIdx.x
                                   : (threadIdx.x < 6 ? gp.gn + 3 * j + (threadIdx.x - 3) : gp.ga + j);
      atomicAdd(to, (r[0] + r[1]) + (r[2] + r[3]));
    }
  }
  if (active) {
    for (int c = 0; c < 3; ++c) {
      atomicAdd(gp.gc + 3 * i + c, gci[c]);
      atomicAdd(gp.gn + 3 * i + c, gni[c]);
    }
    atomicAdd(gp.ga + i, gai);
  }
}

// G and dG/dr of the exact term for every unordered pair (i <= j) at wavenumber k, packed
// (pair q = j (j + 1)/2 + i at out[2q], out[2q + 1]), one thread per pair, as in the primal.
constexpr int kEgdThreads = 128;
__global__ void __launch_bounds__(kEgdThreads) egd_pair_values_kernel(AssemblyParams p, double k, int64_t npairs,
                                                                      double2* __restrict__ out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= npairs) return;
  int64_t j = (int64_t)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
  while (j * (j + 1) / 2 > q) --j;
  while ((j + 1) * (j + 2) / 2 <= q) ++j;
  const int64_t i = q - j * (j + 1) / 2;
  double r, z;
  reduced_coords(p.P[i].c, p.P[j].c, k, r, z);
  if (!egd_takes_quadrature(r, z)) egd_values(r, z, out[2 * q], out[2 * q + 1]);
}

// the same for the pairs above the surface, a warp each (wave_quadrature_kernel, mh_assembly.cu)
__global__ void __launch_bounds__(kEgdThreads) egd_pair_quadrature_kernel(AssemblyParams p, double k,
                                                                          double2* __restrict__ out) {
  __shared__ double sw[kEgdThreads / 32][8 * kGKWarpStack];
  const int64_t n = p.n;
  if (!egd_any_quadrature(p, k)) return;
  for_items_by_warp(
      n * n,
      [&](int64_t t) {
        const int64_t j = t / n, i = t - j * n;
        return i <= j && egd_pair_takes_quadrature(p.P[i].c, p.P[j].c, k);
      },
      [&](int64_t t) {
        const int64_t j = t / n, i = t - j * n, pair = packed_pair(i, j);
        double r, z;
        reduced_coords(p.P[i].c, p.P[j].c, k, r, z);
        double2 G, Gr;
        egd_pair_quadrature(r, z, p.quad_rtol, p.quad_atol, sw[threadIdx.x >> 5], &G, &Gr);
        if ((threadIdx.x & 31) == 0) {
          out[2 * pair] = G;
          out[2 * pair + 1] = Gr;
        }
      });
}

// dS/dk and dD/dk of the exact term from the packed values: S = sc a k G(k dis, k Z) and
// D = sc a k^2 (u G_r + n_3 G_z) (u = n . offset / dis, zero for r <= 1e-6), so with
// (r, z) = k (dis, Z):  dS/dk = sc a (G + r G_r + z G_z),
// dD/dk = sc a k (2 (u G_r + n_3 G_z) + u (r G_rr + z G_rz) + n_3 (r G_rz + z G_zz)).
template <bool DIRECT>
__global__ void __launch_bounds__(kRows) egd_dk_kernel(AssemblyParams p, double k, const double2* __restrict__ gv,
                                                       double2* __restrict__ dS, double2* __restrict__ dD) {
  __shared__ PanelRec sp[kCols];
  const int64_t n = p.n;
  const int64_t i0 = blockIdx.x * (int64_t)kRows;
  const int64_t j0 = blockIdx.y * (int64_t)kCols;
  const int64_t i = i0 + threadIdx.x;
  const int ncol = (int)((n - j0) < kCols ? (n - j0) : kCols);
  {
    const double2* src = reinterpret_cast<const double2*>(p.P + j0);
    double2* dst = reinterpret_cast<double2*>(sp);
    for (int q = threadIdx.x; q < ncol * 16; q += blockDim.x) dst[q] = src[q];
  }
  __syncthreads();
  if (i >= n) return;
  double ci[3], ni[3];
  for (int c = 0; c < 3; ++c) { ci[c] = p.P[i].c[c]; ni[c] = p.P[i].n[c]; }
  for (int jj = 0; jj < ncol; ++jj) {
    const int64_t j = j0 + jj;
    const PanelRec& Pj = sp[jj];
    double r, z;
    reduced_coords(ci, Pj.c, k, r, z);
    const int64_t q = i <= j ? packed_pair(i, j) : packed_pair(j, i);
    CR<Dn<2>> GF, Gh, Gv;
    egd_terms_from_values(gv[2 * q], gv[2 * q + 1], r, z, GF, Gh, Gv);
    const double dx1 = DIRECT ? Pj.c[0] - ci[0] : ci[0] - Pj.c[0];
    const double dx2 = DIRECT ? Pj.c[1] - ci[1] : ci[1] - Pj.c[1];
    double nv[3];
    if (p.has_fixed) { nv[0] = p.fixed[0]; nv[1] = p.fixed[1]; nv[2] = p.fixed[2]; }
    else if (DIRECT) { nv[0] = Pj.n[0]; nv[1] = Pj.n[1]; nv[2] = Pj.n[2]; }
    else { nv[0] = ni[0]; nv[1] = ni[1]; nv[2] = ni[2]; }
    const double u = fabs(r) > 1e-6 ? k / r * (nv[0] * dx1 + nv[1] * dx2) : 0.0;
    const double a = kMinusInv4Pi * Pj.area;
    const double n3 = nv[2];
    dS[i + j * n] = make_double2(a * (GF.x.v + r * GF.x.d[0] + z * GF.x.d[1]),
                                 a * (GF.y.v + r * GF.y.d[0] + z * GF.y.d[1]));
    const double ux = fabs(r) > 1e-6 ? 1.0 : 0.0;  // the horizontal term is absent for r <= 1e-6
    dD[i + j * n] = make_double2(
        a * k * (2.0 * (u * Gh.x.v + n3 * Gv.x.v) + ux * u * (r * Gh.x.d[0] + z * Gh.x.d[1]) +
                 n3 * (r * Gv.x.d[0] + z * Gv.x.d[1])),
        a * k * (2.0 * (u * Gh.y.v + n3 * Gv.y.v) + ux * u * (r * Gh.y.d[0] + z * Gh.y.d[1]) +
                 n3 * (r * Gv.y.d[0] + z * Gv.y.d[1])));
  }
}

// out[i + j n] = alpha sum_h U[i + h n] conj(V[j + h n])  (a rank-nh outer product, N x N)
__global__ void outer_adj_kernel(int64_t n, int nh, const double2* __restrict__ U, const double2* __restrict__ V,
                                 double alpha, double2* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t j = blockIdx.y;
  if (i >= n) return;
  double2 s = make_double2(0.0, 0.0);
  for (int h = 0; h < nh; ++h) {
    const double2 u = U[i + h * n], v = V[j + h * n];
    s.x += u.x * v.x + u.y * v.y;
    s.y += u.y * v.x - u.x * v.y;
  }
  out[i + j * n] = make_double2(alpha * s.x, alpha * s.y);
}

// dS_W/dk and dD_W/dk of the Wu term (the S, D entries of _assemble_wu_centers_loop,
// matrix_assembly.jl:343-369, differentiated in the wavenumber): hh = k dis and
// vv = k (z_i + z_j) carry their k-derivatives dis and z_i + z_j as one dual direction
// through the same fits, and k itself is the seeded variable of the prefactors.  One
// thread per unordered pair (as in wave_kernel; every ordered pair, always eight columns per CTA:
// 450 panels 238 us, now 96); the Rankine part does not depend on k.
template <bool DIRECT>
__global__ void __launch_bounds__(kRows) wave_dk_kernel(AssemblyParams p, const double* __restrict__ ks,
                                                        double2* __restrict__ dS, double2* __restrict__ dD,
                                                        int cols) {
  __shared__ PanelRec sp[kCols];
  const int64_t n = p.n;
  const int64_t i0 = blockIdx.x * (int64_t)kRows;
  const int64_t j0 = blockIdx.y * (int64_t)cols;
  if (i0 > j0 + cols - 1) return;  // strictly below the diagonal
  const int64_t i = i0 + threadIdx.x, first = i - (threadIdx.x & 31);
  const int ncol = (int)((n - j0) < cols ? (n - j0) : cols);
  {
    const double2* src = reinterpret_cast<const double2*>(p.P + j0);
    double2* dst = reinterpret_cast<double2*>(sp);
    for (int q = threadIdx.x; q < ncol * 16; q += blockDim.x) dst[q] = src[q];
  }
  __syncthreads();
  const double k = ks[0];
  const int64_t il = i < n ? i : n - 1;
  double ci[3], ni[3];
  for (int c = 0; c < 3; ++c) { ci[c] = p.P[il].c[c]; ni[c] = p.P[il].n[c]; }
  const double ai = p.P[il].area;
  for (int jj = 0; jj < ncol; ++jj) {
    const int64_t j = j0 + jj;
    const PanelRec& Pj = sp[jj];
    if (first > j || first >= n) {  // the barriers of wu_terms_t
      CtaStep()();
      CtaStep()();
      continue;
    }
    // _wu_reduced_hh_vv (wu.jl:7-18)
    const double d2 = (ci[0] - Pj.c[0]) * (ci[0] - Pj.c[0]) + (ci[1] - Pj.c[1]) * (ci[1] - Pj.c[1]);
    const double purt = 1e-18;
    const double dis = (d2 == 0) ? sqrt(d2 + purt * purt) - purt : fx::sqrt_pos(d2);
    const double zz = ci[2] + Pj.c[2];
    Dn<1> H(k * dis), V(k * zz), K = Dn<1>::var(k, 0);
    H.d[0] = dis;
    V.d[0] = zz;
    CR<Dn<1>> GF, Gh, Gv;
    wu_terms_t(H, V, GF, Gh, Gv, CtaStep());
    if (i > j || i >= n) continue;
    const double dx1 = DIRECT ? Pj.c[0] - ci[0] : ci[0] - Pj.c[0];
    const double dx2 = DIRECT ? Pj.c[1] - ci[1] : ci[1] - Pj.c[1];
    // _wu_sd (wu.jl:112-127) on duals: s = k GF a, g = k (k^2/hh dx Gh, k^2/hh dy Gh, k Gv)
    Dn<1> dr1(0.0), dr2(0.0);
    if (fabs(H.v) > 1e-6) {
      const Dn<1> f = K * K / H;
      dr1 = f * dx1;
      dr2 = f * dx2;
    }
    const Dn<1> sr = K * GF.x, si = K * GF.y;
    const Dn<1> g0r = K * (dr1 * Gh.x), g0i = K * (dr1 * Gh.y);
    const Dn<1> g1r = K * (dr2 * Gh.x), g1i = K * (dr2 * Gh.y);
    const Dn<1> g2r = K * (K * Gv.x), g2i = K * (K * Gv.y);
    double nv[3];
    if (p.has_fixed) { nv[0] = p.fixed[0]; nv[1] = p.fixed[1]; nv[2] = p.fixed[2]; }
    else if (DIRECT) { nv[0] = Pj.n[0]; nv[1] = Pj.n[1]; nv[2] = Pj.n[2]; }
    else { nv[0] = ni[0]; nv[1] = ni[1]; nv[2] = ni[2]; }
    const double a = kMinusInv4Pi * Pj.area;
    const int64_t idx = i + j * n;
    dS[idx] = make_double2(a * sr.d[0], a * si.d[0]);
    dD[idx] = make_double2(a * (nv[0] * g0r.d[0] + nv[1] * g1r.d[0] + nv[2] * g2r.d[0]),
                           a * (nv[0] * g0i.d[0] + nv[1] * g1i.d[0] + nv[2] * g2i.d[0]));
    if (i == j) continue;
    // (j, i): the horizontal offset changes its sign, area and normal are the other panel's
    if (!p.has_fixed)
      for (int c = 0; c < 3; ++c) nv[c] = DIRECT ? ni[c] : Pj.n[c];
    const double am = kMinusInv4Pi * ai;
    const int64_t mdx = j + i * n;
    dS[mdx] = make_double2(am * sr.d[0], am * si.d[0]);
    dD[mdx] = make_double2(am * (nv[2] * g2r.d[0] - nv[0] * g0r.d[0] - nv[1] * g1r.d[0]),
                           am * (nv[2] * g2i.d[0] - nv[0] * g0i.d[0] - nv[1] * g1i.d[0]));
  }
}

// RS += Re(c sum_h lS_h rS_h^T), RD += Re(-c sum_h lD_h rD_h^T)
__global__ void weights_accumulate_kernel(int64_t n, WaveWeights w, double* __restrict__ RS, double* __restrict__ RD) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t j = blockIdx.y;
  if (i >= n) return;
  double2 s = make_double2(0, 0), d = s;
  for (int h = 0; h < w.nh; ++h) {
    s = zadd(s, cmulz(w.lS[i + h * n], w.rS[j + h * n]));
    d = zadd(d, cmulz(w.lD[i + h * n], w.rD[j + h * n]));
  }
  s = cmulz(w.c, s);
  d = cmulz(w.c, d);
  RS[i + j * n] += s.x;
  RD[i + j * n] -= d.x;
}

// O(N) terms of one frequency (direct): force weights w_h = i rho omega (-n . dof_h) a and
// boundary conditions b_h = -i omega (n . dof_h) depend on n and a.
//   Re(c phi_h[i] dw_h[i]) + Re(c t_h[i] db_h[i]),  t_h = S^T lam_h
// O(N) terms of one frequency (direct) for cotangents c[q, col] (influenced q; columns: the
// n_rad radiating dofs, then the n_beta headings; J = sum Re(c F), F the forces of the
// columns plus, for the headings, the Froude-Krylov forces):
//   force weights  f_q = i rho omega (-n . dof_q) a, paired with psi_q = sum_col c[q, col] phi_col;
//   radiation      b_r = -i omega (n . dof_r), paired with t_r = S^T lam_r (lam = D^-T w);
//   diffraction    b_beta = -(v . n), v = omega e^{k z} e^{i k wbar} (cos b, sin b, -i), also
//                  paired with t_beta, depends on the centre through e^{kz + ikwbar};
//   Froude-Krylov  sum p_beta (-n . dof_q) a, p_beta = rho g e^{k z} e^{i k wbar}.
// Each thread owns one panel.
__global__ void rhs_adjoint_kernel(int64_t n, const double* __restrict__ N, const double* __restrict__ A,
                                   const double* __restrict__ C, const double* __restrict__ dofs,
                                   const int32_t* __restrict__ rad, int n_rad, const int32_t* __restrict__ inf,
                                   int n_inf, int n_beta, const double* __restrict__ betas, double omega, double rho,
                                   double gacc, const double2* __restrict__ cw, const double2* __restrict__ phi,
                                   const double2* __restrict__ t, double* __restrict__ gc, double* __restrict__ gn,
                                   double* __restrict__ ga, double* __restrict__ gd) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ncol = n_rad + n_beta;
  const double n0 = N[3 * i], n1 = N[3 * i + 1], n2 = N[3 * i + 2], a = A[i];
  const double k = omega * omega / gacc;
  double g0 = 0, g1 = 0, g2 = 0, gav = 0, c0 = 0, c1 = 0, c2 = 0;
  for (int q = 0; q < n_inf; ++q) {
    const double* dof = dofs + (int64_t)inf[q] * n * 3 + 3 * i;
    const double disp = n0 * dof[0] + n1 * dof[1] + n2 * dof[2];
    double2 psi = make_double2(0.0, 0.0);
    for (int r = 0; r < ncol; ++r) psi = zadd(psi, cmulz(cw[q + (int64_t)r * n_inf], phi[i + (int64_t)r * n]));
    // Re(psi * i s) = -s Im(psi):  d/dn with s = rho omega (-dof) a, d/da with s = rho omega (-disp)
    double re = -psi.y * rho * omega;  // coefficient of the real factor (-disp a) below
    // Froude-Krylov of every heading: Re(c p) times the same real factor, and its centre terms
    for (int b = 0; b < n_beta; ++b) {
      double sb, cb;
      sincos(betas[b], &sb, &cb);
      const double wbar = C[3 * i] * cb + C[3 * i + 1] * sb;
      double sw, cw_;
      sincos(k * wbar, &sw, &cw_);
      const double pa = rho * gacc * exp(k * C[3 * i + 2]);
      const double2 cp = cmulz(cw[q + (int64_t)(n_rad + b) * n_inf], make_double2(pa * cw_, pa * sw));
      re += cp.x;
      // d p / d centre = p (i k cos b, i k sin b, k):  Re(cp (i k cos b)) = -k cos b Im(cp)
      const double f = -disp * a;
      c0 += -k * cb * cp.y * f;
      c1 += -k * sb * cp.y * f;
      c2 += k * cp.x * f;
    }
    g0 += re * (-dof[0] * a);
    g1 += re * (-dof[1] * a);
    g2 += re * (-dof[2] * a);
    gav += re * (-disp);
    double* gdi = gd + ((int64_t)inf[q] * n + i) * 3;
    gdi[0] += re * (-n0 * a);
    gdi[1] += re * (-n1 * a);
    gdi[2] += re * (-n2 * a);
  }
  for (int r = 0; r < n_rad; ++r) {
    const double* dof = dofs + (int64_t)rad[r] * n * 3 + 3 * i;
    // b = -i omega disp:  Re(t (-i omega) x) = omega Im(t) x for x = dof (d/dn) and x = n (d/d dof)
    const double ty = t[i + (int64_t)r * n].y;
    g0 += omega * ty * dof[0];
    g1 += omega * ty * dof[1];
    g2 += omega * ty * dof[2];
    double* gdi = gd + ((int64_t)rad[r] * n + i) * 3;
    gdi[0] += omega * ty * n0;
    gdi[1] += omega * ty * n1;
    gdi[2] += omega * ty * n2;
  }
  for (int b = 0; b < n_beta; ++b) {
    double sb, cb;
    sincos(betas[b], &sb, &cb);
    const double wbar = C[3 * i] * cb + C[3 * i + 1] * sb;
    double sw, cw_;
    sincos(k * wbar, &sw, &cw_);
    const double e = omega * exp(k * C[3 * i + 2]);
    const double2 amp = make_double2(e * cw_, e * sw);  // v = amp (cos b, sin b, -i)
    const double2 v0 = make_double2(amp.x * cb, amp.y * cb), v1 = make_double2(amp.x * sb, amp.y * sb);
    const double2 v2 = make_double2(amp.y, -amp.x);
    const double2 tb = t[i + (int64_t)(n_rad + b) * n];
    // b = -(v . n):  d/dn = -v;  d/dc = b (i k cos b, i k sin b, k)
    g0 += -cmulz(tb, v0).x;
    g1 += -cmulz(tb, v1).x;
    g2 += -cmulz(tb, v2).x;
    const double2 bv = make_double2(-(v0.x * n0 + v1.x * n1 + v2.x * n2), -(v0.y * n0 + v1.y * n1 + v2.y * n2));
    const double2 tbv = cmulz(tb, bv);
    c0 += -k * cb * tbv.y;
    c1 += -k * sb * tbv.y;
    c2 += k * tbv.x;
  }
  gn[3 * i] += g0;
  gn[3 * i + 1] += g1;
  gn[3 * i + 2] += g2;
  ga[i] += gav;
  gc[3 * i] += c0;
  gc[3 * i + 1] += c1;
  gc[3 * i + 2] += c2;
}

// w_r[i] = conj(sum_q c[q, r] i rho omega (-n . dof_q) a)   (conjugated for the A^H solve)
__global__ void force_weights_kernel(int64_t n, const double* __restrict__ N, const double* __restrict__ A,
                                     const double* __restrict__ dofs, const int32_t* __restrict__ inf, int n_inf,
                                     int n_rad, const double2* __restrict__ cw, double omega, double rho,
                                     double2* __restrict__ wconj) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int r = blockIdx.y;
  if (i >= n || r >= n_rad) return;
  double2 w = make_double2(0.0, 0.0);
  for (int q = 0; q < n_inf; ++q) {
    const double* dof = dofs + (int64_t)inf[q] * n * 3 + 3 * i;
    const double disp = N[3 * i] * dof[0] + N[3 * i + 1] * dof[1] + N[3 * i + 2] * dof[2];
    const double s = rho * omega * -disp * A[i];  // the force weight is i s
    const double2 c = cw[q + (int64_t)r * n_inf];
    w = zadd(w, make_double2(-c.y * s, c.x * s));
  }
  wconj[i + (int64_t)r * n] = make_double2(w.x, -w.y);
}

__global__ void conj_kernel(int64_t count, double2* __restrict__ x) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < count) x[q].y = -x[q].y;
}

}  // namespace

int64_t static_adjoint_work(int64_t n) { return kGeo * n; }

void launch_static_adjoint(cudaStream_t st, LaunchCounter lc, const AssemblyParams& p, const double* RS,
                           const double* RD, double* gc, double* gn, double* ga, double* gv, double* work) {
  dim3 grid((unsigned)((p.n + kRows - 1) / kRows), (unsigned)((p.n + kCols - 1) / kCols));
  cudaMemsetAsync(work, 0, sizeof(double) * kGeo * p.n, st);
  cudaFuncSetAttribute(static_adjoint_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStaticAdjSmem);
  cudaFuncSetAttribute(static_adjoint_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStaticAdjSmem);
  const GradPtrs gp{gc, gn, ga, gv};
  if (p.direct)
    MH_LAUNCH(lc, st, "adjoint_static", static_adjoint_kernel<true><<<grid, kRows, kStaticAdjSmem, st>>>(p, RS, RD, gp, work));
  else
    MH_LAUNCH(lc, st, "adjoint_static", static_adjoint_kernel<false><<<grid, kRows, kStaticAdjSmem, st>>>(p, RS, RD, gp, work));
  MH_LAUNCH(lc, st, "adjoint_geometry",
            birk_geometry_adjoint_kernel<<<(unsigned)((3 * p.n + 63) / 64), 64, 0, st>>>(p.n, p.V, work, gv));
}

void launch_wave_adjoint(cudaStream_t st, LaunchCounter lc, const AssemblyParams& p, double k, const double2* lS,
                         const double2* rS, const double2* lD, const double2* rD, int nh, double2 c,
                         const double2* egd_values, double* gc, double* gn, double* ga, double* RS, double* RD) {
  WaveWeights w{lS, rS, lD, rD, nh, c};
  dim3 grid((unsigned)((p.n + kRows - 1) / kRows), (unsigned)((p.n + kCols - 1) / kCols));
  const GradPtrs gp{gc, gn, ga, nullptr};
  if (p.gfs & MH_GF_WU) {
    if (p.direct)
      MH_LAUNCH(lc, st, "adjoint_wave", (wave_adjoint_kernel<true, kWaveWu><<<grid, kRows, 0, st>>>(p, k, w, nullptr, gp)));
    else
      MH_LAUNCH(lc, st, "adjoint_wave", (wave_adjoint_kernel<false, kWaveWu><<<grid, kRows, 0, st>>>(p, k, w, nullptr, gp)));
  } else if (p.gfs & MH_GF_EXACT_DELHOMMEAU) {
    if (p.direct)
      MH_LAUNCH(lc, st, "adjoint_wave",
                (wave_adjoint_kernel<true, kWaveExact><<<grid, kRows, 0, st>>>(p, k, w, egd_values, gp)));
    else
      MH_LAUNCH(lc, st, "adjoint_wave",
                (wave_adjoint_kernel<false, kWaveExact><<<grid, kRows, 0, st>>>(p, k, w, egd_values, gp)));
  }
  dim3 g2((unsigned)((p.n + 255) / 256), (unsigned)p.n);
  MH_LAUNCH(lc, st, "adjoint_weights", weights_accumulate_kernel<<<g2, 256, 0, st>>>(p.n, w, RS, RD));
}

int64_t egd_packed_pairs(int64_t n) { return n * (n + 1) / 2; }

void launch_egd_pair_values(cudaStream_t st, LaunchCounter lc, const AssemblyParams& p, double k, double2* out) {
  const int64_t m = egd_packed_pairs(p.n);
  if (m <= 0) return;
  MH_LAUNCH(lc, st, "egd_pair_values",
            egd_pair_values_kernel<<<(unsigned)((m + kEgdThreads - 1) / kEgdThreads), kEgdThreads, 0, st>>>(p, k, m, out));
  MH_LAUNCH(lc, st, "egd_pair_values",
            egd_pair_quadrature_kernel<<<(unsigned)std::min<int64_t>((p.n * p.n + 3) / 4, 16 * 152), kEgdThreads, 0,
                                         st>>>(p, k, out));
}

void launch_egd_dk(cudaStream_t st, LaunchCounter lc, const AssemblyParams& p, double k, const double2* values,
                   double2* dS, double2* dD) {
  dim3 grid((unsigned)((p.n + kRows - 1) / kRows), (unsigned)((p.n + kCols - 1) / kCols));
  if (p.direct)
    MH_LAUNCH(lc, st, "wave_dk", egd_dk_kernel<true><<<grid, kRows, 0, st>>>(p, k, values, dS, dD));
  else
    MH_LAUNCH(lc, st, "wave_dk", egd_dk_kernel<false><<<grid, kRows, 0, st>>>(p, k, values, dS, dD));
}

void launch_outer_adj(cudaStream_t st, LaunchCounter lc, int64_t n, int nh, const double2* U, const double2* V,
                      double alpha, double2* out) {
  dim3 grid((unsigned)((n + 255) / 256), (unsigned)n);
  MH_LAUNCH(lc, st, "outer", outer_adj_kernel<<<grid, 256, 0, st>>>(n, nh, U, V, alpha, out));
}

void launch_rhs_adjoint(cudaStream_t st, LaunchCounter lc, int64_t n, const double* N, const double* A,
                        const double* C, const double* dofs, const int32_t* rad, int n_rad, const int32_t* inf,
                        int n_inf, int n_beta, const double* betas, double omega, double rho, double gacc,
                        const double2* cw, const double2* phi, const double2* t, double* gc, double* gn, double* ga,
                        double* gd) {
  MH_LAUNCH(lc, st, "adjoint_rhs",
            rhs_adjoint_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(n, N, A, C, dofs, rad, n_rad, inf, n_inf,
                                                                             n_beta, betas, omega, rho, gacc, cw, phi,
                                                                             t, gc, gn, ga, gd));
}

void launch_force_weights(cudaStream_t st, LaunchCounter lc, int64_t n, const double* N, const double* A,
                          const double* dofs, const int32_t* inf, int n_inf, int n_rad, const double2* cw,
                          double omega, double rho, double2* wconj) {
  dim3 grid((unsigned)((n + 127) / 128), (unsigned)n_rad);
  MH_LAUNCH(lc, st, "adjoint_force_weights",
            force_weights_kernel<<<grid, 128, 0, st>>>(n, N, A, dofs, inf, n_inf, n_rad, cw, omega, rho, wconj));
}

void launch_wave_dk(cudaStream_t st, LaunchCounter lc, const AssemblyParams& p, const double* k_dev, double2* dS,
                    double2* dD) {
  const int64_t rt = (p.n + kRows - 1) / kRows;
  const int cols = columns_per_cta(rt * p.n / 2);
  dim3 grid((unsigned)rt, (unsigned)((p.n + cols - 1) / cols));
  if (p.direct)
    MH_LAUNCH(lc, st, "wave_dk", wave_dk_kernel<true><<<grid, kRows, 0, st>>>(p, k_dev, dS, dD, cols));
  else
    MH_LAUNCH(lc, st, "wave_dk", wave_dk_kernel<false><<<grid, kRows, 0, st>>>(p, k_dev, dS, dD, cols));
}

void launch_conj(cudaStream_t st, LaunchCounter lc, int64_t count, double2* x) {
  if (count <= 0) return;
  MH_LAUNCH(lc, st, "conj", conj_kernel<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(count, x));
}

}  // namespace mh
