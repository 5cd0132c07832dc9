// mh_digits.cuh -- exact digit splitting of FP64 values for the tensor-core FP64 products
// (mh_ozaki.cu, mh_zgemv_tc.cu), in integer arithmetic on the FP64 bit fields.
//
// A row (or column) of values with largest biased exponent emax (|v| < 2^E, E = emax - 1022)
// is scaled to a 55-bit fixed point X = round(v 2^(55 - E)) and cut into eight balanced
// base-128 digits d_0 .. d_7 in [-64, 64], X = sum_p d_p 128^(7 - p) (the GEMV), or seven
// balanced base-256 digits in [-128, 128] (the LU update); each digit is exact in BF16.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mh {
namespace dg {

constexpr int kDigits = 8;

// biased exponent field of v (0 for zero and subnormals)
__device__ __forceinline__ int biased_exp(double v) {
  return (int)((__double_as_longlong(v) >> 52) & 0x7FF);
}

// the scale exponent E of a row or column from its largest biased exponent
__device__ __forceinline__ int scale_of(int emax_biased) { return emax_biased > 0 ? emax_biased - 1022 : 0; }

// round(v 2^(55 - E)), rounding half away from zero; zero and subnormal entries give 0
__device__ __forceinline__ long long fixed55(double v, int emax_biased) {
  const long long bits = __double_as_longlong(v);
  const int ev = (int)((bits >> 52) & 0x7FF);
  const unsigned long long m4 = ev == 0 ? 0ull : ((unsigned long long)(bits & 0xFFFFFFFFFFFFFLL) | 0x10000000000000ull) << 2;
  int s = emax_biased - ev;  // >= 0: m4 is the value at s = 0; from 56 on it rounds to 0
  s = s < 63 ? s : 63;
  const long long X = (long long)((m4 + ((1ull << s) >> 1)) >> s);
  return bits < 0 ? -X : X;
}

// two BF16 values of small integers (|d| <= 128, eight significant bits) in one 32-bit word, the first in the low half
__device__ __forceinline__ uint32_t bf16x2(int d0, int d1) {
  const float f0 = __int_as_float(0x4B400000 + d0) - 12582912.0f;
  const float f1 = __int_as_float(0x4B400000 + d1) - 12582912.0f;
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// Four consecutive K values (half a 16-byte row chunk of the canonical K-major layout) of one
// row: their 16 digit planes (re/im x 8 digits) as packed BF16 pairs, pk[part][digit][0..1].
// With 64 added to every digit beforehand (one 64-bit addition, which does all the carries) digit p
// is a bit field u_p = d_p + 64 in [0, 128] of the sum; two of them set into the mantissas of BF16
// 128.0 and 192 subtracted from both in one packed operation are the digits: 45 instructions
// per value, where digits peeled off one by one and converted through FP32 took about 100.
__device__ __forceinline__ uint32_t digit_pair(uint32_t u0, uint32_t u1, uint32_t mask) {
  const uint32_t t = (__byte_perm(u0, u1, 0x5410) & mask) | 0x43004300u;
  uint32_t r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(t), "r"(0x43404340u));
  return r;
}
__device__ __forceinline__ void split4(const double2 (&v)[4], int emax, uint32_t (&pk)[2][kDigits][2]) {
  constexpr long long kBias = 0x81020408102040ll;  // 64 in each of the eight base-128 digits
#pragma unroll
  for (int c = 0; c < 4; c += 2) {
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const unsigned long long x0 = (unsigned long long)(fixed55(part ? v[c].y : v[c].x, emax) + kBias);
      const unsigned long long x1 = (unsigned long long)(fixed55(part ? v[c + 1].y : v[c + 1].x, emax) + kBias);
#pragma unroll
      for (int p = 0; p < kDigits; ++p)
        pk[part][p][c >> 1] = digit_pair((uint32_t)(x0 >> (7 * (7 - p))), (uint32_t)(x1 >> (7 * (7 - p))),
                                         p == 0 ? 0x00FF00FFu : 0x007F007Fu);
    }
  }
}

// Seven balanced base-256 digits in [-128, 128] of the same X (|X| < 2^55), most significant
// first: X = sum_p d_p 256^(6 - p).  With 128 added to every digit beforehand (one 64-bit addition,
// which does all the carries, for X up to 2^55 into the 57th bit) they are the sum's bytes, the top one
// with what is above it.  Each is exact in BF16 (eight significant bits).
constexpr int kDigits7 = 7;
__device__ __forceinline__ void digits7(long long X, int (&d)[kDigits7]) {
  const unsigned long long u = (unsigned long long)(X + 0x80808080808080ll);
  const unsigned int lo = (unsigned int)u, hi = (unsigned int)(u >> 32);
  d[6] = (int)(lo & 255u) - 128;
  d[5] = (int)((lo >> 8) & 255u) - 128;
  d[4] = (int)((lo >> 16) & 255u) - 128;
  d[3] = (int)(lo >> 24) - 128;
  d[2] = (int)(hi & 255u) - 128;
  d[1] = (int)((hi >> 8) & 255u) - 128;
  d[0] = (int)(hi >> 16) - 128;
}

// Eight consecutive K values (one 16-byte row chunk) of one row: their seven base-256 digit planes
__device__ __forceinline__ void split7(const double2 (&v)[8], int emax, uint32_t (&pk)[2][kDigits7][4]) {
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    int a0[kDigits7], a1[kDigits7], b0[kDigits7], b1[kDigits7];
    digits7(fixed55(v[c].x, emax), a0);
    digits7(fixed55(v[c + 1].x, emax), a1);
    digits7(fixed55(v[c].y, emax), b0);
    digits7(fixed55(v[c + 1].y, emax), b1);
#pragma unroll
    for (int p = 0; p < kDigits7; ++p) {
      pk[0][p][c >> 1] = bf16x2(a0[p], a1[p]);
      pk[1][p][c >> 1] = bf16x2(b0[p], b1[p]);
    }
  }
}

}  // namespace dg
}  // namespace mh
