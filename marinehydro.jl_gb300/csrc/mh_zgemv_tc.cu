// mh_zgemv_tc.cu -- Y = A X (or R = B - A X) for a batch of dense complex FP64 matrices and up
// to 8 right-hand sides, FP64-accurate, on the BF16 tensor cores (Ozaki splitting).
//
// With 7 right-hand sides a complex matrix-vector product does 28 FP64 FMAs per 16 bytes of
// A, so on GB300 it is bound by the FP64 pipe, not by HBM (S B of the frequency sweep: 0.9
// TFLOP/s, 7.4 ms for 30 matrices of 2000 panels).  Here A is cut, 32 columns at a time,
// into eight balanced base-128 digits per entry (a 55-bit fixed point per row and block,
// exact in BF16), X likewise per column and block, and the digit products accumulate
// exactly in FP32 tensor memory, as in the LU's tensor-core update (mh_ozaki.cu).  Each
// block's exact partial sums are converted to FP64 once and added up over the blocks in
// FP64, so the result carries FP64 rounding (it feeds the FP64 residuals of the
// iterative refinement, which must be FP64-accurate).
//
//   zgemv_xsplit_kernel: X (n x g, g <= 8) -> per 32-row block one 128 x 32 BF16 operand
//     tile: row 16 q + 8 part + j is digit q of part (re/im) of column j, so digits q .. 7
//     stack along N; and one exponent per column and block.
//   zgemv_tc_kernel: one CTA (512 threads) per 128-row tile of one matrix and split of its
//     columns, looping over the split's 32-column blocks in halves of 16: four threads per row
//     hold the FP64 block in registers, cut a half into 16 digit planes in shared memory
//     (integer arithmetic on the FP64 bit fields, no FP64 instructions) and load that half of
//     the next block; one thread issues 16 tcgen05.mma (A digit p of Re A and Im A against the
//     stacked X digits 0 .. 7-p, N = 16 (8-p)) into one of two 256-column TMEM buffers, which run
//     under the cutting of the next half; the previous block's accumulators are combined in
//     integers, with one FP64 addition per real output.
//   zgemv_reduce_kernel: the splits' sums, in order.
// Bound: the integer pipe that cuts the digits (45 instructions per value) and the epilogue; the
// products run under the cutting of the next half.  Four matrices of order 8000 with four
// right-hand sides 4.03 -> 2.45 ms (8.1 us per block with the cutting and the products in turn; splits
// and the shorter cutting alone 3.19), four of 1400 365 -> 92 us and
// twelve of 430 122 -> 37 us (44 and 48 CTAs became 132 and 144), five of 640 167 -> 20 us.
// Every wait is bounded; on timeout the kernel raises the caller's flag, drains (bounded)
// and frees its tensor memory.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "mh_digits.cuh"
#include "mh_internal.cuh"
#include "mh_tc.cuh"

namespace mh {

namespace {

constexpr int kZvRows = 128;                 // rows per CTA (MMA M)
constexpr int kZvK = 32;                     // columns of A per block
constexpr int kZvDigits = 8;
constexpr int kZvRhs = 8;                    // right-hand sides per launch
constexpr int kZvHalf = kZvK / 2;             // columns of a half block (MMA K)
constexpr int kZvPlane = kZvRows * kZvHalf * 2;  // one 128 x 16 BF16 digit plane (4 KB)
constexpr int kZvADig = 2 * kZvDigits * kZvPlane;  // 16 planes of a half block (64 KB), two of them
constexpr int kZvXTile = 128 * kZvK * 2;     // X operand tile: 128 N-rows x 32 K (8 KB)
constexpr int kZvThreads = 512;
constexpr uint32_t kZvTmemCols = 512;        // 2 buffers x (Re A: 128, Im A: 128)
constexpr uint32_t kZvWaitPolls = 1u << 26;
constexpr size_t kZvSmem = 2 * (size_t)kZvADig + 2 * kZvXTile;
constexpr int kZvMaxSplit = 32;
constexpr int kZvMaxCtas = 6 * 152;          // with more than one split: bounds the partial sums

// BF16 bits of a small integer (|d| <= 64): through the FP32 magic number, exact
__device__ __forceinline__ uint32_t bf16_of_small(int d) {
  const float f = __int_as_float(0x4B400000 + d) - 12582912.0f;
  return __float_as_uint(f) >> 16;
}

__device__ __forceinline__ void digits_of(long long X, int (&d8)[kZvDigits]) {
#pragma unroll
  for (int p = kZvDigits - 1; p > 0; --p) {
    const long long t = ((X + 64) & 127) - 64;
    d8[p] = (int)t;
    X = (X - t) >> 7;
  }
  d8[0] = (int)X;
}

__device__ __forceinline__ int scale_exp(double maxabs) {
  if (!(maxabs > 0.0)) return 0;
  int e;
  frexp(maxabs, &e);
  return e;
}

// X columns r0 .. r0+g-1 of matrix b -> per block the operand tile and the column exponents
__global__ void __launch_bounds__(256) zgemv_xsplit_kernel(BatchDesc d, const double2* __restrict__ Xall,
                                                           int64_t xstride, int r0, int g, int64_t nkb,
                                                           unsigned char* __restrict__ xt, int* __restrict__ xexp) {
  const int64_t kb = blockIdx.x, b = blockIdx.y, n = d.n;
  const int j = threadIdx.x >> 5, kk = threadIdx.x & 31;  // warp j: column j, lane: row of the block
  const int64_t row = kb * kZvK + kk;
  // K position: a thread of the product kernel cuts columns 8 s .. 8 s + 3 into the first half
  // block and 8 s + 4 .. 8 s + 7 into the second
  const int pos = ((kk >> 2) & 1) * kZvHalf + (kk >> 3) * 4 + (kk & 3);
  double2 v = make_double2(0.0, 0.0);
  if (j < g && row < n) v = Xall[b * xstride + row + (int64_t)(r0 + j) * n];
  double mx = fmax(fabs(v.x), fabs(v.y));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const int f = scale_exp(mx);
  if (kk == 0) xexp[(b * nkb + kb) * kZvRhs + j] = f;
  unsigned char* tile = xt + (b * nkb + kb) * (int64_t)kZvXTile;
  int dre[kZvDigits], dim[kZvDigits];
  digits_of(llrint(ldexp(v.x, 55 - f)), dre);
  digits_of(llrint(ldexp(v.y, 55 - f)), dim);
#pragma unroll
  for (int q = 0; q < kZvDigits; ++q) {
    const uint32_t o_re = tc::kmajor_offset(16 * q + j, pos, kZvK), o_im = tc::kmajor_offset(16 * q + 8 + j, pos, kZvK);
    *reinterpret_cast<uint16_t*>(tile + o_re) = (uint16_t)bf16_of_small(dre[q]);
    *reinterpret_cast<uint16_t*>(tile + o_im) = (uint16_t)bf16_of_small(dim[q]);
  }
}

// two consecutive FP32 TMEM columns of this thread's lane, no wait
__device__ __forceinline__ void tmem_ld2_nowait(uint32_t taddr, uint32_t& a, uint32_t& b) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ int int_of_exact(uint32_t fbits) {
  return __float_as_int(__uint_as_float(fbits) + 12582912.0f) - 0x4B400000;
}

// v 2^e, rounded to 53 bits half away from zero, on the integer pipe (FP64 only where the result
// leaves the normal range)
__device__ __forceinline__ double scaled(long long v, int e) {
  const unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
  if (a == 0) return 0.0;
  const int lz = __clzll((long long)a);
  const int be = e + 63 - lz + 1023;  // biased exponent before rounding
  if (be < 1 || be > 2045) return ldexp((double)v, e);
  const unsigned long long m = a << lz;
  const unsigned long long mant = (m >> 11) + ((m >> 10) & 1ull);  // a carry moves on into the exponent
  return __longlong_as_double((long long)((((unsigned long long)(be - 1) << 52) + mant) | (v < 0 ? 1ull << 63 : 0ull)));
}

__global__ void zgemv_reduce_kernel(int64_t n, int g, int64_t batch, int nsplit, const double2* __restrict__ part,
                                    double2* __restrict__ Yall, int64_t xstride, int r0,
                                    const double2* __restrict__ Ball) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, per = g * n;
  if (q >= per * batch) return;
  const int64_t b = q / per, o = b * xstride + r0 * n + (q - b * per);
  double2 s = part[q];
#pragma unroll 4
  for (int js = 1; js < nsplit; ++js) {
    const double2 v = part[js * per * batch + q];
    s.x += v.x;
    s.y += v.y;
  }
  if (Ball) { const double2 bb = Ball[o]; s = make_double2(bb.x - s.x, bb.y - s.y); }
  Yall[o] = s;
}

// Splits of the columns: one CTA per 128-row tile leaves SMs idle (44 CTAs for four matrices of
// 1400) or a nearly empty last wave (252 for four of 8000), so the splits that minimise waves x
// blocks per CTA, with two blocks' time for a CTA's start and one for the sums.
int zgemv_split(int64_t n, int64_t batch) {
  const int64_t nkb = (n + kZvK - 1) / kZvK, tiles = (n + kZvRows - 1) / kZvRows * batch;
  int best = 1;
  int64_t best_t = 0;
  for (int q = 1; q <= kZvMaxSplit && q <= nkb && (q == 1 || q * tiles <= kZvMaxCtas); ++q) {
    const int64_t t = (tiles * q + 151) / 152 * ((nkb + q - 1) / q + 2) + (q > 1 ? 1 : 0);
    if (q == 1 || t < best_t) {
      best = q;
      best_t = t;
    }
  }
  return best;
}

__global__ void __launch_bounds__(kZvThreads, 1) zgemv_tc_kernel(BatchDesc d, const double2* __restrict__ Aall,
                                                            const double2* __restrict__ Ball,
                                                            double2* __restrict__ Yall, int64_t xstride, int r0,
                                                            int g, int64_t nkb,
                                                            const unsigned char* __restrict__ xt,
                                                            const int* __restrict__ xexp, int subtract,
                                                            double2* __restrict__ part,
                                                            int* __restrict__ timeout_flag) {
  extern __shared__ __align__(1024) unsigned char zsm[];
  __shared__ __align__(8) uint64_t mbar_load, mbar_mma[2];
  __shared__ uint32_t tmem_base;
  unsigned char* sAd = zsm;                       // [half][part][digit] planes
  unsigned char* sX[2] = {sAd + 2 * kZvADig, sAd + 2 * kZvADig + kZvXTile};
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n = d.n, b = blockIdx.y;
  const int64_t row0 = blockIdx.x * (int64_t)kZvRows;
  const int rows_valid = (int)((n - row0) < kZvRows ? (n - row0) : kZvRows);
  const double2* A = Aall + b * d.stride;
  if (tid == 0) {
    tc::mbar_init(&mbar_load, 1);
    tc::mbar_init(&mbar_mma[0], 1);
    tc::mbar_init(&mbar_mma[1], 1);
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base, kZvTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  // this CTA's blocks [kb0, kb1): split blockIdx.z of gridDim.z
  const int64_t kb0 = nkb * blockIdx.z / gridDim.z, kb1 = nkb * (blockIdx.z + 1) / gridDim.z;
  // the X operand tile of block kb0 + it
  auto load_x = [&](int it) {
    tc::mbar_arrive_expect_tx(&mbar_load, kZvXTile);
    tc::bulk_g2s(sX[it & 1], xt + (b * nkb + kb0 + it) * (int64_t)kZvXTile, kZvXTile, &mbar_load);
  };
  if (tid == 0) load_x(0);

  // split mapping: four threads per row, eight columns each (rows past n and columns past n are
  // zero); a half's values are loaded as soon as the half before them is cut
  const int srow = tid >> 2, sq = tid & 3;
  double2 vals[2][4];
  auto load_a = [&](int64_t kb, int h) {
    const int64_t c0 = kb * kZvK + 8 * sq + 4 * h;
    const double2* a = A + row0 + srow + c0 * n;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      vals[h][c] = (srow < rows_valid && c0 + c < n) ? __ldg(a + c * n) : make_double2(0.0, 0.0);
  };
  load_a(kb0, 0);
  load_a(kb0, 1);
  // epilogue mapping: TMEM lane = row (warp % 4 picks the lane quadrant), warp / 4 picks
  // the two right-hand sides j0, j0 + 1 of this thread
  const int erow = (warp & 3) * 32 + lane, j0 = 2 * (warp >> 2);
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
  double2 acc[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  __shared__ int s_rowexp[2][kZvRows];
  bool failed = false;
  int loads_pending = 1, mma_pending = 0;  // mma_pending: halves whose products nobody has waited for

  auto epilogue = [&](int it) {
    if (j0 >= g) return;  // no right-hand side here
    const uint32_t base = tmem + lane_off + (uint32_t)(it & 1) * 256u;
    // (Re A | Im A) x (Xr | Xi) for digit sums d = 0..7 and this thread's two columns
    uint32_t v[kZvDigits][8];
#pragma unroll
    for (int dd = 0; dd < kZvDigits; ++dd) {
      const uint32_t c = base + (uint32_t)(16 * dd + j0);
      tmem_ld2_nowait(c, v[dd][0], v[dd][1]);               // Re A Xr (j0, j0+1)
      tmem_ld2_nowait(c + 8u, v[dd][2], v[dd][3]);          // Re A Xi
      tmem_ld2_nowait(c + 128u, v[dd][4], v[dd][5]);        // Im A Xr
      tmem_ld2_nowait(c + 136u, v[dd][6], v[dd][7]);        // Im A Xi
    }
    tmem_wait_ld();
    const int er = s_rowexp[it & 1][erow];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int pr[4], pi[4];
#pragma unroll
      for (int dd = 0; dd < kZvDigits; ++dd) {
        // T_d of the complex product: Re = ReA Xr - ImA Xi, Im = ReA Xi + ImA Xr (|.| < 2^22)
        const int tr = int_of_exact(v[dd][0 + h]) - int_of_exact(v[dd][6 + h]);
        const int ti = int_of_exact(v[dd][2 + h]) + int_of_exact(v[dd][4 + h]);
        if (dd & 1) { pr[dd >> 1] = pr[dd >> 1] * 128 + tr; pi[dd >> 1] = pi[dd >> 1] * 128 + ti; }
        else { pr[dd >> 1] = tr; pi[dd >> 1] = ti; }
      }
      // sum_d T_d 128^-d = (hr + lr 2^-28) 2^-21, |hr| < 2^40, |lr| < 2^43
      const long long hr = (long long)pr[0] * 16384 + pr[1], lr = (long long)pr[2] * 16384 + pr[3];
      const long long hi = (long long)pi[0] * 16384 + pi[1], li = (long long)pi[2] * 16384 + pi[3];
      const int e = er + __ldg(xexp + (b * nkb + kb0 + it) * kZvRhs + j0 + h) - 33 - 22;
      acc[h].x += scaled(hr * 4194304 + (lr >> 6), e);
      acc[h].y += scaled(hi * 4194304 + (li >> 6), e);
    }
  };

  // cuts half h of the block in registers into its digit planes
  auto cut = [&](int h, int emax) {
    uint32_t pk[2][kZvDigits][2];  // [part][digit][pairs of columns]
    dg::split4(vals[h], emax, pk);
    unsigned char* dst = sAd + h * kZvADig + tc::kmajor_offset(srow, 4 * sq, kZvHalf);
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int p = 0; p < kZvDigits; ++p)
        *reinterpret_cast<uint2*>(dst + (q * kZvDigits + p) * kZvPlane) = make_uint2(pk[q][p][0], pk[q][p][1]);
  };
  auto issue = [&](int it, int h) {
    tc::fence_after_sync();
    const uint32_t a0 = tc::smem_u32(sAd + h * kZvADig);
    const uint64_t x = tc::smem_desc(tc::smem_u32(sX[it & 1]) + (uint32_t)h * 256, 128, (kZvK / 8) * 128);
    const uint32_t tb = tmem + (uint32_t)(it & 1) * 256u;
#pragma unroll 1
    for (int p = 0; p < kZvDigits; ++p) {
      const uint32_t id = tc::idesc_bf16_f32(kZvRows, 16 * (kZvDigits - p));
#pragma unroll
      for (int q = 0; q < 2; ++q)
        tc::mma_bf16(tb + (uint32_t)(128 * q + 16 * p),
                     tc::smem_desc(a0 + (uint32_t)(q * kZvDigits + p) * kZvPlane, 128, (kZvHalf / 8) * 128), x, id,
                     (p == 0 && h == 0) ? 0u : 1u);
    }
    tc::mma_commit(&mbar_mma[h]);
  };
  const int nit = (int)(kb1 - kb0);
  for (int it = 0; it < nit; ++it) {
    int emax = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      emax = max(emax, max(dg::biased_exp(vals[c >> 2][c & 3].x), dg::biased_exp(vals[c >> 2][c & 3].y)));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 1));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 2));
    bool ok = tc::mbar_wait(&mbar_load, (uint32_t)(it & 1), kZvWaitPolls);
    // the planes of this half are free once the products of the block before are done
    if (it > 0) ok = tc::mbar_wait(&mbar_mma[0], (uint32_t)((it - 1) & 1), kZvWaitPolls) && ok;
    cut(0, emax);
    if (it + 1 < nit) load_a(kb0 + it + 1, 0);
    tc::fence_proxy_async_smem();
    if (__syncthreads_or(!ok)) { failed = true; break; }
    --loads_pending;
    if (it > 0) --mma_pending;
    if (tid == 0) issue(it, 0);
    // |v| < 2^E with E = emax - 1022 (the exponent scale of this row and block); every warp is past
    // the epilogue that read this buffer
    if (sq == 0) s_rowexp[it & 1][srow] = dg::scale_of(emax);
    ++mma_pending;
    if (it > 0) ok = tc::mbar_wait(&mbar_mma[1], (uint32_t)((it - 1) & 1), kZvWaitPolls);
    cut(1, emax);
    if (it + 1 < nit) load_a(kb0 + it + 1, 1);
    tc::fence_proxy_async_smem();
    if (__syncthreads_or(!ok)) { failed = true; break; }
    if (it > 0) --mma_pending;
    if (tid == 0) {
      issue(it, 1);
      if (it + 1 < nit) load_x(it + 1);  // the other X buffer is free
    }
    ++mma_pending;
    if (it + 1 < nit) ++loads_pending;
    tc::fence_after_sync();
    if (it > 0) epilogue(it - 1);
    tc::fence_before_sync();
  }
  if (!failed) {
    const int it = nit - 1;
    bool ok = tc::mbar_wait(&mbar_mma[0], (uint32_t)(it & 1), kZvWaitPolls);
    ok = tc::mbar_wait(&mbar_mma[1], (uint32_t)(it & 1), kZvWaitPolls) && ok;
    if (__syncthreads_or(!ok)) failed = true;
    else {
      mma_pending = 0;
      tc::fence_after_sync();
      epilogue(it);
    }
  }
  if (failed) {
    // whatever is in flight ends before the shared and the tensor memory are released (a wait for
    // the phase that is already over returns at once)
    if (tid == 0) atomicExch(timeout_flag, 1);
    if (mma_pending > 0)
      for (int h = 0; h < 2; ++h) {
        tc::mbar_wait(&mbar_mma[h], 0, kZvWaitPolls);
        tc::mbar_wait(&mbar_mma[h], 1, kZvWaitPolls);
      }
    if (loads_pending > 0) {
      tc::mbar_wait(&mbar_load, 0, kZvWaitPolls);
      tc::mbar_wait(&mbar_load, 1, kZvWaitPolls);
    }
  } else {
    const int64_t i = row0 + erow;
    if (erow < rows_valid) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = j0 + h;
        if (j >= g) continue;
        const int64_t o = b * xstride + i + (int64_t)(r0 + j) * n;
        double2 y = acc[h];
        if (part) {  // summed and subtracted by zgemv_reduce_kernel
          part[((blockIdx.z * (int64_t)gridDim.y + b) * g + j) * n + i] = y;
          continue;
        }
        if (subtract) { const double2 bb = Ball[o]; y = make_double2(bb.x - y.x, bb.y - y.y); }
        Yall[o] = y;
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kZvTmemCols);
}

}  // namespace

size_t tc_zgemv_workspace_bytes(int64_t n, int64_t batch) {
  const int64_t nkb = (n + kZvK - 1) / kZvK;
  // splits x matrices of this many matrices or fewer
  const int64_t sums = std::max<int64_t>(batch, kZvMaxCtas / ((n + kZvRows - 1) / kZvRows));
  const size_t partial = (size_t)std::min<int64_t>(sums, kZvMaxSplit * batch) * kZvRhs * (size_t)n * sizeof(double2);
  return (size_t)batch * (size_t)nkb * ((size_t)kZvXTile + kZvRhs * sizeof(int)) + 256 + partial;
}

void tc_zgemv(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
              int64_t nrhs, int64_t xstride, double2* Y, const double2* B, void* ws, int* timeout_flag) {
  const int64_t n = d.n;
  if (n <= 0 || nrhs <= 0 || d.batch <= 0) return;
  const int64_t nkb = (n + kZvK - 1) / kZvK;
  unsigned char* xt = static_cast<unsigned char*>(ws);
  int* xexp = reinterpret_cast<int*>(xt + d.batch * nkb * (int64_t)kZvXTile);
  const int ns = zgemv_split(n, d.batch);
  // the partial sums behind the exponents, on a 256-byte boundary as the tiles' start
  const size_t head = ((size_t)d.batch * (size_t)nkb * (kZvXTile + kZvRhs * sizeof(int)) + 255) / 256 * 256;
  double2* part = ns > 1 ? reinterpret_cast<double2*>(xt + head) : nullptr;
  cudaFuncSetAttribute(zgemv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZvSmem);
  for (int64_t r0 = 0; r0 < nrhs; r0 += kZvRhs) {
    const int g = (int)((nrhs - r0) < kZvRhs ? (nrhs - r0) : kZvRhs);
    MH_LAUNCH(lc, st, "zgemv_tc_split",
              zgemv_xsplit_kernel<<<dim3((unsigned)nkb, (unsigned)d.batch), 256, 0, st>>>(d, X, xstride, (int)r0, g,
                                                                                           nkb, xt, xexp));
    const dim3 grid((unsigned)((n + kZvRows - 1) / kZvRows), (unsigned)d.batch, (unsigned)ns);
    MH_LAUNCH(lc, st, "zgemv_tc",
              zgemv_tc_kernel<<<grid, kZvThreads, kZvSmem, st>>>(d, A, B, Y, xstride, (int)r0, g, nkb, xt, xexp,
                                                                 B != nullptr ? 1 : 0, part, timeout_flag));
    if (part) {
      const int64_t tot = g * n * d.batch;
      MH_LAUNCH(lc, st, "zgemv_tc_sum",
                zgemv_reduce_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(n, g, d.batch, ns, part, Y, xstride,
                                                                                  (int)r0, B));
    }
  }
}

}  // namespace mh
