// mh_lu.cu -- batched dense complex LU with partial pivoting and multi-RHS solves.
//
// Replaces linsolve / _linearsolve / gpu_linsolve (matrix_assembly.jl:396-434),
// whose CPU path is LinearSolve LUFactorization -> LAPACK zgetrf/zgetrs and whose
// CUDA path is cuSOLVER through `\` on a CuArray.  Same semantics as zgetrf:
// right-looking blocked LU, pivot = first row of maximal |re|+|im| (izamax), rows
// swapped across the whole matrix, info = index of the first exactly-zero pivot.
//
// Work split per panel step k (nb = 32 columns):
//   panel_cluster_kernel  a thread-block cluster of P CTAs per matrix: the panel's
//                  rows are split over the P CTAs and held in shared memory; pivot
//                  candidates and their rows are pushed through distributed shared
//                  memory with one cluster barrier per column, so the panel's FP64
//                  rank-1 updates run on P SMs instead of one
//   panel_kernel   the same on one CTA straight from global memory, for panels too
//                  tall for the cluster's shared memory
//   laswp_kernel   the panel's row interchanges applied to every column outside it,
//                  as one permutation of at most 64 rows (a warp per column)
//   trsm_lanes_kernel, trsm_kernel   U12 = L11^-1 A12 with L11 in shared memory: 8 or 32 lanes
//                  per column in FP64, one thread per column in FP32
//   gemm3m_kernel  A22 -= L21 U12 on the CUDA cores (FP64); the tensor cores' updates are in
//                  mh_ozaki.cu (FP64) and mh_bf16x3.cu (FP32, always)
// Templated on the real type: double (the plain FP64 path) and float (the factor
// used by mixed-precision iterative refinement).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <initializer_list>
#include <type_traits>

#include "mh_fixpoint.cuh"
#include "mh_internal.cuh"
#include "mh_per_device.h"

namespace mh {

namespace {

constexpr int kNB = 32;

template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r;
}
template <typename C> __device__ __forceinline__ C cconj(C a) { C r; r.x = a.x; r.y = -a.y; return r; }
// c - a*b with fused multiply-adds
template <typename C> __device__ __forceinline__ C cfms(C c, C a, C b) {
  C r;
  r.x = fma(-a.x, b.x, c.x); r.x = fma(a.y, b.y, r.x);
  r.y = fma(-a.x, b.y, c.y); r.y = fma(-a.y, b.x, r.y);
  return r;
}
// c + a*b
template <typename C> __device__ __forceinline__ C cfma(C c, C a, C b) {
  C r;
  r.x = fma(a.x, b.x, c.x); r.x = fma(-a.y, b.y, r.x);
  r.y = fma(a.x, b.y, c.y); r.y = fma(a.y, b.x, r.y);
  return r;
}
template <typename C> __device__ __forceinline__ C crecip(C a) {
  // 1 / a (Smith)
  C r;
  if (fabs(a.x) >= fabs(a.y)) {
    auto q = a.y / a.x; auto den = a.x + a.y * q;
    r.x = 1 / den; r.y = -q / den;
  } else {
    auto q = a.x / a.y; auto den = a.y + a.x * q;
    r.x = q / den; r.y = -1 / den;
  }
  return r;
}
// FP64: 1/a = conj(a) f / |a f|^2 with a scaled by a power of two f (so |a f| is near 1), the
// reciprocal of the squared magnitude on the integer pipe (fx::recip): seven FP64 operations
// instead of Smith's three divisions -- this is the pivot reciprocal on the panel's
// per-column critical path, computed by one lane while the CTA waits.  Within a few ulps.
template <> __device__ __forceinline__ double2 crecip<double2>(double2 a) {
  const int ex = (int)((__double_as_longlong(a.x) >> 52) & 0x7FF);
  const int ey = (int)((__double_as_longlong(a.y) >> 52) & 0x7FF);
  const int e = ex > ey ? ex : ey;  // biased exponent of the larger part (a != 0)
  const double f = __longlong_as_double((long long)(2046 - e) << 52);  // 2^(1023 - (e - 1023)), exact
  const double sx = a.x * f, sy = a.y * f;
  const double rf = fx::recip(fma(sx, sx, sy * sy)) * f;
  return make_double2(sx * rf, -sy * rf);
}
// FP32: the same scaling with one division
template <> __device__ __forceinline__ float2 crecip<float2>(float2 a) {
  const int ex = (__float_as_int(a.x) >> 23) & 0xFF, ey = (__float_as_int(a.y) >> 23) & 0xFF;
  const int e = ex > ey ? ex : ey;
  const float f = __int_as_float((254 - e) << 23);
  const float sx = a.x * f, sy = a.y * f;
  const float rf = __fdividef(1.0f, fmaf(sx, sx, sy * sy)) * f;
  return make_float2(sx * rf, -sy * rf);
}
template <typename C> __device__ __forceinline__ C czero() { C r; r.x = 0; r.y = 0; return r; }

__device__ __forceinline__ double2 shfl_c(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ float2 shfl_c(float2 v, int src) {
  return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// ------------------------------- panel ---------------------------------------
template <typename T>
__global__ void __launch_bounds__(512) panel_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                    int32_t* __restrict__ ipiv_all, int32_t* __restrict__ info_all,
                                                    int64_t k) {
  using C = typename cplx_t<T>::type;
  __shared__ T wv[16];
  __shared__ int wi[16];
  __shared__ int s_piv;
  __shared__ T s_best;
  const int64_t n = d.order(blockIdx.x);
  if (k >= n) return;  // a grouped batch: this matrix is factored
  C* A = Aall + d.offset(blockIdx.x);
  int32_t* ipiv = ipiv_all + blockIdx.x * ipiv_stride(d.n);
  const int64_t kend = (k + kNB < n) ? k + kNB : n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  for (int64_t j = k; j < kend; ++j) {
    T best = -1;
    int bi = (int)n;
    for (int64_t i = j + tid; i < n; i += blockDim.x) {
      C a = A[i + j * n];
      T v = fabs(a.x) + fabs(a.y);
      if (v > best) { best = v; bi = (int)i; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      T ob = __shfl_down_sync(0xffffffffu, best, off);
      int oi = __shfl_down_sync(0xffffffffu, bi, off);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { wv[warp] = best; wi[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
      best = lane < nwarp ? wv[lane] : (T)-1;
      bi = lane < nwarp ? wi[lane] : (int)n;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        T ob = __shfl_down_sync(0xffffffffu, best, off);
        int oi = __shfl_down_sync(0xffffffffu, bi, off);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (lane == 0) { s_piv = bi; s_best = best; }
    }
    __syncthreads();
    const int64_t p = s_piv;
    if (tid == 0) ipiv[j] = (int32_t)p;
    if (!(s_best > 0)) {
      // exactly zero column: zgetf2 records info and moves on
      if (tid == 0 && info_all[blockIdx.x] == 0) info_all[blockIdx.x] = (int32_t)(j + 1);
      if (tid == 0) ipiv[j] = (int32_t)j;
      __syncthreads();
      continue;
    }
    if (p != j) {  // inside the panel; laswp_kernel moves the rest of the rows
      for (int64_t c = k + tid; c < kend; c += blockDim.x) {
        C t = A[j + c * n];
        A[j + c * n] = A[p + c * n];
        A[p + c * n] = t;
      }
    }
    __syncthreads();
    const C inv = crecip(A[j + j * n]);
    for (int64_t i = j + 1 + tid; i < n; i += blockDim.x) A[i + j * n] = cmul(A[i + j * n], inv);
    __syncthreads();
    const int64_t m = n - j - 1, w = kend - j - 1;
    if (w > 0) {
      for (int64_t idx = tid; idx < m * w; idx += blockDim.x) {
        int64_t r = idx % m, c = idx / m;
        int64_t i = j + 1 + r, cc = j + 1 + c;
        A[i + cc * n] = cfms(A[i + cc * n], A[i + j * n], A[j + cc * n]);
      }
    }
    __syncthreads();
  }
}

// ---------------------------- panel on a cluster -------------------------------
constexpr int kPanelThreads = 512;
constexpr int kPanelMaxCtas = 16;  // largest cluster (above 8 CTAs it is a non-portable size)
// panel rows one CTA of a cluster of P holds in shared memory: 32 complex columns each, and the
// candidate rows of two columns and P CTAs, below 227 KB
template <typename T> __host__ __device__ constexpr int panel_rows(int P) {
  return sizeof(T) == 8 ? (P <= 8 ? 430 : 414) : 800;
}
// rows per CTA of a panel of m rows on P CTAs: a multiple of 32 where `cap` allows
__host__ __device__ inline int panel_chunk(int64_t m, int P, int cap) {
  const int64_t c = ((m + P - 1) / P + 31) / 32 * 32;
  return (int)(c < cap ? c : cap);
}
// dynamic shared memory of the panel kernel: the chunk (odd leading dimension), the slots, and in
// FP32 two copies of a column
template <typename T> constexpr size_t panel_smem_bytes(int chunk, int width, int P) {
  return 2 * sizeof(T) * ((size_t)(chunk | 1) * width + 2 * (size_t)P * kNB + (sizeof(T) == 8 ? 0 : 2 * (size_t)chunk));
}

// Pivot candidates compare |re| + |im| through the bit pattern of the (non-negative) value as
// an unsigned integer, which orders like the value (and puts a NaN above every number): FP64
// comparisons run on GB300's narrow FP64 pipe, integer ones do not.  "No candidate" is key 0
// with row INT_MAX, which loses against any row (a zero column is recognised by the key 0).  A NaN
// that wins leaves nothing but NaN; in FP64 it is reported like a zero pivot, so that a matrix that is
// not finite is refused (in FP32 the refinement fails and the FP64 factorization decides).
template <typename T> struct PivotKey;
template <> struct PivotKey<double> {
  using type = unsigned long long;
  static constexpr type kInf = 0x7FF0000000000000ull;
  __device__ static __forceinline__ type of(double v) { return (type)__double_as_longlong(v); }
};
template <> struct PivotKey<float> {
  using type = unsigned;
  static constexpr type kInf = 0xFFFFFFFFu;  // no key is above it
  __device__ static __forceinline__ type of(float v) { return __float_as_uint(v); }
};

// (key, row) of the larger |re| + |im|; ties go to the smaller row (izamax's first maximum)
template <typename K> __device__ __forceinline__ void argmax_merge(K& v, int& i, K ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
// over the warp, by the warp-wide integer reductions (three for a 64-bit key, two for a 32-bit
// one, against five rounds of three shuffles)
__device__ __forceinline__ void warp_argmax(unsigned long long& v, int& i) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  i = (int)__reduce_min_sync(0xffffffffu, (unsigned)((hi == mh && lo == ml) ? i : INT_MAX));
  v = ((unsigned long long)mh << 32) | ml;
}
__device__ __forceinline__ void warp_argmax(unsigned& v, int& i) {
  const unsigned m = __reduce_max_sync(0xffffffffu, v);
  i = (int)__reduce_min_sync(0xffffffffu, (unsigned)(v == m ? i : INT_MAX));
  v = m;
}

// split cluster barrier: arrive (releasing this thread's writes), later wait (acquiring
// every thread's writes before their arrive)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Rows k .. n-1 of the panel (m = n - k panel rows, panel row r = matrix row k + r) are
// split into chunks of `chunk` rows (a multiple of 32, so that no warp of the update is left
// part empty; CTA 0 holds the kb <= 32 diagonal rows), one per CTA, in its shared memory with
// an odd leading dimension (a row's entries then sit in different banks).  Per column j:
//   warp q < P pushes this CTA's candidate (key, row number, reciprocal, a copy of its row) into
//   CTA q's slot (distributed shared memory stores); CTA 0 pushes row j; cluster barrier; every
//   warp picks the winner among the P slots, now local;
//   FP64: a thread per row forms the multipliers l (the interchanged row's from the copy of
//   row j); CTA barrier.  FP32: every item of the update forms its own, from a copy of the
//   column;
//   column j + 1 is updated and searched first, by warps 0 .. 14; then they take the rest of the
//   rank-1 update in items of 32 rows by a few columns while warp 15 merges their candidates
//   and takes the reciprocal of this CTA's; CTA barrier.
// What bounds it: for few rows the chain of barriers, reductions and the reciprocal, for many
// the FP64 pipe (124 FMAs per row at j = 0, two per clock and SM).  A warp issues to one of the
// SM's four FP64 pipes, so the update goes by items and not by one thread per row (that left
// three pipes idle for 32 rows, and a fifth of the time at 400).  Cycles per column, before -> now
// (before: one warp pushed to all CTAs, 500 to 850; the reciprocal was taken on every CTA after
// the barrier, 850 in FP64 and 330 in FP32, now under the update; FP32 scaled in a pass of its own,
// 415; items of four and eight columns were too few for the warps, 2115 and 1190 for the update
// of 32 rows): FP64 200 rows 5290 -> 4590, five matrices of 1000 7080 -> 6170, 3000 12080 -> 10350;
// FP32 430 rows 3290 -> 2390, 1400 3890 -> 3160, 8000 5900 -> 5740.  Measured and dropped: fewer FP64
// operations in the reciprocal, and fewer warps on the FP64 pipe beside it (4730 and 4890 at 200
// rows: the reciprocal's chain is bound by its instructions' latency, not by the pipe).
// Slots of parity j are written again at column j + 2, after the barrier of column j + 1, which
// every CTA reaches only when it is done reading column j's.
constexpr int kItemWarps = kPanelThreads / 32 - 1;  // the last warp merges and takes the reciprocal
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
template <typename T>
__global__ void __launch_bounds__(kPanelThreads) panel_cluster_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                                     int32_t* __restrict__ ipiv_all,
                                                                     int32_t* __restrict__ info_all, int64_t k,
                                                                     int chunk_cap, int width) {
  using C = typename cplx_t<T>::type;
  using K = typename PivotKey<T>::type;
  constexpr int kWarps = kPanelThreads / 32;
  constexpr bool kScaleApart = sizeof(T) == 8;  // multipliers formed once per row (FP64 work is dear)
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char panel_smem[];
  C* sp = reinterpret_cast<C*>(panel_smem);            // chunk x kb, column-major (leading dimension ld)
  C* slots = sp + (size_t)(chunk_cap | 1) * width;     // candidate rows [parity][CTA][kNB]
  __shared__ C pub_j[2][kNB];                          // row j
  __shared__ K cand_v[2][kPanelMaxCtas];
  __shared__ int cand_i[2][kPanelMaxCtas];
  __shared__ C cand_inv[2][kPanelMaxCtas];
  __shared__ K red_v[kWarps];
  __shared__ int red_i[kWarps];
  __shared__ K s_key;
  __shared__ int s_row;
  __shared__ C s_inv;
  const int P = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  C* acol = slots + 2 * P * kNB;  // FP32: column j as the previous update left it [parity][chunk]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t bmat = blockIdx.y, n = d.order(bmat);
  if (k >= n) return;  // a grouped batch: this matrix is factored (the whole cluster leaves)
  cluster_arrive();    // every CTA of the cluster runs before the first push
  C* A = Aall + d.offset(bmat);
  const int64_t m = n - k;
  const int kb = (int)(m < width ? m : width);  // panel width: 32, or 16 for a half of a two-level panel
  const int chunk = panel_chunk(m, P, chunk_cap);
  const int ld = chunk | 1;
  const int r0 = rank * chunk;  // first panel row of this CTA
  const int rows = (int)((m - r0) < chunk ? ((m - r0) > 0 ? (m - r0) : 0) : chunk);
  const int nrb = (rows + 31) >> 5;
  C* Ap = A + (k + r0) + k * n;

#pragma unroll 4
  for (int q = warp; q < nrb * kb; q += kWarps) {
    const int c = q / nrb, i = (q - c * nrb) * 32 + lane;
    if (i < rows) sp[c * ld + i] = Ap[i + c * n];
  }
  // candidate for column 0 (the rows that this thread loaded)
  K best = 0;
  int bi = INT_MAX;
  for (int q = warp; q < nrb; q += kWarps) {
    const int i = q * 32 + lane;
    if (i < rows) {
      const C a = sp[i];
      if (!kScaleApart) acol[i] = a;
      argmax_merge(best, bi, PivotKey<T>::of(fabs(a.x) + fabs(a.y)), r0 + i);
    }
  }
  warp_argmax(best, bi);
  if (lane == 0) { red_v[warp] = best; red_i[warp] = bi; }
  __syncthreads();
  // warp 15: this CTA's candidate in column c, from the `w` warps that searched it
  auto publish = [&](int c, int w) {
    K v = lane < w ? red_v[lane] : (K)0;
    int vi = lane < w ? red_i[lane] : INT_MAX;
    warp_argmax(v, vi);
    C inv = czero<C>();
    if (v != 0) inv = crecip(sp[c * ld + (vi - r0)]);
    if (lane == 0) { s_key = v; s_row = vi; s_inv = inv; }
  };
  if (warp == kItemWarps) publish(0, kWarps);
  // the update's items: nrb of column j + 1, then (column group g, row block rb) in turn, item q
  // to warp q % kItemWarps; this warp's first item past column j + 1, and its step
  const int searchers = nrb < kItemWarps ? nrb : kItemWarps;
  const int qb = nrb > 0 ? ((nrb - warp + kItemWarps - 1) / kItemWarps * kItemWarps + warp - nrb) : 0;
  const int first = nrb > warp ? qb : warp - nrb;
  const int g0 = nrb > 0 ? first / nrb : 0, rb0 = nrb > 0 ? first - g0 * nrb : 0;
  const int dg = nrb > 0 ? kItemWarps / nrb : 0, drb = nrb > 0 ? kItemWarps - dg * nrb : 0;
  cluster_wait();
  for (int j = 0; j < kb; ++j) {
    const int par = j & 1;
    __syncthreads();
    if (warp < P) {
      const int li = s_row - r0;
      C* slot = slots + (par * P + rank) * kNB + lane;
      if (s_row != INT_MAX && lane < kb) *cl.map_shared_rank(slot, (unsigned)warp) = sp[lane * ld + li];
      if (rank == 0 && lane < kb) *cl.map_shared_rank(&pub_j[par][lane], (unsigned)warp) = sp[lane * ld + j];
      if (lane == 0) {
        *cl.map_shared_rank(&cand_v[par][rank], (unsigned)warp) = s_key;
        *cl.map_shared_rank(&cand_i[par][rank], (unsigned)warp) = s_row;
        *cl.map_shared_rank(&cand_inv[par][rank], (unsigned)warp) = s_inv;
      }
    }
    cluster_arrive();
    cluster_wait();
    K v = lane < P ? cand_v[par][lane] : (K)0;
    const int ci = lane < P ? cand_i[par][lane] : INT_MAX;
    int p = ci;
    warp_argmax(v, p);
    const bool zero = v == 0;
    const int win = zero ? 0 : __ffs(__ballot_sync(0xffffffffu, ci == p)) - 1;  // the CTA that holds the pivot
    if (zero) p = j;                                                            // panel row of the pivot
    const C* jrow = pub_j[par];
    const C* urow = zero ? jrow : slots + (par * P + win) * kNB;
    const C inv = zero ? czero<C>() : cand_inv[par][win];
    const int lp = (p != j && rank == win) ? p - r0 : -1;  // this CTA's row that takes row j
    if (kScaleApart) {
      for (int i = tid; i < rows; i += kPanelThreads)
        if (r0 + i > j) sp[j * ld + i] = cmul(i == lp ? jrow[j] : sp[j * ld + i], inv);
      __syncthreads();
    }
    if (warp == kItemWarps) {
      if (p != j) {  // the interchanged rows' entries that the update leaves alone
        if (rank == 0 && lane < kb) sp[lane * ld + j] = urow[lane];
        if (lp >= 0 && lane < j) sp[lane * ld + lp] = jrow[lane];
      }
      if (lane == 0 && rank == 0) {
        ipiv_all[bmat * ipiv_stride(d.n) + k + j] = (int32_t)(k + p);
        if ((zero || v > PivotKey<T>::kInf) && info_all[bmat] == 0) info_all[bmat] = (int32_t)(k + j + 1);
      }
      if (j + 1 < kb) {
        bar_sync(1, 32 * (searchers + 1));
        publish(j + 1, searchers);
      }
      continue;
    }
    // the multiplier of row i
    auto multiplier = [&](int i) {
      if (kScaleApart) return sp[j * ld + i];
      return cmul(i == lp ? jrow[j] : acol[par * chunk + i], inv);
    };
    best = 0;
    bi = INT_MAX;
    for (int rb = warp; rb < nrb; rb += kItemWarps) {
      const int i = rb * 32 + lane;
      if (i >= rows || r0 + i <= j) continue;
      const C l = multiplier(i);
      if (!kScaleApart) sp[j * ld + i] = l;
      if (j + 1 < kb) {
        const C x = cfms(i == lp ? jrow[j + 1] : sp[(j + 1) * ld + i], l, urow[j + 1]);
        sp[(j + 1) * ld + i] = x;
        if (!kScaleApart) acol[(par ^ 1) * chunk + i] = x;
        argmax_merge(best, bi, PivotKey<T>::of(fabs(x.x) + fabs(x.y)), r0 + i);
      }
    }
    if (j + 1 < kb && warp < searchers) {
      warp_argmax(best, bi);
      if (lane == 0) { red_v[warp] = best; red_i[warp] = bi; }
      __syncwarp();
      bar_arrive(1, 32 * (searchers + 1));
    }
    auto rest = [&](auto width_of_item) {
      constexpr int GC = decltype(width_of_item)::value;
      int g = g0, rb = rb0;
      while (j + 2 + g * GC < kb) {
        const int i = rb * 32 + lane, c0 = j + 2 + g * GC;
        if (i < rows && r0 + i > j) {
          const C l = multiplier(i);
          C x[GC];
#pragma unroll
          for (int t = 0; t < GC; ++t)
            if (c0 + t < kb) x[t] = i == lp ? jrow[c0 + t] : sp[(c0 + t) * ld + i];
#pragma unroll
          for (int t = 0; t < GC; ++t)
            if (c0 + t < kb) sp[(c0 + t) * ld + i] = cfms(x[t], l, urow[c0 + t]);
        }
        g += dg;
        rb += drb;
        if (rb >= nrb) { rb -= nrb; ++g; }
      }
    };
    if (nrb > 0) {
      // As few columns per item as keep the multipliers' loads (FP32: and products) in the shade.
      // All panels of one factorization, ms, this rule against 1, 2, 4 and 8 columns throughout: FP64
      // order 200 0.437 (0.440 0.451 0.442 0.544), 900 2.30 (2.31 2.37 2.37 2.75), 4500 20.4 (20.0 20.5
      // 21.3 23.8); FP32 200 0.238 (0.240 0.237 0.246 0.276), 900 1.26 (1.27 1.25 1.27 1.41), 4500 8.52
      // (8.81 8.49 8.29 8.73).
      if (nrb <= 2) rest(std::integral_constant<int, sizeof(T) == 8 ? 1 : 2>());
      else if (sizeof(T) == 8 || nrb <= 6) rest(std::integral_constant<int, sizeof(T) == 8 ? 2 : 4>());
      else rest(std::integral_constant<int, 8>());
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int q = warp; q < nrb * kb; q += kWarps) {
    const int c = q / nrb, i = (q - c * nrb) * 32 + lane;
    if (i < rows) Ap[i + c * n] = sp[c * ld + i];
  }
}

// The interchanges of panel step k as one permutation: final row dst = original row src for
// at most 64 (dst, src) pairs (-1: none).  Slot s < 32 is panel row s, slot 32 + q is the
// row below the diagonal block that step q chose first.  Runs on warp 0.
__device__ void panel_permutation(const int32_t* __restrict__ ipiv, int64_t k, int kb, int* s_slot,
                                  int* s_content, int* s_dst, int* s_src) {
  const int lane = threadIdx.x & 31;
  const int p = lane < kb ? (int)(ipiv[k + lane] - k) : lane;  // panel row chosen at step lane
  int first = lane;
  for (int q = 31; q >= 0; --q) {
    const int pq = __shfl_sync(0xffffffffu, p, q);
    if (q < lane && pq == p) first = q;
  }
  s_slot[lane] = p < kNB ? p : kNB + first;
  s_content[lane] = lane;
  s_content[lane + 32] = lane + 32;
  __syncwarp();
  if (lane == 0)
    for (int j = 0; j < kb; ++j) {
      const int a = j, b = s_slot[j];
      const int t = s_content[a];
      s_content[a] = s_content[b];
      s_content[b] = t;
    }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int sl = lane + 32 * h;
    const int src = s_content[sl];
    const int q = src >= kNB ? src - kNB : 0;
    const int psrc = __shfl_sync(0xffffffffu, p, q);
    const bool live = src != sl;
    s_dst[sl] = live ? (int)(k + (sl < kNB ? sl : p)) : -1;  // slot 32 + lane is the row p of this lane
    s_src[sl] = live ? (int)(k + (src < kNB ? src : psrc)) : -1;
  }
}

// Applies panel step k's interchanges to the columns outside the panel: one warp per
// column, all loads of a column before its stores.
constexpr int kSwpCols = 64;  // columns per CTA (the permutation is built once per CTA)
template <typename T>
__global__ void __launch_bounds__(256) laswp_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                   const int32_t* __restrict__ ipiv_all, int64_t k, int kb) {
  using C = typename cplx_t<T>::type;
  __shared__ int s_slot[32], s_content[64], s_dst[64], s_src[64];
  const int64_t bmat = blockIdx.y, n = d.order(bmat);
  if (k >= n) return;  // a grouped batch: this matrix is factored
  kb = (int)((k + kNB < n) ? kNB : n - k);
  if (threadIdx.x < 32) panel_permutation(ipiv_all + bmat * ipiv_stride(d.n), k, kb, s_slot, s_content, s_dst, s_src);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d0 = s_dst[lane], s0 = s_src[lane], d1 = s_dst[lane + 32], s1 = s_src[lane + 32];
  C* A = Aall + d.offset(bmat);
  const int64_t nout = n + d.extra - kb;  // columns outside the panel, appended right-hand sides included
  const int64_t q0 = blockIdx.x * (int64_t)kSwpCols;
  const int64_t q1 = (q0 + kSwpCols < nout) ? q0 + kSwpCols : nout;
  for (int64_t q = q0 + warp; q < q1; q += 8) {
    C* col = A + (q < k ? q : q + kb) * n;
    C v0 = czero<C>(), v1 = czero<C>();
    if (d0 >= 0) v0 = col[s0];
    if (d1 >= 0) v1 = col[s1];
    __syncwarp();
    if (d0 >= 0) col[d0] = v0;
    if (d1 >= 0) col[d1] = v1;
  }
}

// The interchanges of the kb panel rows at k applied to the columns [c0, c1) (the other half
// of a two-level panel); one warp per column as in laswp_kernel.
template <typename T>
__global__ void __launch_bounds__(256) laswp_cols_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                        const int32_t* __restrict__ ipiv_all, int64_t k, int kb,
                                                        int64_t c0, int64_t c1) {
  using C = typename cplx_t<T>::type;
  __shared__ int s_slot[32], s_content[64], s_dst[64], s_src[64];
  const int64_t bmat = blockIdx.y, n = d.order(bmat);
  if (k + kb > n) return;
  if (threadIdx.x < 32) panel_permutation(ipiv_all + bmat * ipiv_stride(d.n), k, kb, s_slot, s_content, s_dst, s_src);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d0 = s_dst[lane], s0 = s_src[lane], d1 = s_dst[lane + 32], s1 = s_src[lane + 32];
  C* A = Aall + d.offset(bmat);
  const int64_t q0 = c0 + blockIdx.x * (int64_t)kSwpCols;
  const int64_t q1 = (q0 + kSwpCols < c1) ? q0 + kSwpCols : c1;
  for (int64_t q = q0 + warp; q < q1; q += 8) {
    C* col = A + q * n;
    C v0 = czero<C>(), v1 = czero<C>();
    if (d0 >= 0) v0 = col[s0];
    if (d1 >= 0) v1 = col[s1];
    __syncwarp();
    if (d0 >= 0) col[d0] = v0;
    if (d1 >= 0) col[d1] = v1;
  }
}

// U12' = L11'^-1 A[k:k+16, k+16:k+32] of a two-level panel (L11' the unit lower 16 x 16 block of
// the left half): the column-oriented forward substitution with the (15 - r) x 16 updates of
// step r spread over the CTA's threads (GB300's FP64 work has to reach all four schedulers).
template <typename T>
__global__ void __launch_bounds__(256) trsm16_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                    int64_t k) {
  using C = typename cplx_t<T>::type;
  constexpr int H = kNB / 2;
  __shared__ C sL[H][H + 1], sB[H][H + 1];
  const int64_t n = d.order(blockIdx.x);
  if (k + kNB > n) return;
  C* A = Aall + d.offset(blockIdx.x);
  for (int idx = threadIdx.x; idx < H * H; idx += blockDim.x) {
    const int r = idx % H, q = idx / H;
    sL[r][q] = A[(k + r) + (k + q) * n];
    sB[r][q] = A[(k + r) + (k + H + q) * n];
  }
  __syncthreads();
  for (int r = 0; r < H - 1; ++r) {
    const int ne = (H - 1 - r) * H;
    for (int e = threadIdx.x; e < ne; e += blockDim.x) {
      const int srow = r + 1 + e / H, c = e % H;
      sB[srow][c] = cfms(sB[srow][c], sL[srow][r], sB[r][c]);
    }
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < H * H; idx += blockDim.x) {
    const int r = idx % H, q = idx / H;
    A[(k + r) + (k + H + q) * n] = sB[r][q];
  }
}

// ------------------------------- U12 -----------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) trsm_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                   int64_t k) {
  using C = typename cplx_t<T>::type;
  __shared__ C sL[kNB][kNB + 1];
  const int64_t n = d.order(blockIdx.y), ncols = n + d.extra;
  if (k >= n) return;  // this matrix is factored (grouped batches)
  C* A = Aall + d.offset(blockIdx.y);
  const int kb = (int)((k + kNB < n) ? kNB : n - k);
  if (k + kb >= ncols) return;  // nothing right of the panel
  for (int idx = threadIdx.x; idx < kb * kb; idx += blockDim.x) {
    int r = idx % kb, q = idx / kb;
    sL[r][q] = A[(k + r) + (k + q) * n];
  }
  __syncthreads();
  const int64_t c = k + kb + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  C x[kNB];
#pragma unroll
  for (int r = 0; r < kNB; ++r) x[r] = (r < kb) ? A[(k + r) + c * n] : czero<C>();
#pragma unroll
  for (int r = 1; r < kNB; ++r) {
#pragma unroll
    for (int q = 0; q < r; ++q) x[r] = cfms(x[r], sL[r][q], x[q]);
  }
#pragma unroll
  for (int r = 0; r < kNB; ++r)
    if (r < kb) A[(k + r) + c * n] = x[r];
}

// U12 of the second of two panels taken together (rows k + 32 .. k + 63 of the columns right of
// k + 64): L22^-1 (A - L21 Ua), Ua the first panel's U12 already in place; one thread per column.
__global__ void __launch_bounds__(128) trsm_second_kernel(BatchDesc d, float2* __restrict__ Aall, int64_t k) {
  __shared__ float2 sL[2 * kNB][kNB];  // rows k + 32 .. of columns k .. k + 63, by column
  const int64_t n = d.order(blockIdx.y);
  if (k + 2 * kNB >= n) return;  // a grouped batch: no column of this matrix is right of both panels
  float2* A = Aall + d.offset(blockIdx.y);
  for (int idx = threadIdx.x; idx < 2 * kNB * kNB; idx += blockDim.x) {
    const int r = idx & (kNB - 1), q = idx / kNB;
    sL[q][r] = A[(k + kNB + r) + (k + q) * n];
  }
  __syncthreads();
  const int64_t c = k + 2 * kNB + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  float2* col = A + k + c * n;
  float2 x[kNB];
#pragma unroll
  for (int r = 0; r < kNB; ++r) x[r] = col[kNB + r];
#pragma unroll 8
  for (int q = 0; q < kNB; ++q) {
    const float2 u = col[q];
#pragma unroll
    for (int r = 0; r < kNB; ++r) x[r] = cfms(x[r], sL[q][r], u);
  }
#pragma unroll
  for (int q = 0; q < kNB - 1; ++q) {
#pragma unroll
    for (int r = q + 1; r < kNB; ++r) x[r] = cfms(x[r], sL[kNB + q][r], x[q]);
  }
#pragma unroll
  for (int r = 0; r < kNB; ++r) col[kNB + r] = x[r];
}

// FP64: LANES (8 or 32) lanes per column, lane l holding rows l, l + LANES, ..; the column-oriented
// substitution broadcasts x_q within them and every lane updates its rows below q.  A warp gets
// one FP64 instruction per 77 cycles and an SM one per 19, so with few columns the chain counts:
// one thread per column (trsm_kernel) runs 1984 FMAs in a row, 74 us whatever the width, eight lanes
// 320 in 23 us, 32 lanes 124 in 12 us while every SM has one CTA of eight columns and in 20 us while it
// has two.  With more columns the pipe counts, and eight lanes waste less of it (four columns share
// a warp's instruction): 2400 columns in all 23.5 us with eight lanes against 28.6 with 32.
constexpr int kTrsmThreads = 256;
constexpr int64_t kTrsmFewColumns = 2 * 152 * (kTrsmThreads / 32);
template <int LANES>
__global__ void __launch_bounds__(kTrsmThreads) trsm_lanes_kernel(BatchDesc d, double2* __restrict__ Aall, int64_t k) {
  constexpr int kRowsPer = kNB / LANES, kCols = kTrsmThreads / LANES;
  __shared__ double2 sL[kNB][kNB + 1];
  const int64_t n = d.order(blockIdx.y), ncols = n + d.extra;
  if (k >= n) return;  // this matrix is factored (grouped batches)
  double2* A = Aall + d.offset(blockIdx.y);
  const int kb = (int)((k + kNB < n) ? kNB : n - k);
  if (k + kb + blockIdx.x * (int64_t)kCols >= ncols) return;  // nothing right of the panel here
  for (int idx = threadIdx.x; idx < kNB * kNB; idx += blockDim.x) {
    const int r = idx & (kNB - 1), q = idx / kNB;
    sL[r][q] = (r < kb && q < kb) ? A[(k + r) + (k + q) * n] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int64_t c = k + kb + blockIdx.x * (int64_t)kCols + threadIdx.x / LANES;
  const bool live = c < ncols;
  const int l = threadIdx.x & (LANES - 1), base = threadIdx.x & 31 & ~(LANES - 1);  // first lane of this column
  double2 x[kRowsPer];
#pragma unroll
  for (int t = 0; t < kRowsPer; ++t)
    x[t] = (live && l + LANES * t < kb) ? A[(k + l + LANES * t) + c * n] : make_double2(0.0, 0.0);
#pragma unroll
  for (int q = 0; q < kNB - 1; ++q) {
    const double2 xq = shfl_c(x[q / LANES], base | (q & (LANES - 1)));
#pragma unroll
    for (int t = q / LANES; t < kRowsPer; ++t) {
      const int r = l + LANES * t;
      if (r > q) x[t] = cfms(x[t], sL[r][q], xq);
    }
  }
#pragma unroll
  for (int t = 0; t < kRowsPer; ++t)
    if (live && l + LANES * t < kb) A[(k + l + LANES * t) + c * n] = x[t];
}

// ------------------------------ trailing update -------------------------------
// A22 -= L21 U12 in FP64 with Gauss's three-multiplication complex product (the ZGEMM3M
// scheme): per complex multiply-add P1 += ar br, P2 += ai bi, P3 += (ar + ai)(br + bi), and
// at the end Re = P1 - P2, Im = P3 - P1 - P2 -- three FP64 FMAs instead of four.  The sums
// ar + ai, br + bi are formed once per element when the tiles are staged in shared memory
// (three planes: Re, Im, Re + Im).  The product is normwise stable (its error is bounded by
// a small multiple of the unit roundoff times |L21| |U12|), which is the property the LU's
// backward stability rests on; componentwise the imaginary parts can differ from the
// four-multiplication product in the last digits.
// Tile: 16 RM x 16 RM outputs per CTA of 256 threads.  The FP64 pipe bounds it at every tile size
// (98 % busy; an RM = 4 tile keeps an SM for 95 us, RM = 2 24 us, RM = 1 6 us), so the tile only
// has to be small enough that the launch's tiles fill the SMs evenly: RM = 2 from 8 tiles per
// SM, RM = 1 below.  Per panel step: order 200 110 -> 12 us, 450 111 -> 21 us, five of 1000
// 374 -> 300 us.
constexpr int kG3KC = 16;
template <int RM>
__global__ void __launch_bounds__(256) gemm3m_kernel(BatchDesc d, double2* __restrict__ Aall, int64_t k) {
  constexpr int kG3RM = RM, kG3TM = 16 * RM;
  __shared__ double sAr[kG3KC][kG3TM + 1], sAi[kG3KC][kG3TM + 1], sAs[kG3KC][kG3TM + 1];
  __shared__ double sBr[kG3KC][kG3TM + 1], sBi[kG3KC][kG3TM + 1], sBs[kG3KC][kG3TM + 1];
  const int64_t n = d.order(blockIdx.z);
  if (k + kNB >= n) return;  // no trailing block for this matrix (grouped batches)
  double2* A = Aall + d.offset(blockIdx.z);
  const int kb = (int)((k + kNB < n) ? kNB : n - k);
  const int64_t base = k + kb;
  const int64_t row0 = base + blockIdx.x * (int64_t)kG3TM;
  const int64_t col0 = base + blockIdx.y * (int64_t)kG3TM;
  if (row0 >= n || col0 >= n) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double p1[kG3RM][kG3RM], p2[kG3RM][kG3RM], p3[kG3RM][kG3RM];
#pragma unroll
  for (int r = 0; r < kG3RM; ++r)
#pragma unroll
    for (int c = 0; c < kG3RM; ++c) p1[r][c] = p2[r][c] = p3[r][c] = 0.0;
  for (int k0 = 0; k0 < kb; k0 += kG3KC) {
    for (int idx = threadIdx.x; idx < kG3KC * kG3TM; idx += 256) {
      const int r = idx % kG3TM, q = idx / kG3TM;
      const int64_t gi = row0 + r;
      const int kk = k0 + q;
      const double2 v = (gi < n && kk < kb) ? A[gi + (k + kk) * n] : make_double2(0.0, 0.0);
      sAr[q][r] = v.x;
      sAi[q][r] = v.y;
      sAs[q][r] = v.x + v.y;
    }
    for (int idx = threadIdx.x; idx < kG3KC * kG3TM; idx += 256) {
      const int q = idx % kG3KC, c = idx / kG3KC;
      const int64_t gc = col0 + c;
      const int kk = k0 + q;
      const double2 v = (gc < n && kk < kb) ? A[(k + kk) + gc * n] : make_double2(0.0, 0.0);
      sBr[q][c] = v.x;
      sBi[q][c] = v.y;
      sBs[q][c] = v.x + v.y;
    }
    __syncthreads();
#pragma unroll 4
    for (int q = 0; q < kG3KC; ++q) {
      double ar[kG3RM], ai[kG3RM], as[kG3RM];
#pragma unroll
      for (int r = 0; r < kG3RM; ++r) {
        ar[r] = sAr[q][tx + 16 * r];
        ai[r] = sAi[q][tx + 16 * r];
        as[r] = sAs[q][tx + 16 * r];
      }
#pragma unroll
      for (int c = 0; c < kG3RM; ++c) {
        const double br = sBr[q][ty + 16 * c], bi = sBi[q][ty + 16 * c], bs = sBs[q][ty + 16 * c];
#pragma unroll
        for (int r = 0; r < kG3RM; ++r) {
          p1[r][c] = fma(ar[r], br, p1[r][c]);
          p2[r][c] = fma(ai[r], bi, p2[r][c]);
          p3[r][c] = fma(as[r], bs, p3[r][c]);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < kG3RM; ++c) {
    const int64_t gc = col0 + ty + 16 * c;
    if (gc >= n) continue;
#pragma unroll
    for (int r = 0; r < kG3RM; ++r) {
      const int64_t gi = row0 + tx + 16 * r;
      if (gi < n) {
        double2 v = A[gi + gc * n];
        v.x -= p1[r][c] - p2[r][c];
        v.y -= p3[r][c] - p1[r][c] - p2[r][c];
        A[gi + gc * n] = v;
      }
    }
  }
}

// ------------------------------ substitution ---------------------------------
// After the last panel step lu_finish_kernel turns the factors into what the substitutions read:
// the 32 x 32 diagonal blocks of L and U are replaced by their inverses (each in its own
// triangle, L's unit diagonal implied) and the pivot sequence by the row permutation it
// composes to (x = b[sigma] applies the interchanges).  Block substitution with inverted
// diagonal blocks turns the 64-step dependent chain of each block into a product (Higham,
// Accuracy and Stability of Numerical Algorithms, 2nd ed., sec. 14.2; 14.3 for its error), and
// both are done once per factorization, whatever the number of solves.
// The product's residual exceeds the substitution's by up to k = | |T| |T^-1| |_inf of the block,
// so in FP64 a triangle with k above 512 stays as it is and is solved by substitution (its bit
// in the block's flag word: 1 for L, 2 for U).  Second-kind boundary operators have k of 1 to 20,
// random matrices 100 to 300, a Hilbert-like matrix millions.  FP32 factors are refined.
// |x| to FP32 precision from the bits (a conversion instruction would run on the FP64 pipe): 0
// below FP32's normal range, a NaN pattern above it
__device__ __forceinline__ float magnitude_f32(double x) {
  const unsigned hi = (unsigned)(__double_as_longlong(x) >> 32) & 0x7FFFFFFFu;
  const int e = (int)(hi >> 20) - 896;  // biased exponent in FP32
  return e <= 0 ? 0.0f : (e >= 255 ? __uint_as_float(0x7FFFFFFFu) : __uint_as_float((unsigned)e << 23 | (hi & 0xFFFFFu) << 3));
}
__device__ __forceinline__ float magnitude_f32(float x) { return fabsf(x); }
constexpr int kFinishThreads = 256;
constexpr int kFinishMaxSmem = 2 * 4 * 12288;  // the permutation of the largest order the library takes
constexpr float kFinishGrowth = 512.0f;
template <typename T>
__global__ void __launch_bounds__(kFinishThreads) lu_finish_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ Aall,
                                                                  int32_t* __restrict__ ipiv_all, int nblk) {
  using C = typename cplx_t<T>::type;
  __shared__ C sM[kNB][kNB + 1], sX[kNB][kNB + 1];
  __shared__ C rd[kNB];
  __shared__ float ssum[2][kNB];
  extern __shared__ int finish_smem[];
  const int64_t n = d.order(blockIdx.y);
  int32_t* ipiv = ipiv_all + blockIdx.y * ipiv_stride(d.n);
  const int tid = threadIdx.x;
  const bool upper_only = d.extra > 0;  // the right-hand sides went through the factorization: only U is solved
  if ((int)blockIdx.x == nblk) {
    if (upper_only) return;
    // the permutation: sequential in the pivots, one thread, from shared memory
    int* sig = finish_smem;
    int* piv = finish_smem + d.n;
    for (int64_t i = tid; i < n; i += kFinishThreads) { sig[i] = (int)i; piv[i] = ipiv[i]; }
    __syncthreads();
    if (tid == 0) {
      int next = piv[0];
      for (int j = 0; j < (int)n; ++j) {
        const int q = next;
        next = j + 1 < (int)n ? piv[j + 1] : 0;  // off the exchange's chain
        const int a = sig[j], b = sig[q];
        sig[j] = b;
        sig[q] = a;
      }
    }
    __syncthreads();
    for (int64_t i = tid; i < n; i += kFinishThreads) ipiv[i] = sig[i];
    return;
  }
  const int64_t jb = (int64_t)blockIdx.x * kNB;
  if (jb >= n) return;
  const int bw = (int)(n - jb < kNB ? n - jb : kNB);
  C* A = Aall + d.offset(blockIdx.y) + jb + jb * n;
  // the block and the identity: L X = I runs on the strict lower triangles of sM and sX, U X = I
  // on the upper ones, at the same time (their steps touch different entries)
  for (int e = tid; e < kNB * kNB; e += kFinishThreads) {
    const int r = e & (kNB - 1), c = e / kNB;
    sM[r][c] = (r < bw && c < bw) ? A[r + c * n] : czero<C>();
    C x = czero<C>();
    if (r == c) x.x = 1;
    sX[r][c] = x;
  }
  __syncthreads();
  if (tid < bw) {
    rd[tid] = crecip(sM[tid][tid]);
    sX[tid][tid] = rd[tid];  // the diagonal of U^-1 (L^-1's is 1)
  }
  __syncthreads();
  for (int s = 0; s < bw - 1; ++s) {
    // L: column oriented, once row s of X is final rows q > s take -L[q][s] X[s][c], c <= s
    // U: from the bottom, once row t of X is final rows q < t take -U[q][t] X[t][c], c >= t, and row
    // t - 1 is then scaled by 1 / U[t-1][t-1]
    const int t = bw - 1 - s, w = s + 1, ne = (bw - 1 - s) * w;
    for (int e = tid + (upper_only ? ne : 0); e < 2 * ne; e += kFinishThreads) {
      if (e < ne) {
        const int q = s + 1 + e / w, c = e % w;
        C x = c == s ? czero<C>() : sX[s][c];
        if (c == s) x.x = 1;
        sX[q][c] = cfms(sX[q][c], sM[q][s], x);
      } else {
        const int q = (e - ne) / w, c = t + (e - ne) % w;
        const C v = cfms(sX[q][c], sM[q][t], sX[t][c]);
        sX[q][c] = q == t - 1 ? cmul(v, rd[q]) : v;
      }
    }
    __syncthreads();
  }
  bool keep_l = false, keep_u = false;
  if (sizeof(T) == 8) {
    // k of both triangles, in FP32: row sums of |X|, then |T| times them
    const int r = tid & (kNB - 1), part = tid >> 5;
    auto mag = [](C v) { return magnitude_f32(v.x) + magnitude_f32(v.y); };
    if (part < 2) {
      float sum = 0.0f;
      for (int c = 0; c < bw; ++c) {
        if (part == 0) sum += c < r ? mag(sX[r][c]) : (c == r ? 1.0f : 0.0f);
        else if (c >= r) sum += mag(sX[r][c]);
      }
      ssum[part][r] = sum;
    }
    __syncthreads();
    float k = 0.0f;
    if (part < 2 && r < bw)
      for (int c = 0; c < bw; ++c) {
        if (part == 0) k += c < r ? mag(sM[r][c]) * ssum[0][c] : (c == r ? ssum[0][c] : 0.0f);
        else if (c >= r) k += mag(sM[r][c]) * ssum[1][c];
      }
    const bool big = !(k <= kFinishGrowth);  // also for NaN
    keep_l = __syncthreads_or(part == 0 && big);
    keep_u = __syncthreads_or(part == 1 && big);
  }
  if (tid == 0) ipiv[d.n + blockIdx.x] = (keep_l ? 1 : 0) | (keep_u ? 2 : 0);
  for (int e = tid; e < kNB * kNB; e += kFinishThreads) {
    const int r = e & (kNB - 1), c = e / kNB;
    if (r < bw && c < bw && !(r > c ? keep_l || upper_only : keep_u)) A[r + c * n] = sX[r][c];
  }
}

// One cluster of P CTAs per (group of g <= kSG right-hand sides, matrix).  The 32-row blocks of
// the solution are dealt out cyclically (block b to CTA b % P); each CTA keeps its blocks'
// entries of the g vectors in shared memory.  The solve is a sequence of 2 nblk block steps (L
// then U, or U^H then L^H for A^H x = b = U^H L^H P^T x).  At step s every CTA has x_s, the
// block solved last, in a slot of its own.  The owner of block s + 1 takes x_s into that block's
// rows, multiplies by the inverted diagonal block and pushes the result into the slots of all
// P CTAs (four warps, one per FP64 pipe; both 32 x 32 operands were brought into shared
// memory a step ahead); all arrive at the split cluster barrier, take x_s into the rest of
// their rows, and wait.  Three slots: a CTA may still read x_(s-1) while x_(s+1) arrives.
//
// Bound: the chain of 2 nblk steps (two 32 x 32 products by g vectors on one SM, 2300 g cycles
// each in FP64, and a barrier), or for many right-hand sides the FP64 pipes of the SMs in use;
// solve_shape trades the two; in FP32 the latency of a step's loads, which prefetch_rows brings
// into L2 a step ahead.  With the diagonal blocks solved by substitution and always eight
// vectors on up to 8 CTAs -> now, on a GB300: FP64 order 200, 2 vectors 215 -> 65 us; five of
// 1000, 7 vectors 1.78 -> 0.52 ms; 2999, 9 vectors 10.9 -> 1.7 ms; FP32 four of 8000, 4 vectors
// 11.0 -> 2.3 ms.  lu_finish_kernel adds 45 us at order 200, 70 us at 2999.
constexpr int kSG = 8;
constexpr int kSolveThreads = 512;
constexpr int kSolveMaxCtas = 16;
constexpr int kSolveMaxSmem = 220 * 1024;
constexpr int kBlkLd = kNB + 1;

// kind of block step s and its block index.  KIND 0: unit lower L; 1: upper U; 2: lower U^H; 3:
// unit upper L^H.
template <bool ADJ> __device__ __forceinline__ void solve_step(int s, int nblk, int& kind, int& bI) {
  if (s < nblk) { kind = ADJ ? 2 : 0; bI = s; }
  else { kind = ADJ ? 3 : 1; bI = 2 * nblk - 1 - s; }
}

// rows of block b2 take the contribution of block bI at this step?
__device__ __forceinline__ bool step_updates(int kind, int bI, int b2) {
  return (kind == 0 || kind == 2) ? (b2 > bI) : (b2 < bI);
}

// entry (i, j) of the triangular factor of this kind, off its diagonal blocks
template <typename C>
__device__ __forceinline__ C factor_entry(const C* __restrict__ LU, int64_t n, int kind, int64_t i, int64_t j) {
  return kind >= 2 ? cconj(__ldg(LU + j + i * n)) : __ldg(LU + i + j * n);
}

// entry (r, c) of what stands in diagonal block jb (bw x bw) of this kind: the inverse, or the
// block itself where it was left
template <typename C>
__device__ __forceinline__ C inverse_entry(const C* __restrict__ LU, int64_t n, int kind, int64_t jb, int bw, int r,
                                           int c) {
  C v = czero<C>();
  if (r >= bw || c >= bw) return v;
  const bool unit = kind == 0 || kind == 3, low = kind == 0 || kind == 2;
  if (unit && r == c) { v.x = 1; return v; }
  if (low ? c > r : c < r) return v;
  return factor_entry(LU, n, kind, jb + r, jb + c);
}

// sum over the lanes that share a row of an RW-row group (lanes RW apart)
template <int RW, typename C> __device__ __forceinline__ C row_sum(C v) {
#pragma unroll
  for (int off = 16; off >= RW; off >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, off);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, off);
  }
  return v;
}

// x_i -= M(i, block bI) x_s for the local rows that step (kind, bI) updates, skipping local block
// `skip`: a warp takes RW rows, its 32 / RW lanes per row every (32 / RW)-th column
template <int RW, typename C>
__device__ __forceinline__ void solve_update_rows(const C* __restrict__ LU, int64_t n, int kind, int bI, int P, int rank,
                                                  int g, int ln, C* xl, const C* xs, int nloc, int skip) {
  constexpr int CG = 32 / RW, NC = 32 / CG;  // lanes per row, columns per lane
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t jb = (int64_t)bI * 32;
  const int bw = (int)((jb + 32 < n) ? 32 : n - jb);
  const int cg = lane / RW;
  for (int li0 = warp * RW; li0 < nloc; li0 += (kSolveThreads / 32) * RW) {
    const int lb = li0 >> 5, b2 = rank + lb * P;
    if (lb == skip || !step_updates(kind, bI, b2)) continue;
    const int li = li0 + (lane & (RW - 1));
    const int64_t i = (int64_t)b2 * 32 + (li & 31);
    C mrow[NC];
#pragma unroll
    for (int t = 0; t < NC; ++t) {
      const int c = cg + CG * t;
      mrow[t] = (i < n && c < bw) ? factor_entry(LU, n, kind, i, jb + c) : czero<C>();
    }
    for (int q = 0; q < g; ++q) {
      C acc = czero<C>();
#pragma unroll
      for (int t = 0; t < NC; ++t) acc = cfma(acc, mrow[t], xs[q * kBlkLd + cg + CG * t]);
      acc = row_sum<RW>(acc);
      if (cg == 0) xl[(int64_t)q * ln + li] = csub(xl[(int64_t)q * ln + li], acc);
    }
  }
}

// this CTA's rows of the factor's block column bI (the operand of the update of its step) into L2:
// a step's loads are short of one another's latency, so they should not wait for HBM
template <typename C>
__device__ __forceinline__ void prefetch_rows(const C* __restrict__ LU, int64_t n, int kind, int bI, int P, int rank,
                                              int nlb) {
  constexpr int lines = 32 * (int)sizeof(C) / 128;  // 128-byte lines of 32 entries
  const int64_t jb = (int64_t)bI * 32;
  for (int e = threadIdx.x; e < nlb * 32 * lines; e += kSolveThreads) {
    const int part = e % lines, c = (e / lines) & 31, b2 = rank + e / (32 * lines) * P;
    if (!step_updates(kind, bI, b2)) continue;
    const int64_t i = (int64_t)b2 * 32;
    // the line's entries run along the rows (L, U) or along the columns (their adjoints)
    const int64_t off = part * (128 / (int)sizeof(C));
    const int64_t row = kind >= 2 ? jb + off : i + off, col = kind >= 2 ? i + c : jb + c;
    if (row < n && col < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(LU + row + col * n));
  }
}

// out[r] = sum_c blk[r][c] x[c] for row r = 8 warp + (lane & 7) of a 32 x 32 block, on every lane
// of the row (warps 0 to 3)
template <typename C>
__device__ __forceinline__ C block_times(const C* blk, const C* x) {
  const int lane = threadIdx.x & 31, r = (threadIdx.x >> 5) * 8 + (lane & 7), cg = lane >> 3;
  C a0 = czero<C>(), a1 = czero<C>();
#pragma unroll
  for (int t = 0; t < 8; t += 2) {
    a0 = cfma(a0, blk[r * kBlkLd + cg + 4 * t], x[cg + 4 * t]);
    a1 = cfma(a1, blk[r * kBlkLd + cg + 4 * t + 4], x[cg + 4 * t + 4]);
  }
  return row_sum<8>(cadd(a0, a1));
}

template <typename T> constexpr size_t solve_smem_bytes(int group, int ln) {
  return 2 * sizeof(T) * ((size_t)group * ln + 4 * kNB * kBlkLd + 4 * (size_t)group * kBlkLd);
}

template <typename T, bool ADJ>
__global__ void __launch_bounds__(kSolveThreads, 2) solve_cluster_kernel(BatchDesc d, const typename cplx_t<T>::type* __restrict__ LUall,
                                                                     const int32_t* __restrict__ sigma_all,
                                                                     typename cplx_t<T>::type* __restrict__ Xall,
                                                                     int64_t nrhs, int64_t xstride, int group, int ln,
                                                                     int upper_only) {
  using C = typename cplx_t<T>::type;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char solve_smem[];
  __shared__ int kept[2];                        // flag words of the staged diagonal blocks
  C* xl = reinterpret_cast<C*>(solve_smem);      // group x ln, vector-major
  C* blk = xl + (int64_t)group * ln;             // [2][M(next, current), inverse(next)] 32 x kBlkLd
  C* slots = blk + 4 * kNB * kBlkLd;             // [3] group x kBlkLd: solved blocks
  C* rb = slots + 3 * group * kBlkLd;            // group x kBlkLd: the next block's right-hand sides
  const int P = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int64_t n = d.order(blockIdx.z);
  const int nblk = (int)((n + 31) / 32);
  const C* LU = LUall + d.offset(blockIdx.z);
  const int32_t* sig = sigma_all + blockIdx.z * ipiv_stride(d.n);
  const int32_t* flags = sig + d.n;
  C* X = Xall + d.xoffset(blockIdx.z, xstride);
  const int64_t r0 = blockIdx.y * (int64_t)group;
  const int g = (int)((r0 + group <= nrhs) ? group : nrhs - r0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nlb = (nblk - rank + P - 1) / P;  // blocks of this CTA (may be 0)
  const int nloc = nlb > 0 ? nlb * 32 : 0;
  for (int w = tid; w < nloc * g; w += kSolveThreads) {
    const int li = w % nloc, q = w / nloc;
    const int64_t i = (int64_t)(rank + (li >> 5) * P) * 32 + (li & 31);
    C v = czero<C>();
    if (i < n) v = X[((ADJ || upper_only) ? i : (int64_t)sig[i]) + (r0 + q) * n];
    xl[(int64_t)q * ln + li] = v;
  }
  const int nsteps = 2 * nblk;
  const int s0 = upper_only ? nblk : 0;  // upper_only: the U steps alone
  constexpr int kPer = kNB * kNB / kSolveThreads;  // entries of a block per thread
  // the operands of step s into registers / from registers into buffer s & 1
  auto fetch = [&](int s, C (&va)[kPer], C (&vi)[kPer]) {
    int kind, bI, pkind, pI;
    solve_step<ADJ>(s, nblk, kind, bI);
    if (tid == 0) kept[s & 1] = flags[bI];
    solve_step<ADJ>(s - 1, nblk, pkind, pI);
    const int64_t jb = (int64_t)bI * 32, jp = (int64_t)pI * 32;
    const int bw = (int)((jb + 32 < n) ? 32 : n - jb), pw = (int)((jp + 32 < n) ? 32 : n - jp);
    const bool upd = s > s0 && step_updates(pkind, pI, bI);
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      // consecutive threads along the memory-contiguous direction of this kind
      const int x = (tid + e * kSolveThreads) & 31, y = (tid + e * kSolveThreads) >> 5;
      const int r = kind >= 2 ? y : x, c = kind >= 2 ? x : y;
      va[e] = (upd && r < bw && c < pw) ? factor_entry(LU, n, pkind, jb + r, jp + c) : czero<C>();
      vi[e] = inverse_entry(LU, n, kind, jb, bw, r, c);
    }
  };
  auto stash = [&](int s, const C (&va)[kPer], const C (&vi)[kPer]) {
    int kind, bI;
    solve_step<ADJ>(s, nblk, kind, bI);
    C* b = blk + (s & 1) * 2 * kNB * kBlkLd;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const int x = (tid + e * kSolveThreads) & 31, y = (tid + e * kSolveThreads) >> 5;
      const int r = kind >= 2 ? y : x, c = kind >= 2 ? x : y;
      b[r * kBlkLd + c] = va[e];
      b[kNB * kBlkLd + r * kBlkLd + c] = vi[e];
    }
  };
  auto owner = [&](int s) {
    int kind, bI;
    solve_step<ADJ>(s, nblk, kind, bI);
    return bI % P;
  };
  // warps 0 to 3 of the owner of step s: x_s = inverse (b_s - M x_(s-1)), pushed to every CTA
  auto solve_block = [&](int s) {
    int kind, bI;
    solve_step<ADJ>(s, nblk, kind, bI);
    const C* b = blk + (s & 1) * 2 * kNB * kBlkLd;
    const C* xp = slots + ((s + 2) % 3) * group * kBlkLd;  // x_(s-1)
    const int r = warp * 8 + (lane & 7), cgi = lane >> 3;
    C* xb = xl + (bI / P) * 32 + r;
    for (int q = 0; q < g; ++q) {
      C v = xb[(int64_t)q * ln];
      if (s > s0) v = csub(v, block_times(b, xp + q * kBlkLd));
      if (cgi == 0) rb[q * kBlkLd + r] = v;
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (kept[s & 1] & ((kind == 0 || kind == 3) ? 1 : 2)) {
      // this block was left as it is: substitution, one warp per vector, then the push
      const C* m = b + kNB * kBlkLd;
      const bool low = kind == 0 || kind == 2;
      for (int q = warp; q < g; q += 4) {
        const int bw = (int)((int64_t)bI * 32 + 32 < n ? 32 : n - (int64_t)bI * 32);
        C x = rb[q * kBlkLd + lane];
        C rdl = czero<C>();
        if (lane < bw) rdl = crecip(m[lane * kBlkLd + lane]);
        for (int e = 0; e < bw; ++e) {
          const int c = low ? e : bw - 1 - e;
          if (lane == c) x = cmul(x, rdl);
          const C xc = shfl_c(x, c);
          if (low ? lane > c : lane < c) x = cfms(x, m[lane * kBlkLd + c], xc);
        }
        if (lane >= bw) x = czero<C>();
        xl[(int64_t)q * ln + (bI / P) * 32 + lane] = x;
        C* slot = slots + (s % 3) * group * kBlkLd + q * kBlkLd + lane;
        for (int t = 0; t < P; ++t) *cl.map_shared_rank(slot, (unsigned)t) = x;
      }
      return;
    }
    for (int q = 0; q < g; ++q) {
      const C v = block_times(b + kNB * kBlkLd, rb + q * kBlkLd);
      if (cgi == 0) xb[(int64_t)q * ln] = v;
      C* slot = slots + (s % 3) * group * kBlkLd + q * kBlkLd + r;
      for (int t = cgi; t < P; t += 4) *cl.map_shared_rank(slot, (unsigned)t) = v;
    }
  };
  C va[kPer], vi[kPer];
  cluster_arrive();  // every CTA of the cluster runs before the first push
  for (int s = s0; s < s0 + 2 && s < nsteps; ++s)
    if (owner(s) == rank) {
      fetch(s, va, vi);
      stash(s, va, vi);
    }
  cluster_wait();
  __syncthreads();
  if (owner(s0) == rank && warp < 4) solve_block(s0);
  cluster_arrive();
  cluster_wait();
  for (int s = s0; s < nsteps; ++s) {
    int kind, bI, skip = -1;
    solve_step<ADJ>(s, nblk, kind, bI);
    const bool last = s + 1 == nsteps;
    if (!last && owner(s + 1) == rank) {
      int nkind, nbI;
      solve_step<ADJ>(s + 1, nblk, nkind, nbI);
      skip = nbI / P;
      if (warp < 4) solve_block(s + 1);
    }
    if (!last) cluster_arrive();  // x_(s+1) pushed
    const bool ahead = s + 2 < nsteps && owner(s + 2) == rank;
    if (ahead) fetch(s + 2, va, vi);
    if (!last) {
      int nkind, nbI;
      solve_step<ADJ>(s + 1, nblk, nkind, nbI);
      prefetch_rows<C>(LU, n, nkind, nbI, P, rank, nlb);
    }
    const C* xs = slots + (s % 3) * group * kBlkLd;
    solve_update_rows<8, C>(LU, n, kind, bI, P, rank, g, ln, xl, xs, nloc, skip);
    if (ahead) stash(s + 2, va, vi);
    __syncthreads();
    if (!last) cluster_wait();
  }
  for (int w = tid; w < nloc * g; w += kSolveThreads) {
    const int li = w % nloc, q = w / nloc;
    const int64_t i = (int64_t)(rank + (li >> 5) * P) * 32 + (li & 31);
    if (i < n) X[(ADJ ? (int64_t)sig[i] : i) + (r0 + q) * n] = xl[(int64_t)q * ln + li];
  }
}

// ------------------------------ Y = A X (FP64) --------------------------------
constexpr int kGemvRows = 32;     // outputs per CTA, one per lane
constexpr int kGemvWarps = 8;     // each takes 8 of the kGemvCols terms of a step
constexpr int kGemvCols = 8 * kGemvWarps;
constexpr int kGemvNR = 8;
constexpr int kGemvLd = 9;
constexpr int kGemvMaxCtas = 4 * 152;

// partial[js][b][r][i] = sum_{j in chunk js} A_b[i, j] X_b[j, r]  (ADJ: A^H).  A CTA computes 32
// outputs: per step of 64 terms each warp has its eight matrix entries per output in flight at
// once (ADJ: read along the columns, 128 bytes at a time, and turned in shared memory), and the
// warps' sums are added at the end.  Bound: the FP64 pipe for several right-hand sides, latency for
// few (one warp instruction per 19 cycles and SM, 77 for a single warp).  A thread per output
// that loaded one entry at a time, down a column for A^H, took 568 us for order 1400 (A^H, four
// matrices for A 574), 93 us at 450 and 79 us at 200; now 151 (131), 11 and 9.
template <bool ADJ>
__global__ void __launch_bounds__(32 * kGemvWarps) zgemm_partial_kernel(BatchDesc d, const double2* __restrict__ Aall,
                                                                       const double2* __restrict__ Xall, int64_t nrhs,
                                                                       int64_t xstride, int64_t jchunk, int r0,
                                                                       double2* __restrict__ part) {
  __shared__ double2 sX[kGemvNR][kGemvCols];
  __shared__ double2 sT[kGemvWarps][32 * kGemvLd];  // ADJ: entries [output][term]; at the end the warps' sums
  const int64_t n = d.n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = blockIdx.x * (int64_t)kGemvRows, i = i0 + lane;
  const int64_t js = blockIdx.y;
  const int64_t b = blockIdx.z;
  const double2* A = Aall + b * d.stride;
  const double2* X = Xall + b * xstride;
  const int64_t ja = js * jchunk, jbnd = (ja + jchunk < n) ? ja + jchunk : n;
  const int g = (int)((r0 + kGemvNR <= nrhs) ? kGemvNR : nrhs - r0);
  double2 acc[kGemvNR];
#pragma unroll
  for (int r = 0; r < kGemvNR; ++r) acc[r] = make_double2(0.0, 0.0);
  double2* tile = sT[warp];
  for (int64_t jb = ja; jb < jbnd; jb += kGemvCols) {
    const int64_t j0 = jb + 8 * warp;
    double2 a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int64_t jj = ADJ ? j0 + (lane & 7) : j0 + q, ii = ADJ ? i0 + (lane >> 3) + 4 * q : i;
      a[q] = (jj < jbnd && ii < n) ? __ldg(ADJ ? A + jj + ii * n : A + ii + jj * n) : make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < g * kGemvCols; e += 32 * kGemvWarps) {
      const int r = e / kGemvCols, c = e & (kGemvCols - 1);
      sX[r][c] = jb + c < jbnd ? X[jb + c + (r0 + r) * n] : make_double2(0.0, 0.0);
    }
    if (ADJ) {
#pragma unroll
      for (int q = 0; q < 8; ++q) tile[((lane >> 3) + 4 * q) * kGemvLd + (lane & 7)] = cconj(a[q]);
    }
    __syncthreads();
    if (ADJ) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = tile[lane * kGemvLd + q];
    }
    if (j0 < jbnd) {
#pragma unroll
      for (int r = 0; r < kGemvNR; ++r)
        if (r < g) {
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[r] = cfma(acc[r], a[q], sX[r][8 * warp + q]);
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kGemvNR; ++r)
    if (r < g) tile[r * 32 + lane] = acc[r];
  __syncthreads();
  if (warp < g && i < n) {
    double2 s = sT[0][warp * 32 + lane];
#pragma unroll
    for (int w = 1; w < kGemvWarps; ++w) s = cadd(s, sT[w][warp * 32 + lane]);
    part[((js * d.batch + b) * nrhs + r0 + warp) * n + i] = s;
  }
}

__global__ void zgemm_reduce_kernel(BatchDesc d, int64_t nrhs, int64_t nsplit, const double2* __restrict__ part,
                                    double2* __restrict__ Yall, int64_t ystride, const double2* __restrict__ Ball,
                                    int subtract_from_b) {
  const int64_t n = d.n;
  const int64_t per = nrhs * n;
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= per * d.batch) return;
  const int64_t b = q / per, e = q % per;
  double2 s = make_double2(0.0, 0.0);
  for (int64_t js = 0; js < nsplit; ++js) {
    double2 v = part[(js * d.batch + b) * per + e];
    s.x += v.x;
    s.y += v.y;
  }
  if (subtract_from_b) {
    double2 bb = Ball[b * ystride + e];
    s = make_double2(bb.x - s.x, bb.y - s.y);
  }
  Yall[b * ystride + e] = s;
}

// Splits of the sum: four CTAs per SM, each with at least half a step of terms
int64_t gemm_split(int64_t n, int64_t batch) {
  const int64_t rows = (n + kGemvRows - 1) / kGemvRows;
  const int64_t want = kGemvMaxCtas / (rows * batch), most = (n + kGemvCols / 2 - 1) / (kGemvCols / 2);
  return std::max<int64_t>(1, std::min(want, most));
}

__global__ void z_to_c_kernel(const double2* __restrict__ s, float2* __restrict__ d, int64_t count) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < count) d[q] = make_float2((float)s[q].x, (float)s[q].y);
}

__global__ void c_to_z_kernel(const float2* __restrict__ s, double2* __restrict__ d, int64_t count) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < count) d[q] = make_double2((double)s[q].x, (double)s[q].y);
}

__global__ void ir_update_kernel(double2* __restrict__ X, const float2* __restrict__ Cc, int64_t count) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < count) { X[q].x += (double)Cc[q].x; X[q].y += (double)Cc[q].y; }
}

// out[col] = max_i |re| + |im| over column col of R, and out[ncols + col] of X (blockIdx.y 0, 1):
// columns of n entries, nrhs per matrix, the matrices' xstride apart.  All columns in one launch:
// two per matrix, 4.4 us each, were a tenth of a 12-frequency sweep of 430 panels.
__global__ void col_inf_norm_kernel(int64_t n, int64_t nrhs, int64_t xstride, const double2* __restrict__ R,
                                    const double2* __restrict__ Xs, double* __restrict__ out) {
  const int64_t col = blockIdx.x + blockIdx.y * (int64_t)gridDim.x;
  const double2* X = (blockIdx.y ? Xs : R) + blockIdx.x / nrhs * xstride + blockIdx.x % nrhs * n;
  double m = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    double2 v = X[i];
    double a = fabs(v.x) + fabs(v.y);
    m = a > m ? a : m;
  }
  __shared__ double red[8];
  for (int off = 16; off > 0; off >>= 1) { double o = __shfl_down_sync(0xffffffffu, m, off); m = o > m ? o : m; }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = red[w] > r ? red[w] : r;
    out[col] = r;
  }
}


// the FP32 copy of matrix b (column stride n, matrix stride stride32; a grouped batch: at the
// matrix's own element offset) and, in the same pass
// over A, out[b] = max_i sum_j |re|+|im| (|.|_inf, order independent via atomicMax on the bits
// of a non-negative double; out zeroed first).  128 rows x 8 column slices per CTA, the
// slices' partial row sums added in a fixed order.
__global__ void __launch_bounds__(1024) convert_norm_kernel(BatchDesc d, const double2* __restrict__ A,
                                                            float2* __restrict__ A32, int64_t stride32,
                                                            unsigned long long* __restrict__ out) {
  __shared__ double part[8][128];
  const int64_t i = blockIdx.x * (int64_t)128 + threadIdx.x;
  const int64_t b = blockIdx.y;
  // a grouped batch: the FP32 copies sit at the same element offsets as the matrices
  const int64_t n = d.order(b);
  const double2* Ab = A + d.offset(b);
  float2* Cb = A32 + (d.offsets ? d.offsets[b] : b * stride32);
  const int64_t j0 = (n * threadIdx.y) / 8, j1 = (n * (threadIdx.y + 1)) / 8;
  double s = 0.0;
  if (i < n) {
#pragma unroll 4
    for (int64_t j = j0; j < j1; ++j) {
      const double2 v = Ab[i + j * n];
      Cb[i + j * n] = make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
      s += fabs(v.x) + fabs(v.y);
    }
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && i < n) {
    double t = 0.0;
    for (int y = 0; y < 8; ++y) t += part[y][threadIdx.x];
    atomicMax(out + b, (unsigned long long)__double_as_longlong(t));
  }
}

}  // namespace

void convert_with_norms(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, float2* A32,
                        int64_t stride32, double* out) {
  cudaMemsetAsync(out, 0, sizeof(double) * d.batch, st);
  dim3 grid((unsigned)((d.n + 127) / 128), (unsigned)d.batch);
  MH_LAUNCH(lc, st, "convert", convert_norm_kernel<<<grid, dim3(128, 8), 0, st>>>(d, A, A32, stride32,
                                                                                (unsigned long long*)out));
}


int sm_count() {
  static PerDevice<int> counts;
  const int dev = current_device();
  return counts.get(dev, [dev] {
    int v = 152;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  });
}

// Clusters of p CTAs of the panel kernel resident on the GPU at once, by p (clusters are placed
// within one GPC, so this is the occupancy query's answer, not the SM count's); `width` 32 at the
// largest chunk (a full-width panel fills one SM's shared memory), 16 half of it.  The first call on
// a device also sets the kernel's attributes there.
template <typename T>
const int* panel_residency(int width) {
  struct Table { int resident[kPanelMaxCtas + 1]; };
  auto make_table = [](int w) {
    Table t{};
    // the attribute always allows the full-width panel; the query uses this width's size
    int most = 0;
    for (int p = 1; p <= kPanelMaxCtas; ++p) most = std::max(most, (int)panel_smem_bytes<T>(panel_rows<T>(p), kNB, p));
    cudaFuncSetAttribute(panel_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    cudaFuncSetAttribute(panel_cluster_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int p = 1; p <= kPanelMaxCtas; ++p) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)p, 1, 1);
      cfg.blockDim = dim3(kPanelThreads, 1, 1);
      cfg.dynamicSmemBytes = panel_smem_bytes<T>(panel_rows<T>(p), w, p);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)p;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int num = 0;
      if (cudaOccupancyMaxActiveClusters(&num, panel_cluster_kernel<T>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        num = 0;
      }
      t.resident[p] = num;
    }
    return t;
  };
  static PerDevice<Table> full, half;
  return (width < kNB ? half : full).get(current_device(), [&] { return make_table(width < kNB ? kNB / 2 : kNB); }).resident;
}

// the fewest CTAs whose shared memory holds a panel of m rows (0: no cluster does)
template <typename T>
int panel_least_ctas(int64_t m) {
  for (int p = 1; p <= kPanelMaxCtas; ++p)
    if (m <= (int64_t)p * panel_rows<T>(p)) return p;
  return 0;
}

// CTAs per cluster for a panel of m rows in a batch of `batch` matrices: enough to hold the
// panel in shared memory, and more while all `batch` clusters still fit on the GPU at once,
// every CTA has an SM of its own (the panel is FP64-bound per SM) and rows of its own (32 or
// more), up to `cap_ctas` beyond the minimum (the launch-shape table's cluster bound; its
// largest value, 8, stands for the largest cluster of 16); 0 when the panel does not fit the
// largest cluster the GPU can schedule (panel_kernel then runs).
// (resident: panel_residency of the panel's width; sms: of the device.)
template <typename T>
int panel_cluster_size(int64_t m, int64_t batch, int cap_ctas, const int* resident, int sms) {
  const int need = panel_least_ctas<T>(m);
  if (need == 0 || resident[need] <= 0) return 0;
  const int most = cap_ctas >= 8 ? kPanelMaxCtas : cap_ctas;
  int p = need;
  for (int q = need + 1; q <= most; ++q) {
    const int chunk = panel_chunk(m, q, panel_rows<T>(q));
    if ((m + chunk - 1) / chunk != q) continue;  // a CTA would be without rows
    if (resident[q] >= batch && q * batch <= sms) p = q;
  }
  return p;
}

// true when the full-width panel of m rows runs its clusters for all `batch` matrices at once
// (its rows need at most as many CTAs per matrix as fit every cluster on the GPU); a panel that
// does not fit runs in waves, and the FP64 tensor-core path factors it in two halves instead
template <typename T>
bool panel_fits_one_wave(int64_t m, int64_t batch, const int* resident) {
  const int need = panel_least_ctas<T>(m);
  return need > 0 && resident[need] >= batch;
}

template <typename T>
int lu_factor_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, typename cplx_t<T>::type* A,
                      int32_t* ipiv, int32_t* info, void* emu_ws, int* emu_flag) {
  const int64_t n = d.n;
  if (n <= 0 || d.batch <= 0) return 0;
  // appended right-hand sides need the rectangular trailing update of the FP64 tensor-core path;
  // the FP32 update has no other path than the tensor cores'
  if (d.extra > 0 && (sizeof(T) != 8 || !emu_ws || d.orders)) return -1;
  if (sizeof(T) == 4 && !emu_ws) return -1;
  cudaMemsetAsync(info, 0, sizeof(int32_t) * d.batch, st);
  const int sms = sm_count();
  const int *resident = panel_residency<T>(kNB), *resident_half = panel_residency<T>(kNB / 2);
  const int cap_ctas = sizeof(T) == 8 ? lc.tile(n).cluster_f64 : lc.tile(n).cluster_f32;
  // the panel at k0 of `width` columns on a cluster of P CTAs
  auto cluster_panel = [&](int64_t k0, int width, int P) {
    const int chunk = panel_chunk(n - k0, P, panel_rows<T>(P));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P, (unsigned)d.batch, 1);
    cfg.blockDim = dim3(kPanelThreads, 1, 1);
    cfg.dynamicSmemBytes = panel_smem_bytes<T>(chunk, width, P);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MH_LAUNCH(lc, st, sizeof(T) == 8 ? "lu_panel_f64" : "lu_panel_f32",
              cudaLaunchKernelEx(&cfg, panel_cluster_kernel<T>, d, A, ipiv, info, k0, chunk, width));
  };
  // the full-width panel at k0 (on one CTA per matrix when no cluster holds it), and its row
  // interchanges outside of it
  auto full_panel = [&](int64_t k0) {
    const int P = panel_cluster_size<T>(n - k0, d.batch, cap_ctas, resident, sms);
    if (P > 0) {
      cluster_panel(k0, kNB, P);
    } else {
      MH_LAUNCH(lc, st, sizeof(T) == 8 ? "lu_panel_f64" : "lu_panel_f32",
                panel_kernel<T><<<(unsigned)d.batch, 512, 0, st>>>(d, A, ipiv, info, k0));
    }
  };
  auto interchange = [&](int64_t k0, int64_t kb) {
    if (n + d.extra - kb <= 0) return;
    dim3 sg((unsigned)((n + d.extra - kb + kSwpCols - 1) / kSwpCols), (unsigned)d.batch);
    MH_LAUNCH(lc, st, sizeof(T) == 8 ? "lu_laswp_f64" : "lu_laswp_f32",
              laswp_kernel<T><<<sg, 256, 0, st>>>(d, A, ipiv, k0, (int)kb));
  };
  for (int64_t k = 0; k < n; k += kNB) {
    const int64_t kb = (k + kNB < n) ? kNB : n - k;
    if constexpr (sizeof(T) == 4) {
      // two panels per pass over the trailing block: the first panel's update reaches only the
      // second's columns, and both together the rest
      if (emu_ws && bx3_deep(d, n - k - 2 * kNB)) {
        full_panel(k);
        interchange(k, kNB);
        MH_LAUNCH(lc, st, "lu_trsm_f32",
                  trsm_kernel<T><<<dim3((unsigned)((n - k - kNB + 127) / 128), (unsigned)d.batch), 128, 0, st>>>(d, A, k));
        bx3_trailing_update(st, lc, d, A, k, kNB, kNB, emu_ws, emu_flag);
        full_panel(k + kNB);
        interchange(k + kNB, kNB);
        MH_LAUNCH(lc, st, "lu_trsm_f32",
                  trsm_second_kernel<<<dim3((unsigned)((n - k - 2 * kNB + 127) / 128), (unsigned)d.batch), 128, 0, st>>>(
                      d, A, k));
        bx3_trailing_update(st, lc, d, A, k, 2 * kNB, INT64_MAX, emu_ws, emu_flag);
        k += kNB;
        continue;
      }
    }
    // Two-level panel (FP64 with the tensor-core update, tall panels): two 16-column halves
    // on the CUDA cores, the left half's update of the right half (K = 16) on the tensor
    // cores -- half the panel's FP64 work, and half its shared memory per row
    int Pl = 0, P16 = 0;
    if constexpr (sizeof(T) == 8) {
      if (emu_ws && kb == kNB && !d.orders && !panel_fits_one_wave<T>(n - k, d.batch, resident)) {
        Pl = panel_cluster_size<T>(n - k, d.batch, cap_ctas, resident_half, sms);
        P16 = panel_cluster_size<T>(n - k - kNB / 2, d.batch, cap_ctas, resident_half, sms);
      }
    }
    if (Pl > 0 && P16 > 0) {
      if constexpr (sizeof(T) == 8) {
        const int H = kNB / 2;
        cluster_panel(k, H, Pl);
        dim3 sg(1u, (unsigned)d.batch);
        MH_LAUNCH(lc, st, "lu_laswp_f64", laswp_cols_kernel<T><<<sg, 256, 0, st>>>(d, A, ipiv, k, H, k + H, k + kNB));
        MH_LAUNCH(lc, st, "lu_trsm16_f64", trsm16_kernel<T><<<(unsigned)d.batch, 256, 0, st>>>(d, A, k));
        ozaki_trailing_update(st, lc, d, A, k, H, emu_ws, emu_flag, H);
        cluster_panel(k + H, H, P16);
        MH_LAUNCH(lc, st, "lu_laswp_f64", laswp_cols_kernel<T><<<sg, 256, 0, st>>>(d, A, ipiv, k + H, H, k, k + H));
      }
    } else {
      full_panel(k);
    }
    interchange(k, kb);
    const int64_t rest = n - k - kb;              // trailing rows
    const int64_t rest_c = n + d.extra - k - kb;  // columns right of the panel
    if (rest_c <= 0) continue;
    bool trsm_done = false;
    if constexpr (sizeof(T) == 8) {  // FP64 with the tensor-core update: U12 on the tensor cores too
      if (emu_ws && kb == kNB) {
        ozaki_trsm(st, lc, d, A, k, emu_ws, emu_flag);
        trsm_done = true;
      }
    }
    if (!trsm_done) {
      if constexpr (sizeof(T) == 8) {
        const bool few = rest_c * d.batch <= kTrsmFewColumns;
        const int64_t cols = kTrsmThreads / (few ? 32 : 8);
        dim3 tg((unsigned)((rest_c + cols - 1) / cols), (unsigned)d.batch);
        if (few) MH_LAUNCH(lc, st, "lu_trsm_f64", trsm_lanes_kernel<32><<<tg, kTrsmThreads, 0, st>>>(d, A, k));
        else MH_LAUNCH(lc, st, "lu_trsm_f64", trsm_lanes_kernel<8><<<tg, kTrsmThreads, 0, st>>>(d, A, k));
      } else {
        dim3 tg((unsigned)((rest_c + 127) / 128), (unsigned)d.batch);
        MH_LAUNCH(lc, st, "lu_trsm_f32", trsm_kernel<T><<<tg, 128, 0, st>>>(d, A, k));
      }
    }
    if (rest <= 0) continue;
    if (emu_ws) {
      if constexpr (sizeof(T) == 8) {  // FP64 update on the BF16 tensor cores (mh_ozaki.cu)
        ozaki_trailing_update(st, lc, d, A, k, (int)kb, emu_ws, emu_flag);
      } else {  // FP32 update on the BF16 tensor cores (mh_bf16x3.cu)
        bx3_trailing_update(st, lc, d, A, k, (int)kb, INT64_MAX, emu_ws, emu_flag);
      }
      continue;
    }
    if constexpr (sizeof(T) == 8) {  // FP64: three real products per complex multiply-add
      const int64_t t2 = (rest + 31) / 32, t1 = (rest + 15) / 16;
      const bool wide = t2 * t2 * d.batch >= 8 * 152;
      dim3 gg((unsigned)(wide ? t2 : t1), (unsigned)(wide ? t2 : t1), (unsigned)d.batch);
      if (wide) MH_LAUNCH(lc, st, "lu_gemm_f64", gemm3m_kernel<2><<<gg, 256, 0, st>>>(d, A, k));
      else MH_LAUNCH(lc, st, "lu_gemm_f64", gemm3m_kernel<1><<<gg, 256, 0, st>>>(d, A, k));
    }
  }
  const int nblk = (int)((n + kNB - 1) / kNB);
  const size_t fsmem = 2 * sizeof(int) * (size_t)n;
  cudaFuncSetAttribute(lu_finish_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinishMaxSmem);
  MH_LAUNCH(lc, st, sizeof(T) == 8 ? "lu_finish_f64" : "lu_finish_f32",
            lu_finish_kernel<T><<<dim3((unsigned)(nblk + 1), (unsigned)d.batch), kFinishThreads, fsmem, st>>>(
                d, A, ipiv, nblk));
  return 0;
}

// The solve's shape: CTAs per cluster and right-hand sides per cluster, by an estimate of its
// time in SM cycles.  A step's chain is two 32 x 32 products by the g vectors on one SM (2300 g
// cycles each on the FP64 pipes; latency in FP32) and a cluster barrier; its bulk the update of
// half the rows, by the cluster's SMs.  More CTAs shorten the bulk, fewer vectors per cluster
// both, as long as the clusters stay resident and have SMs of their own.  The constants are
// measured phase times; the shape that they pick against the fastest of 42 (P of 1 to 16, g of 1 to
// 8), us: FP64 order 200, 2 vectors 64 (57 at P 6 g 1; the slowest 188), 2999, 9 vectors 1701 (1916 P 16
// g 1; 34 ms), 1000, 40 vectors 618 (614 P 6 g 1; 10.7 ms), five of 1000, 7 vectors 516 (504 P 8 g 1; 8.1
// ms), one of 1000 311 (272 P 16 g 1; 8.1 ms); FP32 twelve of 450, 7 vectors 79 (80 P 4 g 3; 229), four of
// 1400 228 (226 P 12 g 2; 1.2 ms), 4500, 4 vectors 748 (748 P 16 g 1; 8.5 ms).
struct SolveShape { int P, g; };
template <typename T>
SolveShape solve_shape(int64_t n, int64_t nrhs, int64_t batch, bool upper_only) {
  struct Table { int one[kSolveMaxCtas + 1]; };
  // clusters of P CTAs resident at once with one CTA per SM; also sets the kernels' attributes on
  // the device
  static PerDevice<Table> tables;
  const Table& tab = tables.get(current_device(), [] {
    Table t{};
    for (const void* fn : {(const void*)solve_cluster_kernel<T, false>, (const void*)solve_cluster_kernel<T, true>}) {
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSolveMaxSmem);
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    for (int p = 1; p <= kSolveMaxCtas; ++p) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)p, 1, 1);
      cfg.blockDim = dim3(kSolveThreads, 1, 1);
      cfg.dynamicSmemBytes = kSolveMaxSmem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = (unsigned)p;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int num = 0;
      if (cudaOccupancyMaxActiveClusters(&num, solve_cluster_kernel<T, false>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        num = 0;
      }
      t.one[p] = num;
    }
    return t;
  });
  const int64_t nblk = (n + 31) / 32;
  const double steps = (double)(upper_only ? nblk : 2 * nblk);
  SolveShape best{0, 0};
  double best_t = 0.0;
  for (int p = 1; p <= kSolveMaxCtas && p <= nblk; ++p) {
    const int ln = (int)((nblk + p - 1) / p * 32);
    for (int g = 1; g <= kSG && g <= nrhs; ++g) {
      const size_t smem = solve_smem_bytes<T>(g, ln);
      if (smem > kSolveMaxSmem || tab.one[p] <= 0) continue;
      const double clusters = (double)((nrhs + g - 1) / g * batch);
      // a second CTA fits an SM when the shared memory does, and shares its pipes
      const int per_sm = smem <= 110 * 1024 ? 2 : 1;
      const double waves = std::ceil(clusters / ((double)tab.one[p] * per_sm));
      const double share = std::min(std::ceil(clusters / (double)tab.one[p]), (double)per_sm);
      const double rows = 0.5 * (double)n / p;
      double chain, bulk;
      if (sizeof(T) == 8) {
        chain = (4600.0 * g + 1000.0) * share;
        bulk = (rows * 32 * g * 2.4 + 4600.0 * g / p + 1000.0) * share;
      } else {
        chain = 1500.0 + 200.0 * g;
        bulk = 1500.0 + rows * 32 * (0.2 + 0.08 * g) * share;
      }
      const double sync = p == 1 ? 0.0 : 800.0 + 50.0 * p;
      const double t = waves * steps * (std::max(chain, bulk) + sync);
      if (best.P == 0 || t < best_t) {
        best = SolveShape{p, g};
        best_t = t;
      }
    }
  }
  return best;
}

template <typename T>
void lu_solve_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const typename cplx_t<T>::type* LU,
                      const int32_t* ipiv, typename cplx_t<T>::type* X, int64_t nrhs, int64_t xstride,
                      bool adjoint, bool upper_only) {
  const int64_t n = d.n;
  if (n <= 0 || nrhs <= 0 || d.batch <= 0) return;
  upper_only = upper_only && !adjoint;
  const SolveShape sh = solve_shape<T>(n, nrhs, d.batch, upper_only);
  const int64_t nblk = (n + 31) / 32;
  const int ln = (int)((nblk + sh.P - 1) / sh.P * 32);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sh.P, (unsigned)((nrhs + sh.g - 1) / sh.g), (unsigned)d.batch);
  cfg.blockDim = dim3(kSolveThreads, 1, 1);
  cfg.dynamicSmemBytes = solve_smem_bytes<T>(sh.g, ln);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)sh.P;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  lc.pre(st);
  if (adjoint) cudaLaunchKernelEx(&cfg, solve_cluster_kernel<T, true>, d, LU, ipiv, X, nrhs, xstride, sh.g, ln, 0);
  else cudaLaunchKernelEx(&cfg, solve_cluster_kernel<T, false>, d, LU, ipiv, X, nrhs, xstride, sh.g, ln, (int)upper_only);
  lc.post(st, sizeof(T) == 8 ? "lu_solve_f64" : "lu_solve_f32");
}

// Random complex matrices (entries uniform in [-1, 1] x [-1, 1] from a counter-based hash)
// on which the autotuner times factorizations; every column needs partial pivoting.
template <typename T>
__global__ void fill_random_kernel(BatchDesc d, typename cplx_t<T>::type* __restrict__ A, uint64_t seed) {
  const int64_t count = d.n * d.n;
  const int64_t b = blockIdx.y;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < count; q += (int64_t)gridDim.x * blockDim.x) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(b * count + q + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const T re = (T)((double)(z >> 40) * (2.0 / 16777216.0) - 1.0);
    const T im = (T)((double)(z & 0xFFFFFFull) * (2.0 / 16777216.0) - 1.0);
    A[b * d.stride + q] = cmk(re, im);
  }
}

template <typename T>
void fill_random_matrices(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, typename cplx_t<T>::type* A,
                          uint64_t seed) {
  if (d.n <= 0 || d.batch <= 0) return;
  const int64_t blocks = std::min<int64_t>((d.n * d.n + 255) / 256, 1216);
  MH_LAUNCH(lc, st, "fill_random",
            fill_random_kernel<T><<<dim3((unsigned)blocks, (unsigned)d.batch), 256, 0, st>>>(d, A, seed));
}
template void fill_random_matrices<double>(cudaStream_t, LaunchCounter, const BatchDesc&, double2*, uint64_t);
template void fill_random_matrices<float>(cudaStream_t, LaunchCounter, const BatchDesc&, float2*, uint64_t);

template int lu_factor_batched<double>(cudaStream_t, LaunchCounter, const BatchDesc&, double2*, int32_t*, int32_t*,
                                       void*, int*);
template int lu_factor_batched<float>(cudaStream_t, LaunchCounter, const BatchDesc&, float2*, int32_t*, int32_t*,
                                      void*, int*);
template void lu_solve_batched<double>(cudaStream_t, LaunchCounter, const BatchDesc&, const double2*,
                                       const int32_t*, double2*, int64_t, int64_t, bool, bool);
template void lu_solve_batched<float>(cudaStream_t, LaunchCounter, const BatchDesc&, const float2*, const int32_t*,
                                      float2*, int64_t, int64_t, bool, bool);

size_t zgemm_work_elems(int64_t n, int64_t nrhs, int64_t batch) {
  // splits x matrices for this many matrices or fewer (gemm_split)
  const int64_t sums = std::max<int64_t>(batch, kGemvMaxCtas / ((n + kGemvRows - 1) / kGemvRows));
  const size_t fp64 = (size_t)sums * (size_t)nrhs * (size_t)n;
  const size_t tc = (tc_zgemv_workspace_bytes(n, batch) + sizeof(double2) - 1) / sizeof(double2);
  return fp64 > tc ? fp64 : tc;
}

void zgemm_nn_tc_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                         int64_t nrhs, int64_t xstride, double2* Y, double2* work, int* timeout_flag) {
  tc_zgemv(st, lc, d, A, X, nrhs, xstride, Y, nullptr, work, timeout_flag);
}

void residual_tc_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                         const double2* B, int64_t nrhs, int64_t xstride, double2* R, double2* work,
                         int* timeout_flag) {
  tc_zgemv(st, lc, d, A, X, nrhs, xstride, R, B, work, timeout_flag);
}

static void zgemm_impl(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                       int64_t nrhs, int64_t xstride, double2* Y, double2* work, const double2* B, bool adjoint) {
  const int64_t n = d.n;
  if (n <= 0 || nrhs <= 0 || d.batch <= 0) return;
  const int64_t ns = gemm_split(n, d.batch);
  const int64_t jchunk = (n + ns - 1) / ns;
  dim3 grid((unsigned)((n + kGemvRows - 1) / kGemvRows), (unsigned)ns, (unsigned)d.batch);
  for (int r0 = 0; r0 < nrhs; r0 += kGemvNR) {
    lc.pre(st);
    if (adjoint) zgemm_partial_kernel<true><<<grid, 32 * kGemvWarps, 0, st>>>(d, A, X, nrhs, xstride, jchunk, r0, work);
    else zgemm_partial_kernel<false><<<grid, 32 * kGemvWarps, 0, st>>>(d, A, X, nrhs, xstride, jchunk, r0, work);
    lc.post(st, "zgemm_rhs");
  }
  const int64_t tot = nrhs * n * d.batch;
  MH_LAUNCH(lc, st, "zgemm_rhs_reduce",
            zgemm_reduce_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(d, nrhs, ns, work, Y, xstride, B,
                                                                                B != nullptr));
}

void zgemm_nn_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                      int64_t nrhs, int64_t xstride, double2* Y, double2* work) {
  zgemm_impl(st, lc, d, A, X, nrhs, xstride, Y, work, nullptr, false);
}

void zgemm_adj_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                       int64_t nrhs, int64_t xstride, double2* Y, double2* work) {
  zgemm_impl(st, lc, d, A, X, nrhs, xstride, Y, work, nullptr, true);
}

void residual_batched(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, const double2* A, const double2* X,
                      const double2* B, int64_t nrhs, int64_t xstride, double2* R, double2* work, bool adjoint) {
  zgemm_impl(st, lc, d, A, X, nrhs, xstride, R, work, B, adjoint);
}

void convert_z_to_c(cudaStream_t st, LaunchCounter lc, const double2* src, float2* dst, int64_t count) {
  if (count <= 0) return;
  MH_LAUNCH(lc, st, "convert", z_to_c_kernel<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(src, dst, count));
}


void ir_update(cudaStream_t st, LaunchCounter lc, int64_t count, double2* X, const float2* Cc) {
  if (count <= 0) return;
  MH_LAUNCH(lc, st, "ir_update", ir_update_kernel<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(X, Cc, count));
}

void widen_c_to_z(cudaStream_t st, LaunchCounter lc, const float2* src, double2* dst, int64_t count) {
  if (count <= 0) return;
  MH_LAUNCH(lc, st, "convert", c_to_z_kernel<<<(unsigned)((count + 255) / 256), 256, 0, st>>>(src, dst, count));
}

void inf_norms_batched(cudaStream_t st, LaunchCounter lc, int64_t n, int64_t batch, int64_t nrhs, int64_t xstride,
                       const double2* R, const double2* X, double* out) {
  if (batch <= 0 || nrhs <= 0) return;
  MH_LAUNCH(lc, st, "ir_norms",
            col_inf_norm_kernel<<<dim3((unsigned)(batch * nrhs), 2), 256, 0, st>>>(n, nrhs, xstride, R, X, out));
}


}  // namespace mh
