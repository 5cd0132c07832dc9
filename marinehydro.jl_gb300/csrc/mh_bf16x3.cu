// mh_bf16x3.cu -- the FP32 complex LU trailing update (the factors of MH_PREC_MIXED) on the
// BF16 tensor cores by three-way splitting.
//
// Every FP32 entry x of L21 and U12 is cut into three BF16 terms, x0 = bf16(x),
// x1 = bf16(x - x0), x2 = bf16(x - x0 - x1) (8 + 8 + 8 significant bits for FP32's 24), and
// A22 -= L21 U12 is accumulated in FP32 tensor memory from the six products x_p y_q with
// p + q <= 2; the three dropped products are 2^-24 of the leading one, the size of FP32
// rounding.  Each product of two BF16 terms is exact in FP32.  These factors only seed the
// FP64 iterative refinement (the FP64 residual decides convergence), so FP32 accuracy is all
// they need; the CUDA-core FP32 update they replace reached ~18 % of the FP32 FMA peak.
//
// Kernels per update (batched over the matrices), of K = 32 KH columns:
//   bx3_split_rows: L21 -> A tiles [row tile][half][re/im][term] of 128 x 32 BF16 (8 KB each, in
//     the canonical no-swizzle K-major layout);
//   bx3_split_cols: U12 -> B tiles [column tile][half][re/im][term] of 128 x 32 BF16;
//   bx3_gemm: one CTA per (128-row tile, group of 128-column tiles, matrix).  The A tiles stay
//     in shared memory; a thread of its own brings the B tiles, half by half, through a ring of
//     two TMA bulk-copied slots and issues 48 tcgen05.mma per half (M = N = 128, K = 16: 6 term
//     pairs x 2 K-steps x 4 real products, the -Im Im product through the negate-A bit) into a
//     Re and an Im FP32 accumulator (256 TMEM columns), double-buffered; the other eight warps
//     subtract finished tiles from A22, always with the next 32 columns' loads in flight.
// Every wait is bounded: on timeout the kernel raises the caller's flag, drains its copies
// and products (bounded) and frees its tensor memory.
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include "mh_internal.cuh"
#include "mh_tc.cuh"

namespace mh {

namespace {

constexpr int kBxTerms = 3;
constexpr int kBxK = 32;                                 // panel width (the LU's kNB)
constexpr int kBxNB = kBxK;
constexpr int kBxTile = 128;                             // rows of an A tile = columns of a B tile
constexpr int kBxPlane = kBxTile * kBxK * 2;             // bytes of one 128 x 32 BF16 plane
constexpr int kBxTileBytes = 2 * kBxTerms * kBxPlane;    // 48 KB: re/im x 3 terms
constexpr int kBxGroupMax = 8;                           // column tiles per CTA: 1..8 from the
                                                         // launch-shape table (default 4)
constexpr int kBxEpilogue = 256;                         // two threads per output row
constexpr int kBxThreads = kBxEpilogue + 32;             // and a warp that copies and issues
constexpr uint32_t kBxTmemCols = 512;                    // 2 buffers x (Re 128 + Im 128)
constexpr uint32_t kBxWaitPolls = 1u << 26;
constexpr double kBxDeepEntries = 8e6;                   // 64 MB of FP32 complex entries

__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&t)[kBxTerms]) {
  t[0] = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(t[0]);
  t[1] = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(t[1]);
  t[2] = __float2bfloat16_rn(r2);
}

// eight consecutive K values of one row of a tile -> six 16-byte chunks (re/im x 3 terms)
__device__ __forceinline__ void store_terms8(unsigned char* tile, int r, int k8, const float2 (&v)[8]) {
  uint32_t pk[2][kBxTerms][4];
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    __nv_bfloat16 a0[kBxTerms], a1[kBxTerms], b0[kBxTerms], b1[kBxTerms];
    split3(v[c].x, a0);
    split3(v[c + 1].x, a1);
    split3(v[c].y, b0);
    split3(v[c + 1].y, b1);
#pragma unroll
    for (int p = 0; p < kBxTerms; ++p) {
      pk[0][p][c >> 1] = (uint32_t)__bfloat16_as_ushort(a0[p]) | ((uint32_t)__bfloat16_as_ushort(a1[p]) << 16);
      pk[1][p][c >> 1] = (uint32_t)__bfloat16_as_ushort(b0[p]) | ((uint32_t)__bfloat16_as_ushort(b1[p]) << 16);
    }
  }
  const uint32_t off = tc::kmajor_offset(r, k8, kBxK);
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int p = 0; p < kBxTerms; ++p)
      *reinterpret_cast<uint4*>(tile + (part * kBxTerms + p) * kBxPlane + off) =
          make_uint4(pk[part][p][0], pk[part][p][1], pk[part][p][2], pk[part][p][3]);
}

// Both splits of an update in one launch (CTAs [0, half) cut L21, the rest U12), one half of 32
// columns per blockIdx.z.  L21: rows k+kb .. n-1 of columns k .. k+kb-1; U12: columns k+kb .. n-1
// of rows k .. k+kb-1 (kb = 32 KH).  Four threads per row (column), eight columns (rows) each.
__global__ void __launch_bounds__(256) bx3_split_kernel(BatchDesc d, const float2* __restrict__ A, int64_t k,
                                                        int64_t ntile, int64_t half, unsigned char* __restrict__ tA,
                                                        unsigned char* __restrict__ tB) {
  const bool cols = (int64_t)blockIdx.x >= half;
  const int64_t t = ((int64_t)blockIdx.x - (cols ? half : 0)) * blockDim.x + threadIdx.x;
  const int64_t r = t >> 2;  // padded row (column) of the trailing block
  const int kq = (int)(t & 3), h = (int)blockIdx.z, KH = (int)gridDim.z;
  const int64_t b = blockIdx.y;
  if (r >= ntile * kBxTile) return;
  // a grouped batch: this matrix's order, panel width and trailing size (the launch's tile
  // count stays the stride of the term tiles)
  const int64_t n = d.order(b);
  if (k + kBxNB * KH >= n) return;
  const int kb = kBxNB * KH;
  const float2* Ab = A + d.offset(b);
  const bool live = r < n - k - kb;
  float2 v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int kk = h * kBxK + 8 * kq + c;
    const int64_t at = cols ? (k + kk) + (k + kb + r) * n : (k + kb + r) + (k + kk) * n;
    v[c] = live ? Ab[at] : make_float2(0.f, 0.f);
  }
  unsigned char* tile = (cols ? tB : tA) + ((b * ntile + r / kBxTile) * KH + h) * (int64_t)kBxTileBytes;
  store_terms8(tile, (int)(r % kBxTile), 8 * kq, v);
}

// A22 -= L21 U12 over K = 32 KH, on the trailing columns [0, ccols).  Bound: HBM, 16 bytes of
// A22 per entry and pass; a half's products of a 128 x 128 tile take 2 us, the tile's traffic 6 us
// of the SM's share.  So the subtraction never stops for the products (a thread of its own
// issues them; when one thread of the epilogue did, between tiles, four matrices of order 8000
// took 845 us for their largest update at K = 32, 4.8 TB/s; K = 64 now takes 783), and K = 64 makes
// half as many passes: all updates of that factorization 72.1 -> 37.2 ms.
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
template <int KH>
__global__ void __launch_bounds__(kBxThreads, 1) bx3_gemm_kernel(BatchDesc d, float2* __restrict__ A, int64_t k,
                                                               int64_t ntile, const unsigned char* __restrict__ tA,
                                                               const unsigned char* __restrict__ tB,
                                                               int* __restrict__ timeout_flag, int group,
                                                               int64_t ccols) {
  extern __shared__ __align__(1024) unsigned char bsm[];
  __shared__ __align__(8) uint64_t full[2], slot_free[2], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int64_t rt = blockIdx.x, b = blockIdx.z;
  const int64_t ct0 = blockIdx.y * (int64_t)group;
  // a grouped batch: CTAs past this matrix's trailing block leave before any barrier or
  // tensor-memory allocation
  const int64_t n = d.order(b);
  if (k + kBxNB * KH >= n) return;
  const int kb = kBxNB * KH;
  const int64_t rest = n - k - kb, cols = rest < ccols ? rest : ccols;
  if (rt * kBxTile >= rest || ct0 * kBxTile >= cols) return;
  const int64_t ntile_b = (cols + kBxTile - 1) / kBxTile;
  const int ntiles = (int)((ntile_b - ct0) < group ? (ntile_b - ct0) : group);
  const int nsteps = ntiles * KH;  // step s: half s % KH of column tile s / KH
  const int half = tid >> 7;       // column half of an epilogue thread
  const int64_t r = rt * kBxTile + (tid & (kBxTile - 1));
  const bool row_live = r < rest && tid < kBxEpilogue;
  float2* crow = A + d.offset(b) + (k + kb + r) + (k + kb) * n;  // this thread's row of A22
  auto load_c = [&](float2 (&cv)[32], int64_t c0) {
#pragma unroll
    for (int q = 0; q < 32; ++q) cv[q] = (row_live && c0 + q < cols) ? crow[(c0 + q) * n] : make_float2(0.f, 0.f);
  };
  float2 c_lo[32], c_hi[32];
  if (tid < kBxEpilogue) load_c(c_lo, ct0 * kBxTile + half * 64);
  if (tid == 0) {
    for (int q = 0; q < 2; ++q) {
      tc::mbar_init(&full[q], 1);
      tc::mbar_init(&slot_free[q], 1);
      tc::mbar_init(&acc_full[q], 1);
      tc::mbar_init(&acc_empty[q], kBxEpilogue);
    }
    s_fail = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tmem_base, kBxTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  // a bounded wait that also ends when the other role has given up
  auto wait = [&](uint64_t* bar, int phase) {
    for (int q = 0; q < 64; ++q) {
      if (tc::mbar_wait(bar, (uint32_t)(phase & 1), kBxWaitPolls / 64)) return true;
      if (s_fail) return false;
    }
    return false;
  };
  if (tid == kBxEpilogue) {
    unsigned char* As = bsm;
    unsigned char* Bs = bsm + KH * kBxTileBytes;
    // a 48 KB tile as three 16 KB bulk copies
    auto load_tile = [&](unsigned char* dst, const unsigned char* src, uint64_t* bar) {
      for (int q = 0; q < kBxTileBytes; q += 16384) tc::bulk_g2s(dst + q, src + q, 16384, bar);
    };
    auto load_step = [&](int s) {
      tc::mbar_arrive_expect_tx(&full[s & 1], (uint32_t)(kBxTileBytes * (s == 0 ? KH + 1 : 1)));
      if (s == 0)
        for (int h = 0; h < KH; ++h)
          load_tile(As + h * kBxTileBytes, tA + ((b * ntile + rt) * KH + h) * (int64_t)kBxTileBytes, &full[0]);
      load_tile(Bs + (s & 1) * kBxTileBytes, tB + ((b * ntile + ct0) * KH + s) * (int64_t)kBxTileBytes, &full[s & 1]);
    };
    const uint32_t id = tc::idesc_bf16_f32(kBxTile, kBxTile), id_neg = tc::idesc_bf16_f32_nega(kBxTile, kBxTile);
    constexpr uint32_t sbo = (kBxK / 8) * 128;  // 8-row core groups are K * 16 bytes apart
    // the 48 products of step s into accumulator buffer t & 1
    auto issue = [&](int s) {
      const int t = s / KH, h = s - t * KH;
      const uint32_t a0 = tc::smem_u32(As + h * kBxTileBytes), b0 = tc::smem_u32(Bs + (s & 1) * kBxTileBytes);
      const uint32_t t_re = tmem + (uint32_t)(t & 1) * 256u, t_im = t_re + 128u;
      uint32_t acc = h > 0 ? 1u : 0u;
#pragma unroll
      for (int p = 0; p < kBxTerms; ++p)
#pragma unroll
        for (int q = 0; q + p < kBxTerms; ++q)
#pragma unroll
          for (int kk = 0; kk < kBxK / 16; ++kk) {
            const uint32_t ko = (uint32_t)kk * 256;
            const uint64_t ar = tc::smem_desc(a0 + (uint32_t)p * kBxPlane + ko, 128, sbo);
            const uint64_t ai = tc::smem_desc(a0 + (uint32_t)(kBxTerms + p) * kBxPlane + ko, 128, sbo);
            const uint64_t br = tc::smem_desc(b0 + (uint32_t)q * kBxPlane + ko, 128, sbo);
            const uint64_t bi = tc::smem_desc(b0 + (uint32_t)(kBxTerms + q) * kBxPlane + ko, 128, sbo);
            tc::mma_bf16(t_re, ar, br, id, acc);
            tc::mma_bf16(t_re, ai, bi, id_neg, 1u);
            tc::mma_bf16(t_im, ar, bi, id, acc);
            tc::mma_bf16(t_im, ai, br, id, 1u);
            acc = 1u;
          }
      tc::mma_commit(&slot_free[s & 1]);
      if (h == KH - 1) tc::mma_commit(&acc_full[t & 1]);
    };
    int loaded = 0, landed = 0, issued = 0;  // steps
    bool ok = true;
    for (; loaded < 2 && loaded < nsteps; ++loaded) load_step(loaded);
    for (int s = 0; s < nsteps; ++s) {
      const int t = s / KH;
      if (!(ok = wait(&full[s & 1], s >> 1))) break;
      ++landed;
      // the accumulators that tile t - 2 left are read
      if (s == t * KH && t >= 2 && !(ok = wait(&acc_empty[t & 1], (t - 2) >> 1))) break;
      tc::fence_after_sync();
      issue(s);
      ++issued;
      if (s >= 1 && s + 1 < nsteps) {  // the slot of step s - 1 takes step s + 1
        if (!(ok = wait(&slot_free[(s - 1) & 1], (s - 1) >> 1))) break;
        load_step(s + 1);
        ++loaded;
      }
    }
    if (!ok) {  // reported by the host as a timeout
      s_fail = 1;
      atomicExch(timeout_flag, 1);
    }
    // no copy and no product is in flight when the shared and the tensor memory are released
    for (int q = landed; q < loaded; ++q) tc::mbar_wait(&full[q & 1], (uint32_t)((q >> 1) & 1), kBxWaitPolls);
    for (int q = issued > 2 ? issued - 2 : 0; q < issued; ++q)
      tc::mbar_wait(&slot_free[q & 1], (uint32_t)((q >> 1) & 1), kBxWaitPolls);
  } else if (tid < kBxEpilogue) {
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    // A22 -= 32 columns of the accumulators (column c0 of the half of tile t, loaded before)
    auto subtract = [&](const float2 (&cv)[32], int t, int c0) {
      const int64_t cb = (ct0 + t) * kBxTile + half * 64 + c0;
      const uint32_t t_re = tmem + lane_off + (uint32_t)(t & 1) * 256u + (uint32_t)(half * 64 + c0), t_im = t_re + 128u;
#pragma unroll
      for (int h = 0; h < 32; h += 8) {
        float re[8], im[8];
        tc::tmem_ld8(t_re + (uint32_t)h, re);
        tc::tmem_ld8(t_im + (uint32_t)h, im);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (row_live && cb + h + q < cols)
            crow[(cb + h + q) * n] = make_float2(cv[h + q].x - re[q], cv[h + q].y - im[q]);
      }
    };
    for (int t = 0; t < ntiles; ++t) {
      load_c(c_hi, (ct0 + t) * kBxTile + half * 64 + 32);
      const bool ok = wait(&acc_full[t & 1], t >> 1);
      if (!ok) {
        s_fail = 1;
        atomicExch(timeout_flag, 1);
      }
      if (__any_sync(0xffffffffu, !ok)) break;  // the tensor-memory loads are warp-wide
      tc::fence_after_sync();
      subtract(c_lo, t, 0);
      if (t + 1 < ntiles) load_c(c_lo, (ct0 + t + 1) * kBxTile + half * 64);
      subtract(c_hi, t, 32);
      tc::fence_before_sync();
      mbar_arrive(&acc_empty[t & 1]);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kBxTmemCols);
}

}  // namespace

// Two panels of 32 columns per pass over A22 (K = 64) while the trailing
// blocks have kBxDeepEntries together: a pass less against one more small update between the two
// panels (15 us) and a longer triangular solve (22 against 16 us).  Factor and solve of one matrix,
// from 8e6 entries on against from 3.2e7: order 2900 14.1 / 14.1 ms, 4000 20.6 / 21.0, 5500 31.1 / 33.0,
// 7000 43.7 / 45.9.  In a grouped batch, whose orders
// are within a factor of two of the largest, half of the largest's entries are counted per matrix;
// matrices that end at either panel leave the kernels as they do at K = 32 (ten bodies of
// 300 to 2400 panels at 8 frequencies: updates 9.1 -> 6.1 ms, the batch 46.0 -> 43.5).
bool bx3_deep(const BatchDesc& d, int64_t rest) {
  return d.extra == 0 && rest > 0 &&
         (double)rest * (double)rest * (double)d.batch * (d.orders ? 0.5 : 1.0) >= kBxDeepEntries;
}

size_t bx3_workspace_bytes(int64_t n, int64_t batch) {
  const int64_t t = (n + kBxTile - 1) / kBxTile;
  const int halves = (double)n * (double)n * (double)batch >= kBxDeepEntries ? 2 : 1;
  return (size_t)batch * 2 * (size_t)(t * halves) * kBxTileBytes + 1024;
}

// A22 -= L21 U12 at panel step k over kb <= 64 columns, on the first ccols trailing columns
void bx3_trailing_update(cudaStream_t st, LaunchCounter lc, const BatchDesc& d, float2* A, int64_t k, int kb,
                         int64_t ccols, void* ws, int* timeout_flag) {
  const int64_t rest = d.n - k - kb;
  if (rest <= 0) return;
  const int KH = kb > kBxK ? 2 : 1;
  const int64_t cols = rest < ccols ? rest : ccols;
  const int64_t nt = (rest + kBxTile - 1) / kBxTile, ntc = (cols + kBxTile - 1) / kBxTile;
  unsigned char* tA = static_cast<unsigned char*>(ws);
  unsigned char* tB = tA + d.batch * nt * KH * (int64_t)kBxTileBytes;
  // 4 threads per row / column, 256 per CTA; rows then columns
  dim3 gs((unsigned)((nt + ntc) * 2), (unsigned)d.batch, (unsigned)KH);
  MH_LAUNCH(lc, st, "lu_bx3_split", bx3_split_kernel<<<gs, 256, 0, st>>>(d, A, k, nt, nt * 2, tA, tB));
  const size_t smem = (size_t)(KH + 2) * kBxTileBytes;
  int group = lc.tile(d.n).bx_group * KH;  // the same bytes of B per A tile loaded
  group = group < 1 ? 1 : (group > kBxGroupMax ? kBxGroupMax : group);
  dim3 gg((unsigned)nt, (unsigned)((ntc + group - 1) / group), (unsigned)d.batch);
  auto launch = [&](auto kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    MH_LAUNCH(lc, st, "lu_gemm_bx3",
              kernel<<<gg, kBxThreads, smem, st>>>(d, A, k, nt, tA, tB, timeout_flag, group, ccols));
  };
  if (KH == 2) launch(bx3_gemm_kernel<2>);
  else launch(bx3_gemm_kernel<1>);
}

}  // namespace mh
