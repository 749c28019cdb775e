// Plain FP32 batched GEMM (FFMA) with a cp.async pipeline, for the fp32 row in its plain form.
//
// Semantics follow the reference (hirokitokura/ssblasEx): C <- beta*C, not read when beta == 0
// (src/include/CScale/Xgemm_scale_kernel.hpp:164-176), then C <- C + acc*alpha with one fused
// multiply-add (src/include/GemmCore/Xgemm_kernel_sve_v4x5_1.hpp:93-127). The reference adds
// alpha*acc once per 512-wide K block; here it is added once, which differs only by rounding.
//
// Design: one CTA per (BM x BN tile, instance). op(A) and op(B) tiles reach shared memory through
// a STAGES-deep cp.async ring, always staged [k][mn] (mn contiguous) so that every thread reads
// its TM (TN) consecutive values with 16-byte loads:
//   - an operand whose rows (m or n) are contiguous in global memory is copied in 16-byte chunks
//     along mn (when 16-byte aligned; 4-byte copies otherwise);
//   - an operand whose K is contiguous is transposed by the copy itself: one 4-byte cp.async per
//     element, consecutive threads taking consecutive k of one row.
// Small problems (the 64^3 instances of a 4096-instance batch) keep the whole K in flight from
// the start: with K <= STAGES * BK every stage is issued in the prologue.
// Each thread owns a TM x TN block of C (rows tx*TM.., columns ty*TN..); a warp covers 4 x 8
// threads, so its A reads are 4 distinct 16-byte vectors and its B reads 8 (broadcasts). The products are
// packed fused multiply-adds over pairs of rows (f32x2.cuh), the same results in half the issue slots
// (4096 x 64^3 TT, configuration 9: 0.0785 -> 0.0735 ms; NN, configuration 3: 0.078 -> 0.076).
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "grouped.h"
#include "internal.h"
#include "ptx.cuh"
#include "sgemm_load.cuh"

namespace ssb {
namespace {

struct SgemmArgs {
  long m, n, k, lda, ldb, ldc, batch;
  const float* const* A;
  const float* const* B;
  float* const* C;
  float alpha, beta;
};

// One BM x BN tile of C = alpha op(A) op(B) + beta C for one instance, by the whole CTA: the K loop
// over the stage ring, then the epilogue. Leaves the stage buffers free.
template <int BM, int BN, int BK, int TM, int TN, int STAGES, bool A_MN, bool B_MN>
__device__ __forceinline__ void sgemm_tile(const float* __restrict__ A, const float* __restrict__ B,
                                           float* __restrict__ C, long m, long n, long k, long lda, long ldb,
                                           long ldc, float alpha, float beta, long m0, long n0, float* sm) {
  constexpr int TX = BM / TM, TY = BN / TN, NT = TX * TY;
  constexpr int PA = BM + 4, PB = BN + 4;
  constexpr int STAGE = BK * (PA + PB);
  // warp = 4 (m) x 8 (n) threads
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  constexpr int WX = TX / 4;   // warps along m
  const int tx = (warp % WX) * 4 + lane % 4;
  const int ty = (warp / WX) * 8 + lane / 4;
  const bool vecA = ((uintptr_t)A % 16 == 0) && (lda % 4 == 0);
  const bool vecB = ((uintptr_t)B % 16 == 0) && (ldb % 4 == 0);
  uint64_t acc2[TM / 2][TN];     // pairs of rows
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc2[i][j] = 0;

  const long ktiles = (k + BK - 1) / BK;
  auto issue = [&](long kt) {
    float* sa = sm + (kt % STAGES) * STAGE;
    float* sb = sa + BK * PA;
    sload<BM, BK, NT, A_MN>(sa, A, m, k, lda, m0, kt * BK, vecA);
    sload<BN, BK, NT, B_MN>(sb, B, n, k, ldb, n0, kt * BK, vecB);
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ktiles) issue(s);
    commit_s();
  }
  for (long kt = 0; kt < ktiles; ++kt) {
    wait_s<STAGES - 2>();
    __syncthreads();
    if (kt + STAGES - 1 < ktiles) issue(kt + STAGES - 1);
    commit_s();
    const float* sa = sm + (kt % STAGES) * STAGE;
    const float* sb = sa + BK * PA;
#pragma unroll 4
    for (int kk = 0; kk < BK; ++kk) outer2<TM, TN>(acc2, sa + kk * PA + tx * TM, sb + kk * PB + ty * TN);
  }
  float acc[TM][TN];
  unpack_acc<TM, TN>(acc2, acc);
  wait_s<0>();
  __syncthreads();   // the next tile's copies reuse the stage buffers

  // epilogue: C rows m0 + tx*TM + i (contiguous per thread), columns n0 + ty*TN + j; 16-byte
  // reads and writes when the thread's rows are inside C and C is 16-byte aligned
  const bool read_c = beta != 0.0f;
  const long gi0 = m0 + tx * TM;
  const bool cvec = (((uintptr_t)C) % 16 == 0) && (ldc % 4 == 0) && gi0 + TM <= m;
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    const long gj = n0 + ty * TN + j;
    if (gj >= n) continue;
    float* cp = C + gi0 + gj * ldc;
    if (cvec) {
      float4 cv[TM / 4];
#pragma unroll
      for (int i = 0; i < TM; i += 4) cv[i / 4] = read_c ? *(const float4*)(cp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        float4 o;
        o.x = fmaf(acc[i][j], alpha, read_c ? beta * cv[i / 4].x : 0.0f);
        o.y = fmaf(acc[i + 1][j], alpha, read_c ? beta * cv[i / 4].y : 0.0f);
        o.z = fmaf(acc[i + 2][j], alpha, read_c ? beta * cv[i / 4].z : 0.0f);
        o.w = fmaf(acc[i + 3][j], alpha, read_c ? beta * cv[i / 4].w : 0.0f);
        *(float4*)(cp + i) = o;
      }
    } else {
      float cv[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) cv[i] = (read_c && gi0 + i < m) ? cp[i] : 0.0f;
#pragma unroll
      for (int i = 0; i < TM; ++i)
        if (gi0 + i < m) cp[i] = fmaf(acc[i][j], alpha, read_c ? beta * cv[i] : 0.0f);
    }
  }
}

template <int BM, int BN, int BK, int TM, int TN, int STAGES, int MINB, bool A_MN, bool B_MN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MINB) sgemm_async_kernel(SgemmArgs args) {
  extern __shared__ __align__(16) float sm[];
  const long tiles_m = (args.m + BM - 1) / BM;
  const long m0 = (blockIdx.x % tiles_m) * BM;
  const long n0 = (blockIdx.x / tiles_m) * BN;
  for (long b = blockIdx.y; b < args.batch; b += gridDim.y)
    sgemm_tile<BM, BN, BK, TM, TN, STAGES, A_MN, B_MN>(args.A[b], args.B[b], args.C[b], args.m, args.n, args.k,
                                                       args.lda, args.ldb, args.ldc, args.alpha, args.beta, m0, n0,
                                                       sm);
}

// Grouped form (plain fp32 instances of ssblasGemmGroupedBatchedEx): one CTA per (instance,
// 64 x 64 tile) entry of a tile table whose instances all have this op(A) / op(B) layout; the tile
// shape of configuration 3.
constexpr int kGT = 64, kGBK = 32, kGTM = 4, kGST = 2;
template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__((kGT / kGTM) * (kGT / kGTM), 3)
sgemm_grouped_kernel(const SimtGInst* __restrict__ inst, const int* __restrict__ tiles, const float* const* A,
                     const float* const* B, float* const* C) {
  extern __shared__ __align__(16) float sm[];
  ptx::grid_dep_launch();
  const int* t = tiles + 3 * (long)blockIdx.x;
  const SimtGInst g = inst[t[0]];
  sgemm_tile<kGT, kGT, kGBK, kGTM, kGTM, kGST, A_MN, B_MN>(A[g.idx], B[g.idx], C[g.idx], g.m, g.n, g.k, g.lda, g.ldb,
                                                         g.ldc, g.alpha_f, g.beta_f, (long)t[1] * kGT,
                                                         (long)t[2] * kGT, sm);
  ptx::grid_chain_end();
}

// Register-heavy form for K <= KMAX: one 64 x 64 tile of one instance per CTA of 64 threads, each
// thread an 8 x 8 block of C (tx = t % 8, ty = t / 8: rows 4 tx.. and 32 + 4 tx.., columns 8 ty..). The
// whole K of the tile is requested at once (16-deep slices of the cp.async copies above, both operands
// staged [k][rows]), C (READ_C) is read into registers while the copies land, and the inner
// loop issues 4 shared-memory vector loads per 64 FFMAs. Several CTAs per SM overlap one tile's loads with
// another's products: six without the 64 registers of C, else four.
// The rows as two groups of four, 32 apart: eight lanes then read 128 contiguous bytes, where rows
// 8 tx.. took two passes of the shared memory each, and they read and write whole lines of C. What bounds
// it is those loads (64 bytes per thread and k, 16 passes per warp against 16 of the products' pipe).
// Measured, 4096 x 64^3: TT with C read 0.0735 -> 0.069 ms (0.041 of HBM time), NN 0.079 -> 0.070.
// (Staging a K-contiguous operand as it lies, [rows][k] with 16-byte copies: 0.105 ms against 0.084 then;
// C through L2 prefetches instead of registers, six CTAs: 0.084 against 0.069.)
template <int KMAX, int MINB, bool READ_C, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(64, MINB) sgemm_reg8_kernel(SgemmArgs args, uint32_t tiles_m, uint32_t tiles) {
  constexpr int P = 64 + 4;
  extern __shared__ __align__(16) float sm[];
  float* sa = sm;                 // [KMAX][P] op(A): k, then m
  float* sb = sm + KMAX * P;      // [KMAX][P] op(B): k, then n
  const uint32_t w = blockIdx.x;
  const uint32_t bb = w / tiles, t = w - bb * tiles;
  const uint32_t tn = t / tiles_m;
  const long b = bb;
  const long m0 = (long)(t - tn * tiles_m) * 64, n0 = (long)tn * 64;
  const float* __restrict__ A = args.A[b];
  const float* __restrict__ B = args.B[b];
  float* __restrict__ C = args.C[b];
  const bool vecA = ((uintptr_t)A % 16 == 0) && (args.lda % 4 == 0);
  const bool vecB = ((uintptr_t)B % 16 == 0) && (args.ldb % 4 == 0);
  const int K = (int)args.k;   // <= KMAX (checked by the launcher)
  const int slices = (K + 15) / 16;
  for (int sl = 0; sl < slices; ++sl) {
    sload<64, 16, 64, A_MN>(sa + sl * 16 * P, A, args.m, args.k, args.lda, m0, sl * 16, vecA);
    sload<64, 16, 64, B_MN>(sb + sl * 16 * P, B, args.n, args.k, args.ldb, n0, sl * 16, vecB);
  }
  commit_s();

  const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;
  const long gi0 = m0 + 4 * tx;   // and gi0 + 32
  const bool vecC = (((uintptr_t)C) % 16 == 0) && (args.ldc % 4 == 0);
  const bool cvec[2] = {vecC && gi0 + 4 <= args.m, vecC && gi0 + 36 <= args.m};
  // C of this thread's block, in flight while the operand copies land
  float cv[READ_C ? 8 : 1][8];
  if constexpr (READ_C) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long gj = n0 + ty * 8 + j;
      const float* cp = C + gi0 + gj * args.ldc;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (gj < args.n && cvec[h]) {
          const float4 x = *(const float4*)(cp + 32 * h);
          cv[j][4 * h] = x.x; cv[j][4 * h + 1] = x.y; cv[j][4 * h + 2] = x.z; cv[j][4 * h + 3] = x.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) cv[j][4 * h + i] = (gj < args.n && gi0 + 32 * h + i < args.m) ? cp[32 * h + i] : 0.0f;
        }
      }
    }
  }
  wait_s<0>();
  __syncthreads();

  uint64_t acc2[4][8];           // pairs of rows
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc2[i][j] = 0;
#pragma unroll 4
  for (int kk = 0; kk < K; ++kk) outer2<8, 8, 32>(acc2, sa + kk * P + 4 * tx, sb + kk * P + ty * 8);
  float acc[8][8];
  unpack_acc<8, 8>(acc2, acc);

#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const long gj = n0 + ty * 8 + j;
    if (gj >= args.n) continue;
    float* cp = C + gi0 + gj * args.ldc;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = fmaf(acc[4 * h + i][j], args.alpha, READ_C ? args.beta * cv[READ_C ? j : 0][4 * h + i] : 0.0f);
      if (cvec[h]) {
        *(float4*)(cp + 32 * h) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (gi0 + 32 * h + i < args.m) cp[32 * h + i] = o[i];
      }
    }
  }
}

template <int KMAX, int MINB, bool READ_C, bool A_MN, bool B_MN>
cudaError_t launch_reg8(const SgemmArgs& a, cudaStream_t st) {
  constexpr int SMEM = 2 * KMAX * (64 + 4) * 4;
  auto kern = sgemm_reg8_kernel<KMAX, MINB, READ_C, A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, SMEM)) return e;
  const long tiles_m = (a.m + 63) / 64;
  const long tiles = tiles_m * ((a.n + 63) / 64);
  const long total = tiles * a.batch;
  if (total >= (1L << 31)) return cudaErrorNotSupported;
  kern<<<(unsigned)total, 64, SMEM, st>>>(a, (uint32_t)tiles_m, (uint32_t)tiles);
  return cudaGetLastError();
}

template <int KMAX, int MINB, bool READ_C>
cudaError_t launch_reg8_l(const SgemmArgs& a, bool a_mn, bool b_mn, cudaStream_t st) {
  if (a_mn && b_mn) return launch_reg8<KMAX, MINB, READ_C, true, true>(a, st);
  if (a_mn) return launch_reg8<KMAX, MINB, READ_C, true, false>(a, st);
  if (b_mn) return launch_reg8<KMAX, MINB, READ_C, false, true>(a, st);
  return launch_reg8<KMAX, MINB, READ_C, false, false>(a, st);
}

// K split inside the CTA, for k <= KMAX: one 64 x 64 tile per CTA of 256 threads, four groups of
// 64 threads, each group an 8 x 8 block per thread over a quarter of K (as the 64-thread form
// above), then the four partial tiles meet in shared memory (over the operand buffers) and every
// thread adds its 16 outputs' parts in a fixed order (group 0 + 1 + 2 + 3) and applies alpha and
// beta. Four times the warps of the 64-thread form per tile, so batches of few large-K tiles
// (64 x 128^3: 256 tiles for 148 SMs) keep every scheduler fed.
template <int KMAX, int MINB, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(256, MINB) sgemm_ksplit_kernel(SgemmArgs args, uint32_t tiles_m, uint32_t tiles) {
  constexpr int P = 64 + 4;
  extern __shared__ __align__(16) float sm[];
  float* sa = sm;                 // [KMAX][P] op(A): k, then m
  float* sb = sm + KMAX * P;      // [KMAX][P] op(B): k, then n
  float* red = sm;                // after the products: [4 groups][64 columns][P] partial tiles
  float* sc = sm + 2 * KMAX * P;  // [64 columns][P] C (beta != 0)
  static_assert(2 * KMAX >= 4 * 64, "the partial tiles reuse the operand buffers");
  const uint32_t w = blockIdx.x;
  const uint32_t bb = w / tiles, t = w - bb * tiles;
  const uint32_t tn = t / tiles_m;
  const long b = bb;
  const long m0 = (long)(t - tn * tiles_m) * 64, n0 = (long)tn * 64;
  const float* __restrict__ A = args.A[b];
  const float* __restrict__ B = args.B[b];
  float* __restrict__ C = args.C[b];
  const bool vecA = ((uintptr_t)A % 16 == 0) && (args.lda % 4 == 0);
  const bool vecB = ((uintptr_t)B % 16 == 0) && (args.ldb % 4 == 0);
  const int K = (int)args.k;   // <= KMAX (checked by the launcher)
  const bool read_c = args.beta != 0.0f;
  const bool vecC = ((uintptr_t)C % 16 == 0) && (args.ldc % 4 == 0);
  for (int sl = 0; sl < (K + 15) / 16; ++sl) {
    sload<64, 16, 256, A_MN>(sa + sl * 16 * P, A, args.m, args.k, args.lda, m0, sl * 16, vecA);
    sload<64, 16, 256, B_MN>(sb + sl * 16 * P, B, args.n, args.k, args.ldb, n0, sl * 16, vecB);
  }
  // C tile (columns n0.., rows m0..) staged [column][row], in flight with the operands
  if (read_c)
    for (int sl = 0; sl < 4; ++sl)
      sload<64, 16, 256, true>(sc + sl * 16 * P, C, args.m, args.n, args.ldc, m0, n0 + sl * 16, vecC);
  commit_s();

  // output mapping of the final sum: thread t takes rows 4 (t % 16).., columns 4 (t / 16)..
  const int orow = 4 * (threadIdx.x % 16), ocol = 4 * (threadIdx.x / 16);
  const long gi0 = m0 + orow;
  const bool cvec = vecC && gi0 + 4 <= args.m;
  wait_s<0>();
  __syncthreads();

  const int g = threadIdx.x / 64, t64 = threadIdx.x % 64;
  const int tx = t64 % 8, ty = t64 / 8;
  const int kq = (K + 3) / 4;
  const int k0 = g * kq, k1 = (k0 + kq < K) ? k0 + kq : K;
  uint64_t acc2[4][8];           // pairs of rows
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc2[i][j] = 0;
#pragma unroll 2
  for (int kk = k0; kk < k1; ++kk) outer2<8, 8, 32>(acc2, sa + kk * P + 4 * tx, sb + kk * P + ty * 8);
  float acc[8][8];
  unpack_acc<8, 8>(acc2, acc);
  __syncthreads();   // every group is done with the operand buffers
  float* part = red + g * 64 * P;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float* q = part + (ty * 8 + j) * P + 4 * tx;
    *(float4*)q = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
    *(float4*)(q + 32) = make_float4(acc[4][j], acc[5][j], acc[6][j], acc[7][j]);
  }
  __syncthreads();

#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const long gj = n0 + ocol + j;
    if (gj >= args.n) continue;
    float4 s = *(const float4*)(red + (ocol + j) * P + orow);
#pragma unroll
    for (int gg = 1; gg < 4; ++gg) {
      const float4 x = *(const float4*)(red + gg * 64 * P + (ocol + j) * P + orow);
      s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
    }
    const float sv[4] = {s.x, s.y, s.z, s.w};
    float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (read_c) c4 = *(const float4*)(sc + (ocol + j) * P + orow);
    const float cv[4] = {c4.x, c4.y, c4.z, c4.w};
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = fmaf(sv[i], args.alpha, read_c ? args.beta * cv[i] : 0.0f);
    float* cp = C + gi0 + gj * args.ldc;
    if (cvec) {
      *(float4*)cp = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (gi0 + i < args.m) cp[i] = o[i];
    }
  }
}

template <int KMAX, int MINB, bool A_MN, bool B_MN>
cudaError_t launch_ksplit(const SgemmArgs& a, cudaStream_t st) {
  constexpr int SMEM = (2 * KMAX + 64) * (64 + 4) * 4;
  auto kern = sgemm_ksplit_kernel<KMAX, MINB, A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, SMEM)) return e;
  const long tiles_m = (a.m + 63) / 64;
  const long tiles = tiles_m * ((a.n + 63) / 64);
  const long total = tiles * a.batch;
  if (total >= (1L << 31)) return cudaErrorNotSupported;
  kern<<<(unsigned)total, 256, SMEM, st>>>(a, (uint32_t)tiles_m, (uint32_t)tiles);
  return cudaGetLastError();
}

template <int KMAX, int MINB>
cudaError_t launch_ksplit_l(const SgemmArgs& a, bool a_mn, bool b_mn, cudaStream_t st) {
  if (a_mn && b_mn) return launch_ksplit<KMAX, MINB, true, true>(a, st);
  if (a_mn) return launch_ksplit<KMAX, MINB, true, false>(a, st);
  if (b_mn) return launch_ksplit<KMAX, MINB, false, true>(a, st);
  return launch_ksplit<KMAX, MINB, false, false>(a, st);
}

template <int BM, int BN, int BK, int TM, int TN, int STAGES, int MINB, bool A_MN, bool B_MN>
cudaError_t launch_s(const SgemmArgs& a, cudaStream_t st) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int SMEM = STAGES * BK * (BM + 4 + BN + 4) * 4;
  auto kern = sgemm_async_kernel<BM, BN, BK, TM, TN, STAGES, MINB, A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, SMEM)) return e;
  const long tiles = ((a.m + BM - 1) / BM) * ((a.n + BN - 1) / BN);
  if (tiles > 0x7fffffffL) return cudaErrorInvalidValue;
  dim3 grid((unsigned)tiles, (unsigned)(a.batch < 65535 ? a.batch : 65535));
  kern<<<grid, NT, SMEM, st>>>(a);
  return cudaGetLastError();
}

template <int BM, int BN, int BK, int TM, int TN, int STAGES, int MINB>
cudaError_t launch_sl(const SgemmArgs& a, bool a_mn, bool b_mn, cudaStream_t st) {
  if (a_mn && b_mn) return launch_s<BM, BN, BK, TM, TN, STAGES, MINB, true, true>(a, st);
  if (a_mn) return launch_s<BM, BN, BK, TM, TN, STAGES, MINB, true, false>(a, st);
  if (b_mn) return launch_s<BM, BN, BK, TM, TN, STAGES, MINB, false, true>(a, st);
  return launch_s<BM, BN, BK, TM, TN, STAGES, MINB, false, false>(a, st);
}

}  // namespace

template <bool A_MN, bool B_MN>
cudaError_t launch_sgemm_grouped_layout(const GroupedSimt& s, const GroupedPtrs& p, int lay, cudaStream_t st, bool& follows) {
  constexpr int SMEM = kGST * kGBK * (2 * kGT + 8) * 4;
  auto kern = sgemm_grouped_kernel<A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, SMEM)) return e;
  note_launch();
  return launch_chained(kern, (unsigned)s.nsg[lay], (kGT / kGTM) * (kGT / kGTM), SMEM, st, follows,
                        (const SimtGInst*)s.inst32, (const int*)s.sg_tiles[lay], (const float* const*)p.A,
                        (const float* const*)p.B, (float* const*)p.C);
}

// The plain fp32 tiles of a grouped call, one launch per op(A) / op(B) layout present (layout
// index = 2 * (op(A) rows contiguous) + (op(B) columns contiguous)).
cudaError_t launch_sgemm_grouped(const GroupedSimt& s, const GroupedPtrs& p, cudaStream_t st, bool& follows) {
  if (!s.nsg[0] && !s.nsg[1] && !s.nsg[2] && !s.nsg[3]) return cudaSuccess;
  ProfScope prof("sgemm_grouped", st);
  cudaError_t e = cudaSuccess;
  for (int lay = 0; lay < 4 && e == cudaSuccess; ++lay) {
    if (!s.nsg[lay]) continue;
    switch (lay) {
      case 3: e = launch_sgemm_grouped_layout<true, true>(s, p, lay, st, follows); break;
      case 2: e = launch_sgemm_grouped_layout<true, false>(s, p, lay, st, follows); break;
      case 1: e = launch_sgemm_grouped_layout<false, true>(s, p, lay, st, follows); break;
      default: e = launch_sgemm_grouped_layout<false, false>(s, p, lay, st, follows); break;
    }
  }
  return e;
}

cudaError_t launch_sgemm_async(const BatchDesc& d, int config, cudaStream_t st) {
  SgemmArgs a;
  a.m = d.m; a.n = d.n; a.k = d.k; a.lda = d.lda; a.ldb = d.ldb; a.ldc = d.ldc; a.batch = d.batch;
  a.A = (const float* const*)d.A;
  a.B = (const float* const*)d.B;
  a.C = (float* const*)d.C;
  a.alpha = d.alpha_f;
  a.beta = d.beta_f;
  const bool a_mn = d.transa == SSBLAS_OP_N;   // op(A) rows (m) contiguous
  const bool b_mn = d.transb == SSBLAS_OP_T;   // op(B) columns (n) contiguous
  cudaError_t e;
  // 12 / 13: 64 x 64 tiles, TMA staging and bulk stores (equally spaced, 16-byte aligned
  //   instances): two stages and two C tiles, two CTAs per SM / three and three, one CTA per SM
  if (config == 12 || config == 13) {
    e = launch_sgemm_tma(d, config - 12, st);
    if (e != cudaErrorNotSupported) return e;
  }
  ProfScope prof("sgemm_async", st);
  // 3: 64 x 64 tiles, 256 threads of 4 x 4, 32-deep K stages x 2 (k <= 64 entirely in flight)
  // 4: 128 x 128 tiles, 256 threads of 8 x 8, 16-deep K stages x 3
  // 7: 32 x 64 tiles, 128 threads of 4 x 4, 32-deep K stages x 4 (k <= 128 entirely in flight):
  //   four times the CTAs of configuration 3, for batches whose 64 x 64 tiles fill under a wave
  // 8: 32 x 32 tiles, 64 threads of 4 x 4, 16-deep K stages x 8
  // 9 (k <= 64) / 10 (k <= 128): 64 x 64 tiles, 64 threads of 8 x 8, the whole K at once (5 and 6,
  //   forced or in a tuning file: 9)
  // 11 (k <= 128): 64 x 64 tiles, 256 threads: four 8 x 8 groups over quarters of K, summed in
  //   shared memory
  e = cudaErrorNotSupported;
  if ((config == 9 || config == 5 || config == 6) && d.k <= 64) {
    e = a.beta != 0.0f ? launch_reg8_l<64, 4, true>(a, a_mn, b_mn, st) : launch_reg8_l<64, 6, false>(a, a_mn, b_mn, st);
  } else if (config == 10 && d.k <= 128) {
    e = a.beta != 0.0f ? launch_reg8_l<128, 3, true>(a, a_mn, b_mn, st) : launch_reg8_l<128, 3, false>(a, a_mn, b_mn, st);
  } else if (config == 11 && d.k <= 128) {
    e = launch_ksplit_l<128, 2>(a, a_mn, b_mn, st);
  } else if (config == 4) {
    e = launch_sl<128, 128, 16, 8, 8, 3, 1>(a, a_mn, b_mn, st);
  } else if (config == 7) {
    e = launch_sl<32, 64, 32, 4, 4, 4, 4>(a, a_mn, b_mn, st);
  } else if (config == 8) {
    e = launch_sl<32, 32, 16, 4, 4, 8, 8>(a, a_mn, b_mn, st);
  }
  // configuration 3 serves the rest (and tile counts of 2^31 or more for 9 to 11)
  if (e == cudaErrorNotSupported) e = launch_sl<64, 64, 32, 4, 4, 2, 3>(a, a_mn, b_mn, st);
  note_launch();
  return e;
}

}  // namespace ssb
