// Plain FP64 batched GEMM on the FP64 tensor cores (DMMA: mma.sync.m8n8k4.f64).
//
// The fp64 row of ssblasGemmBatchedEx in its plain (non-emulated) form. Semantics follow the
// reference (hirokitokura/ssblasEx): C <- beta*C, not read when beta == 0
// (src/include/CScale/Xgemm_scale_kernel.hpp:164-176), then C <- C + acc*alpha with one fused
// multiply-add (src/include/GemmCore/Xgemm_kernel_sve_v4x5_1.hpp:93-127). The reference adds
// alpha*acc once per 512-wide K block; here it is added once, which differs only by rounding.
//
// Design: one CTA per (64 x 64 tile, instance). op(A) and op(B) tiles are copied into shared
// memory by cp.async in a STAGES-deep ring (the copies for K step kt + STAGES - 1 are in flight
// while step kt is multiplied), each in the orientation it has in global memory -- the copy
// absorbs op(A)/op(B): an operand whose rows (m or n) are contiguous is staged [k][mn], one whose
// K is contiguous is staged [mn][k]. Each warp owns a WM x WN block of C as (WM/8) x (WN/8)
// DMMA accumulator tiles. Row pitches are 4 (mod 16) doubles, so the fragment loads (lane l reads
// (mn = l/4, k = l%4) of an 8 x 4 block) hit 16 distinct 8-byte bank pairs per half-warp.
//
// 16-byte copies when the instance's base pointer is 16-byte aligned and its ld is even, else
// 8-byte copies; elements outside the matrix are zero-filled by the copy itself (src-size).
#include <cuda_runtime.h>
#include <stdint.h>

#include "dmma_slab.h"
#include "grouped.h"
#include "internal.h"
#include "ptx.cuh"

namespace ssb {
namespace {

struct DmmaArgs {
  long m, n, k, lda, ldb, ldc, batch;
  const double* const* A;
  const double* const* B;
  double* const* C;
  double alpha, beta;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// cp.async of `bytes` valid bytes (0, 8 or 16) into a 16- or 8-byte slot; the rest is zero-filled
struct CpAsync {
  __device__ __forceinline__ void cp16(uint32_t dst, const void* src, int bytes) const {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  }
  __device__ __forceinline__ void cp8(uint32_t dst, const void* src, int bytes) const {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  }
};
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// D (8x8, two per lane) += A (8x4, row) * B (4x8, col)
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

template <int BM, int BN, int BK>
struct DmmaSmem {
  static constexpr int PMN_A = BM + 4;    // [k][m] pitch
  static constexpr int PMN_B = BN + 4;    // [k][n] pitch
  static constexpr int PK = BK + 4;       // [mn][k] pitch
  static constexpr int A_MAX = (BK * PMN_A > BM * PK) ? BK * PMN_A : BM * PK;   // doubles
  static constexpr int B_MAX = (BK * PMN_B > BN * PK) ? BK * PMN_B : BN * PK;
  static constexpr int STAGE = A_MAX + B_MAX;
};

// One BM x BN tile of C = alpha op(A) op(B) + beta C for one instance, by the whole CTA: the K loop
// over the stage ring, then the epilogue. Leaves the stage buffers free (every copy has landed and
// every thread has passed a barrier after its last read).
template <int BM, int BN, int BK, int WM, int WN, int STAGES, bool A_MN, bool B_MN>
__device__ __forceinline__ void dmma_tile(const double* __restrict__ A, const double* __restrict__ B,
                                          double* __restrict__ C, long m, long n, long k, long lda, long ldb,
                                          long ldc, double alpha, double beta, long m0, long n0, double* smem) {
  constexpr int NWM = BM / WM, NWN = BN / WN;
  constexpr int NT = NWM * NWN * 32;
  constexpr int MI = WM / 8, NI = WN / 8;
  using Sm = DmmaSmem<BM, BN, BK>;
  static_assert(Slab<BM, BK, NT, A_MN>::KMAX >= kDmmaMaxK && Slab<BN, BK, NT, B_MN>::KMAX >= kDmmaMaxK, "counts of slabs");
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int wm = warp % NWM, wn = warp / NWM;
  const int fr = lane >> 2, fk = lane & 3;    // fragment row (m or n) and k within an 8x4 block
  Slab<BM, BK, NT, A_MN> ca;
  Slab<BN, BK, NT, B_MN> cb;
  ca.init(A, m, k, lda, m0, threadIdx.x);
  cb.init(B, n, k, ldb, n0, threadIdx.x);

  double acc[MI][NI][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int ktiles = ca.slabs();
  const uint32_t smem0 = smem_addr(smem);
  auto issue = [&](int kt) {     // slabs in order, kt counts them
    const uint32_t sa = smem0 + 8u * (uint32_t)((kt % STAGES) * Sm::STAGE);
    ca.copy(sa, CpAsync{});
    cb.copy(sa + 8u * Sm::A_MAX, CpAsync{});
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ktiles) issue(s);
    cp_commit();
  }
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    if (kt + STAGES - 1 < ktiles) issue(kt + STAGES - 1);
    cp_commit();
    const double* sa = smem + (kt % STAGES) * Sm::STAGE;
    const double* sb = sa + Sm::A_MAX;
#pragma unroll 2
    for (int k4 = 0; k4 < BK / 4; ++k4) {
      const int kk = 4 * k4 + fk;
      double af[MI], bf[NI];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int r = wm * WM + 8 * i + fr;
        af[i] = A_MN ? sa[kk * Sm::PMN_A + r] : sa[r * Sm::PK + kk];
      }
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        const int c = wn * WN + 8 * j + fr;
        bf[j] = B_MN ? sb[kk * Sm::PMN_B + c] : sb[c * Sm::PK + kk];
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) dmma(acc[i][j], af[i], bf[j]);
    }
  }
  cp_wait<0>();
  __syncthreads();   // the next tile's copies reuse the stage buffers

  // epilogue: lane holds C rows m0 + wm*WM + 8i + fr, columns n0 + wn*WN + 8j + 2fk + {0,1}
  const bool read_c = beta != 0.0;
#pragma unroll
  for (int j = 0; j < NI; ++j) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long gj = n0 + wn * WN + 8 * j + 2 * fk + h;
      if (gj >= n) continue;
      double cv[MI];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const long gi = m0 + wm * WM + 8 * i + fr;
        cv[i] = (read_c && gi < m) ? C[gi + gj * ldc] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const long gi = m0 + wm * WM + 8 * i + fr;
        if (gi < m) {
          const double tb = read_c ? beta * cv[i] : 0.0;
          C[gi + gj * ldc] = fma(acc[i][j][h], alpha, tb);
        }
      }
    }
  }
}

// Tiles: 64 x 64, 4 warps of 32 x 32, three 16-deep K slabs in flight (52 KB): with at most 170
// registers a thread three CTAs share an SM, and one's barrier, copies and epilogue run beside the
// others' products. 128 x 128 tiles with one CTA per SM left the FP64 pipe idle a third of the time (every
// warp of the SM at the same barrier) and padded small and ragged sizes more. The pipe's own peak, measured
// with operands in registers, is 36.9 TFLOP/s for every mma.sync f64 shape. Before -> after:
// 32 x 1024^3 NT 2.39 -> 2.05 ms (33.6 TFLOP/s), 64 x (500 x 300 x 700) TN 0.867 -> 0.467 ms,
// 100 x (200 x 150 x 300) NN with odd ld 0.197 -> 0.121 ms, 256 x 128^3 TN 0.0735 -> 0.061 ms.
// Four slabs: 2.10, 0.518, 0.141, 0.073 ms; four CTAs of 128 registers: 2.13, 0.492, 0.124, 0.061 ms.
constexpr int kBM = 64, kBN = 64, kBK = 16, kW = 32, kStages = 3, kMinBlocks = 3;
constexpr int kDmmaThreads = (kBM / kW) * (kBN / kW) * 32;
constexpr int kDmmaSmem = kStages * DmmaSmem<kBM, kBN, kBK>::STAGE * 8;

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kDmmaThreads, kMinBlocks) dmma_gemm_kernel(DmmaArgs args) {
  extern __shared__ __align__(16) double smem[];
  const long tiles_m = (args.m + kBM - 1) / kBM;
  const long m0 = (blockIdx.x % tiles_m) * kBM;
  const long n0 = (blockIdx.x / tiles_m) * kBN;
  for (long b = blockIdx.y; b < args.batch; b += gridDim.y)
    dmma_tile<kBM, kBN, kBK, kW, kW, kStages, A_MN, B_MN>(args.A[b], args.B[b], args.C[b], args.m, args.n, args.k,
                                                         args.lda, args.ldb, args.ldc, args.alpha, args.beta, m0, n0,
                                                         smem);
}

// Grouped form (plain fp64 instances of ssblasGemmGroupedBatchedEx): one CTA per (instance,
// 64 x 64 tile) entry of a tile table whose instances all have this op(A) / op(B) layout.
template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kDmmaThreads, kMinBlocks)
dmma_grouped_kernel(const SimtGInst* __restrict__ inst, const int* __restrict__ tiles, const double* const* A,
                    const double* const* B, double* const* C) {
  extern __shared__ __align__(16) double smem[];
  ptx::grid_dep_launch();
  const int* t = tiles + 3 * (long)blockIdx.x;
  const SimtGInst g = inst[t[0]];
  dmma_tile<kBM, kBN, kBK, kW, kW, kStages, A_MN, B_MN>(A[g.idx], B[g.idx], C[g.idx], g.m, g.n, g.k, g.lda, g.ldb,
                                                       g.ldc, g.alpha_d, g.beta_d, (long)t[1] * kBM,
                                                       (long)t[2] * kBN, smem);
  ptx::grid_chain_end();
}

template <bool A_MN, bool B_MN>
cudaError_t launch_cfg(const DmmaArgs& a, cudaStream_t st) {
  auto kern = dmma_gemm_kernel<A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, kDmmaSmem)) return e;
  const long tiles = ((a.m + kBM - 1) / kBM) * ((a.n + kBN - 1) / kBN);
  if (tiles > 0x7fffffffL) return cudaErrorInvalidValue;
  dim3 grid((unsigned)tiles, (unsigned)(a.batch < 65535 ? a.batch : 65535));
  kern<<<grid, kDmmaThreads, kDmmaSmem, st>>>(a);
  return cudaGetLastError();
}

template <bool A_MN, bool B_MN>
cudaError_t launch_grouped_layout(const GroupedSimt& s, const GroupedPtrs& p, int lay, cudaStream_t st, bool& follows) {
  auto kern = dmma_grouped_kernel<A_MN, B_MN>;
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, kDmmaSmem)) return e;
  note_launch();
  return launch_chained(kern, (unsigned)s.ndmma[lay], kDmmaThreads, kDmmaSmem, st, follows, (const SimtGInst*)s.inst64,
                        (const int*)s.dmma_tiles[lay], (const double* const*)p.A, (const double* const*)p.B,
                        (double* const*)p.C);
}

}  // namespace

// The plain fp64 tiles of a grouped call, one launch per op(A) / op(B) layout present
// (layout index = 2 * (op(A) rows contiguous) + (op(B) columns contiguous)).
cudaError_t launch_dmma_grouped(const GroupedSimt& s, const GroupedPtrs& p, cudaStream_t st, bool& follows) {
  if (!s.ndmma[0] && !s.ndmma[1] && !s.ndmma[2] && !s.ndmma[3]) return cudaSuccess;
  ProfScope prof("dmma_grouped", st);
  cudaError_t e = cudaSuccess;
  for (int lay = 0; lay < 4 && e == cudaSuccess; ++lay) {
    if (!s.ndmma[lay]) continue;
    switch (lay) {
      case 3: e = launch_grouped_layout<true, true>(s, p, lay, st, follows); break;
      case 2: e = launch_grouped_layout<true, false>(s, p, lay, st, follows); break;
      case 1: e = launch_grouped_layout<false, true>(s, p, lay, st, follows); break;
      default: e = launch_grouped_layout<false, false>(s, p, lay, st, follows); break;
    }
  }
  return e;
}

cudaError_t launch_dmma_f64(const BatchDesc& d, cudaStream_t st) {
  DmmaArgs a;
  a.m = d.m; a.n = d.n; a.k = d.k; a.lda = d.lda; a.ldb = d.ldb; a.ldc = d.ldc; a.batch = d.batch;
  a.A = (const double* const*)d.A;
  a.B = (const double* const*)d.B;
  a.C = (double* const*)d.C;
  a.alpha = d.alpha_d;
  a.beta = d.beta_d;
  const bool a_mn = d.transa == SSBLAS_OP_N;   // op(A) rows (m) contiguous
  const bool b_mn = d.transb == SSBLAS_OP_T;   // op(B) columns (n) contiguous
  // One configuration (2 selects the DFMA SIMT kernel, handled by the caller): see the tile constants.
  ProfScope prof("dmma_gemm", st);
  cudaError_t e;
  if (a_mn && b_mn) e = launch_cfg<true, true>(a, st);
  else if (a_mn) e = launch_cfg<true, false>(a, st);
  else if (b_mn) e = launch_cfg<false, true>(a, st);
  else e = launch_cfg<false, false>(a, st);
  note_launch();
  return e;
}

}  // namespace ssb
