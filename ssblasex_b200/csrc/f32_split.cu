// FP32 batched GEMM on the BF16 tensor cores (tcgen05.mma kind::f16), the operands split into BF16
// parts inside the kernel. Two forms of the fp32 row share it:
//   plain (NP = 3)    x = hi + mid + lo exactly (8 + 8 + 8 significand bits), six products
//                     hi hi, hi mid, mid hi, mid mid, hi lo, lo hi: what is left out (mid lo and lo
//                     mid, each up to 2^-25) is at most 2^-24 of a product;
//   3xBF16 (NP = 2)   x ~ hi + lo, three products (the emulation mode of the fp32 row).
// Semantics follow the reference (hirokitokura/ssblasEx): C <- beta*C, not read when beta == 0
// (src/include/CScale/Xgemm_scale_kernel.hpp:164-176), then C <- C + acc*alpha with one fused
// multiply-add (src/include/GemmCore/Xgemm_kernel_sve_v4x5_1.hpp:93-127).
//
// Accuracy of the plain form. The tensor core adds a K step of 16 products and the accumulator
// exactly enough, but truncates the sum to FP32: over a long K that bias would exceed the error of a
// chain of fused multiply-adds (k = 1024, U[-1,1): 1.25e-6 against 5.6e-7 of the 2-norm), and where a
// result is one product, or a few, it would be twice the chain's. So hi hi, whose products have 16 bits, is
// accumulated for one chunk of 32 k only, and the epilogue warps add the chunks in registers, rounding to
// nearest; the smaller products, at most 2^-7 of the magnitudes' sum, have an accumulator of their own for up to
// 32 chunks, which truncates at their magnitude. Measured, 2-norm of the error over that of the result in u =
// 2^-24, a chain / this / all six products in the chunk's accumulator: k = 1024, U[-1,1) 9.6 / 1.9 / 2.0; with 1% of
// outliers 3.3 / 1.9 / 1.9; one nonzero per row 0.42 / 0.43 / 0.76 (the largest error of a product 1.0 / 1.5 / 2.4 u);
// two 0.52 / 0.44 / 0.88; four 0.67 / 0.45 / 1.0; four between 2^-12 and 2^12 0.68 / 0.71 / 1.0. With mid lo and lo
// mid as well, one nonzero per row has the chain's error, and 16 x 1024^3 takes 185 us instead of 156.
// The ends of the range: both operands are scaled by 2^24 before they
// are split (exact, and the lo part of the smallest subnormal is then a BF16 number). Small results need
// nothing else: a sum of 2^-149 is 2^-101 on the accumulator, whose parts down to 2^-24 of it are still ordinary
// FP32 numbers, and it is rounded to FP32's own subnormals once, at the end. Where a sum is not finite (Inf
// and NaN operands, |x| >= 2^104, sums of 2^80 and more) its block of 32 rows is left as it is, and computed
// once the CTA's tiles are done by chains of fused multiply-adds over the operands, so those behave as FP32
// arithmetic does (split_redo).
//
// Design: persistent CTAs over (instance, tile) items, K in chunks of 32:
//   warps 8-15   converters: each thread copies its own 16-byte units of op(A) and op(B), two to four chunks
//                ahead, from the caller's matrices to its own places in shared memory (cp.async; any
//                alignment: 4-byte copies where 16-byte ones are not possible), reads them back, splits
//                them and writes the parts in the layout the tensor core reads -- K-major (64-byte
//                swizzle) where K is contiguous in memory, MN-major (128-byte swizzle) where M or N is, so
//                nothing is transposed
//   warp 16      tensor memory, MMA issue
//   warps 0-7    chunk sums from tensor memory into registers, then alpha * acc + beta * C
// For large tiles two CTAs share a 256 x 256 tile (tcgen05 cta_group::2): each loads, splits and writes
// 128 of its rows and 128 of its columns, half as much per product as alone, and arrives on the leader's
// barriers. Operands cross HBM once as fp32 and no plane is written back: the operands of a tile are split
// again for every tile that shares them, which is cheaper than the 10 bytes per element of a split pass.
// What bounds it (16 x 1024^3 plain, a pair's chunk of 1820 cycles): the 128 B per cycle of shared memory
// (units in and out 64 KB, parts in 48 KB, 12 MMAs reading 96 KB: 1660 cycles; the MMAs alone 1540). With
// the units in registers, as before, the wait for a stage queued behind the loads and a chunk of a 128 x 128
// tile took 1850 cycles; so did one of a pair while its arrivals asked for a cluster-wide release.
// Measured in short bursts (us, FFMA kernels -> this one): 16 x 1024^3 NN 802 -> 154 (223 TFLOP/s; back to back
// 165); 4 x 2048^3 1730 -> 305; 64 x 128^3 NN, beta = 0.5 16.7 -> 12; 200 x (200 x 200 x 300) TT, beta = 1 243 -> 73;
// 2 x 128^2 x 4096 190 -> 99.
// 3xBF16 (split pass and tiled GEMM -> this kernel): 256 x 256^3 0.130 -> 0.039, 16 x 1024^3 0.096; a grouped
// call's 5000 instances of 8 to 512 each way 0.564 -> 0.39.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"
#include "grouped.h"
#include "internal.h"
#include "ptx.cuh"
#include "sgemm_load.cuh"
#include "tile_rules.h"

namespace ssb {
namespace {

constexpr int kKC = 32;                      // K elements per chunk
constexpr int kConvThreads = 256;            // warps 8-15
constexpr int kSplitThreads = 32 * 20;       // the last warpgroup's first warp issues the MMAs
constexpr int kUnitRow = 16 * kConvThreads;  // bytes of one unit of every converter thread
constexpr float kScale = 0x1p24f, kUnscale = 0x1p-48f;   // plain form: of the operands, and of their sums
// Plain form: tiles of a worker per launch, a byte each for the blocks to compute again. (Launches of so many
// tiles take 10 ms and more.)
constexpr uint32_t kRedoTiles = 4096;
constexpr uint32_t kSumChunks = 32;               // plain form: chunks of one accumulator of the smaller products

// NP parts per operand, AR rows of op(A) (64 when m <= 64) and BN columns of op(B) converted per CTA and
// chunk. PAIR: two CTAs (a cluster) share a 256 x 256 tile -- each converts 128 of its rows and 128 of its
// columns and holds 128 rows of the result, and the leader's MMAs (cta_group::2) read both CTAs'
// parts -- so per product a CTA loads, splits, writes and reads half as much.
template <int NP_, int AR_, int BN_, bool PAIR_ = false>
struct Split {
  static constexpr int NP = NP_, AR = AR_, BN = BN_;
  static constexpr bool PAIR = PAIR_;
  static constexpr int A_PLANE = AR * kKC * 2;
  static constexpr int B_PLANE = BN * kKC * 2;
  static constexpr int STAGE = NP * (A_PLANE + B_PLANE);
  static constexpr int UA = AR * kKC / 4 / kConvThreads, UB = BN * kKC / 4 / kConvThreads;   // 16-byte units per thread
  // chunks of fp32 units in flight, and stages of parts, in 224 KB
  static constexpr int RAW_STAGE = (UA + UB) * kUnitRow;
  static constexpr int RAW = RAW_STAGE > 24 * 1024 ? (NP == 3 ? 2 : 3) : 4;
  static constexpr int STAGES = (224 * 1024 - RAW * RAW_STAGE) / STAGE > 6 ? 6 : (224 * 1024 - RAW * RAW_STAGE) / STAGE;
  static constexpr int TM = PAIR ? 256 : 128, TN = PAIR ? 2 * BN : BN;   // the tile
  static constexpr bool PROMOTE = NP == 3;
  // accumulators in flight, TN columns each: NACC of a tile (3xBF16), or of a chunk's hi hi (plain), where NSUM more
  // hold the smaller products. A pair's single ones cost nothing, since the smaller products of the next chunk run
  // while hi hi is read; a 128 x 128 tile has three, so that the next tile is under way during this one's end
  // (two and two: 100 x 256^3 31 -> 33 us, 74 x (256 x 256 x 128) 15.0 -> 15.7).
  static constexpr int NACC = PROMOTE ? (PAIR ? 1 : TN == 128 ? 3 : 6) : PAIR ? 2 : 4;
  static constexpr int NSUM = !PROMOTE ? 0 : TN == 64 ? 2 : 1;
  static constexpr int SUMS = PROMOTE ? NSUM : 1;   // (to count them by, also in code that does not run)
  static constexpr int TMEM_COLS = (NACC + NSUM) * TN;
  // registers per thread: 640 threads x 96 at launch = 61,440 for 256 converters, 256 epilogue threads (the
  // plain form's hold a sum per output, 128 a thread in a pair) and the 128 of the issuing warp's warpgroup (32
  // made that warp's loop of the plain form spill: 2 x 128^2 x 4096 101 -> 107 us)
  static constexpr int ISSUE_REGS = PROMOTE && !PAIR ? 40 : 32;
  static constexpr int CONV_REGS = !PROMOTE ? 104 : PAIR ? 56 : TN == 128 ? 80 : 104;
  static constexpr int EPI_REGS = (ISSUE_REGS > 32 ? 216 : 224) - CONV_REGS;
  // the MMA reads 128 rows of every A part: with AR = 64 the upper 64 come from whatever follows
  // (within the stage, since B follows A), and their products are never read
  static constexpr int SMEM = 1024 + STAGES * STAGE + RAW * RAW_STAGE + 512;
  static_assert(STAGE % 1024 == 0 && NP * B_PLANE >= 4096 && SMEM <= 232448, "stages");
  static_assert(TMEM_COLS == 256 || TMEM_COLS == 512, "tensor memory comes in powers of two");
  static_assert(256 * (CONV_REGS + EPI_REGS) + 128 * ISSUE_REGS <= kSplitThreads * 96, "registers");
};

// One tile of a grouped launch as a worker's warps see it: its record and its instance's matrices. A
// scheduler warp reads both up to kRing tiles ahead of the others, eight at a time (a lane per tile, so a
// batch costs one chain of dependent loads), into a ring in shared memory.
struct SplitItem {
  SplitRec r;
  const float* A;
  const float* B;
  float* C;
  int valid, pad;            // valid = 0 ends the worker's tiles
};
constexpr uint32_t kRing = 16;

struct SplitArgs {
  long m, n, k, lda, ldb, ldc;
  const float* const* A;
  const float* const* B;
  float* const* C;
  float alpha, beta;
  int a_mn, b_mn;          // op(A) rows / op(B) columns contiguous in memory
  uint32_t tiles_m, tiles_mn, first, total;   // of this launch: tiles [first, first + total)
  int* err;
  uint32_t wait_limit;
  int skip;                // injected fault: CTA 0 never signals its first chunk
  const SplitRec* recs;    // grouped launches: one per tile
};

// One work item: the tile at (m0, n0) of instance b.
struct SplitTile {
  uint32_t b;
  long m0, n0;
};
template <class F>
__device__ __forceinline__ SplitTile split_tile(const SplitArgs& a, uint32_t t) {
  const uint32_t b = (a.first + t) / a.tiles_mn, r = a.first + t - b * a.tiles_mn;
  const uint32_t nt = r / a.tiles_m;
  return {b, (long)(r - nt * a.tiles_m) * F::TM, (long)nt * F::TN};
}

// One operand as a converter thread sees it: its unit i (4 consecutive elements along the contiguous
// dimension) of the next chunk is at p + i * step.
//   mn: a unit is 4 rows at one k; a warp takes whole k lines of ROWS; unit i is 256 / (ROWS / 4) k on
//   else a unit is 4 k of one row, 8 lanes a row; unit i is 32 rows on
struct SplitOperand {
  const float *p, *base;
  int step, adv;           // elements between units, between chunks (ld < 2^25)
  int rows, k;             // valid rows from this thread's unit 0 on; valid k from the next chunk on
  int units, bytes;        // units with a row inside the matrix, and the valid bytes of one inside K
  bool mn, vec, full;      // full: every unit of the tile's whole chunks is inside the matrix
};
// A thread's units with a row inside the matrix, `rows` of which are left from its unit 0 on.
template <int ROWS>
__device__ __forceinline__ int split_units(int rows, bool mn) {
  constexpr int U = ROWS * kKC / 4 / kConvThreads;
  return rows <= 0 ? 0 : mn ? U : min(U, (rows + 31) / 32);
}
template <int ROWS>
__device__ __forceinline__ SplitOperand split_operand(const float* X, long rows, long K, long ld, bool mn, long r0,
                                                      int t) {
  constexpr int RG = ROWS / 4;
  SplitOperand o;
  o.base = X;
  o.mn = mn;
  o.vec = ((uintptr_t)X % 16) == 0 && ld % 4 == 0;
  o.full = o.vec && rows - r0 >= ROWS;
  const int rr = mn ? 4 * (t % RG) : t / 8, kk = mn ? t / RG : 4 * (t % 8);
  o.p = X + (mn ? r0 + rr + kk * ld : (r0 + rr) * ld + kk);
  o.step = (mn ? kConvThreads / RG : 32) * (int)ld;
  o.adv = mn ? kKC * (int)ld : kKC;
  o.rows = (int)(rows - r0 < ROWS ? rows - r0 : ROWS) - rr;
  o.k = (int)K;
  o.units = split_units<ROWS>(o.rows, mn);
  o.bytes = mn && o.rows < 4 ? 4 * o.rows : 16;
  return o;
}

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy16_if(bool on, uint32_t dst, const float* src, int bytes) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %3, 0;\n@p cp.async.cg.shared.global [%0], [%1], 16, %2;\n}" ::"r"(dst),
               "l"(src), "r"(bytes), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
// Copies the units of the next chunk to this thread's places, unit i at dst + i * 4096 (zeros outside the
// matrix); the operand moves on to the chunk after it. SKIP: units past the matrix's rows stay as they are.
template <int ROWS, int U, bool SKIP>
__device__ __forceinline__ void split_copy(SplitOperand& o, int t, uint32_t dst) {
  constexpr int RG = ROWS / 4;
  const float* src = o.p;
  if (o.full && o.k >= kKC) {
#pragma unroll
    for (int i = 0; i < U; ++i, src += o.step) copy16(dst + i * kUnitRow, src, 16);
  } else if (SKIP && o.vec && o.k >= kKC) {
#pragma unroll
    for (int i = 0; i < U; ++i, src += o.step)
      copy16_if(i < o.units, dst + i * kUnitRow, src, o.bytes);
  } else {
#pragma unroll
    for (int i = 0; i < U; ++i, src += o.step) {
      if (SKIP && i >= o.units) break;
      const int kk = o.mn ? t / RG + i * (kConvThreads / RG) : 4 * (t % 8);
      int n = o.mn ? (o.k > kk ? o.rows : 0) : (o.rows > 32 * i ? o.k - kk : 0);   // valid elements
      n = n < 0 ? 0 : n > 4 ? 4 : n;
      const float* q = n > 0 ? src : o.base;
      if (o.vec) {
        copy16(dst + i * kUnitRow, q, 4 * n);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) copy4(dst + i * kUnitRow + 4 * e, n > e ? q + e : q, n > e);
      }
    }
  }
  o.p += o.adv;
  o.k -= kKC;
}

// Two values rounded to bf16 (low half = first), and (REST) what rounding left of them.
template <bool REST>
__device__ __forceinline__ uint32_t take_bf16(uint64_t& v) {
  float x, y;
  unpack2(v, x, y);
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const uint32_t w = *(const uint32_t*)&h;
  if (REST) v = fma2(pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), pack2(-1.f, -1.f), v);
  return w;
}

// Splits this thread's units (unit i at raw + i * 4096; SOME: the first `units` of them) and writes the NP
// parts of the operand.
template <int NP, int ROWS, int U, bool SOME>
__device__ __forceinline__ void split_store(uint32_t raw, uint32_t dst, bool mn, int t, int units) {
  constexpr int PLANE = ROWS * kKC * 2;
  constexpr int RG = ROWS / 4;
  uint32_t off, step;
  if (mn) {
    // blocks of 64 rows x 32 k lines of 128 bytes; lines kk, kk + 8q: the swizzle (kk % 8) is fixed
    const uint32_t rg = t % RG, kk = t / RG;
    off = (rg >> 4) * (kKC * 128u) + kk * 128u + ((((rg & 15u) >> 1) ^ (kk & 7u)) << 4) + ((rg & 1u) << 3);
    step = (kConvThreads / RG) * 128u;
  } else {
    // lines of 64 bytes; rows rr + 32 i: the swizzle ((rr / 2) % 4) is fixed
    const uint32_t rr = t / 8, kq = t % 8;
    off = rr * 64u + (((kq >> 1) ^ ((rr >> 1) & 3u)) << 4) + ((kq & 1u) << 3);
    step = 32 * 64u;
  }
  // all reads before the first write: the units' conversions then overlap. (SOME: by predicates, since a
  // branch per unit would take that overlap away and measured 1.8 times as long on whole tiles)
  uint64_t v[U][2] = {};
#pragma unroll
  for (int i = 0; i < U; ++i)
    if (SOME)
      asm volatile("{\n.reg .pred p;\nsetp.lt.s32 p, %3, %4;\n@p ld.shared.v2.b64 {%0, %1}, [%2];\n}"
                   : "+l"(v[i][0]), "+l"(v[i][1])
                   : "r"(raw + i * kUnitRow), "r"(i), "r"(units)
                   : "memory");
    else
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[i][0]), "=l"(v[i][1]) : "r"(raw + i * kUnitRow) : "memory");
  if constexpr (NP == 3) {
#pragma unroll
    for (int i = 0; i < U; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) v[i][h] = mul2(v[i][h], pack2(kScale, kScale));
  }
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    uint32_t w[U][2];
#pragma unroll
    for (int i = 0; i < U; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) w[i][h] = p + 1 < NP ? take_bf16<true>(v[i][h]) : take_bf16<false>(v[i][h]);
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (SOME)
        asm volatile("{\n.reg .pred p;\nsetp.lt.s32 p, %3, %4;\n@p st.shared.v2.b32 [%0], {%1, %2};\n}" ::"r"(
                         dst + off + i * step + p * PLANE),
                     "r"(w[i][0]), "r"(w[i][1]), "r"(i), "r"(units)
                     : "memory");
      else
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + off + i * step + p * PLANE), "r"(w[i][0]), "r"(w[i][1])
                     : "memory");
  }
}

// The flagged blocks of one tile again, by the 256 epilogue threads: C <- alpha * acc + beta * C with acc a chain
// of fused multiply-adds in k order. Block w (bit w of `flags`) is what epilogue warp w left unwritten: rows
// 32 (w % 4) of the CTA's ROWS from m0 on, columns HALF (w / 4) from n0 on. FFMA tiles of ROWS x 128 (64) in the
// shared memory that the tensor-core pipeline no longer uses, slabs of 32 k, four in flight; a thread has 8 (4)
// columns and rows in groups of four, 64 apart.
// Measured (us, the whole call; before: a chain per output in the epilogue, a load for every product): all of C out of
// range 16 x 1024^3 7710 -> 1130 (the FFMA kernels 800, in range 152), 200 x (200 x 200 x 300) 1960 -> 460 (243, 74);
// an Inf in one row of each matrix 16 x 1024^3 4300 -> 645. With 4 columns a thread everywhere 1435.
template <int ROWS, int HALF>
__device__ __forceinline__ void split_redo(const SplitArgs& a, uint32_t b, long m0, long n0, uint32_t flags, float* sm) {
  constexpr int BK = 32, ST = 4, NC = HALF < 64 ? 64 : 128, TM = ROWS / 16, TN = NC / 16, PA = ROWS + 4, PB = NC + 4;
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int tx = (warp % 2) * 8 + lane % 8, ty = (warp / 2) * 4 + lane / 8;   // a warp: 8 (rows) x 4 (columns)
  const float *A = a.A[b], *B = a.B[b];
  const bool vecA = (uintptr_t)A % 16 == 0 && a.lda % 4 == 0, vecB = (uintptr_t)B % 16 == 0 && a.ldb % 4 == 0;
  const int slabs = (int)((a.k + BK - 1) / BK);
#pragma unroll 1
  for (int c0 = 0; c0 < 2 * HALF; c0 += NC) {
    if (HALF == NC && ((flags >> (4 * (c0 / HALF))) & 0xfu) == 0) continue;
    auto load = [&](int i) {
      float* sa = sm + (i % ST) * BK * (PA + PB);
      if (a.a_mn) sload<ROWS, BK, 256, true>(sa, A, a.m, a.k, a.lda, m0, (long)i * BK, vecA);
      else sload<ROWS, BK, 256, false>(sa, A, a.m, a.k, a.lda, m0, (long)i * BK, vecA);
      if (a.b_mn) sload<NC, BK, 256, true>(sa + BK * PA, B, a.n, a.k, a.ldb, n0 + c0, (long)i * BK, vecB);
      else sload<NC, BK, 256, false>(sa + BK * PA, B, a.n, a.k, a.ldb, n0 + c0, (long)i * BK, vecB);
    };
    uint64_t acc2[TM / 2][TN] = {};
#pragma unroll 1
    for (int i = 1 - ST; i < slabs; ++i) {     // (the loads once in the code)
      if (i >= 0) {
        wait_s<ST - 2>();
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      if (i + ST - 1 < slabs) load(i + ST - 1);
      commit_s();
      if (i < 0) continue;
      const float* sa = sm + (i % ST) * BK * (PA + PB);
      const float* sb = sa + BK * PA;
#pragma unroll 4
      for (int kk = 0; kk < BK; ++kk) outer2<TM, TN, 64>(acc2, sa + kk * PA + 4 * tx, sb + kk * PB + TN * ty);
    }
    wait_s<0>();
    asm volatile("bar.sync 1, 256;" ::: "memory");   // the next columns' copies reuse the buffers
    float acc[TM][TN];
    unpack_acc<TM, TN>(acc2, acc);
#pragma unroll
    for (int h = 0; h < TM / 4; ++h) {
      const int row = 64 * h + 4 * tx, col = c0 + TN * ty;
      if (!((flags >> (4 * (col / HALF) + row / 32)) & 1u)) continue;
      float* C = a.C[b] + m0 + row + (n0 + col) * a.ldc;
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (m0 + row + i < a.m && n0 + col + j < a.n) {
            float* p = C + i + j * a.ldc;
            *p = fmaf(acc[4 * h + i][j], a.alpha, a.beta != 0.0f ? a.beta * *p : 0.0f);
          }
    }
  }
}

// GROUPED: the tiles, their shapes and scalars come from a.recs. What bounds it on mixed small shapes (8 to 512
// each way: 875 MB in 0.39 ms, 2.2 TB/s) is the converters' own instructions, 1 us a chunk whether it is
// whole or not: a second group of converter warps (which took them below 64 registers) made it 1.8 times
// as long, so the units of rows outside the matrix are left out instead (0.403 -> 0.390 ms).
template <class F, bool GROUPED>
__global__ void __launch_bounds__(kSplitThreads, 1) f32_split_kernel(const SplitArgs a, const SplitArgs again) {
  static_assert(!GROUPED || (!F::PAIR && !F::PROMOTE), "grouped launches: 3xBF16, one CTA per tile");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* stages = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* raw = stages + F::STAGES * F::STAGE;                  // [RAW] fp32 units, a place per thread
  uint64_t* full = (uint64_t*)(raw + F::RAW * F::RAW_STAGE);     // parts written (converter warps)
  uint64_t* empty = full + F::STAGES;                            // parts read by the MMAs (commit)
  uint64_t* acc_full = empty + F::STAGES;                        // [NACC] sums complete (commit)
  uint64_t* acc_empty = acc_full + F::NACC;                      // [NACC] sums read (8 warps)
  uint64_t* sum_empty = acc_empty + F::NACC;                     // [NSUM] smaller products read (8 warps)
  uint64_t* drain = sum_empty + F::NSUM;
  uint64_t* ring_full = drain + 1;                               // [kRing] record written (scheduler)
  uint64_t* ring_empty = ring_full + kRing;                      // [kRing] record read (17 warps)
  uint32_t* tmem_slot = (uint32_t*)(ring_empty + kRing);
  SplitItem* ring = (SplitItem*)((uint8_t*)full + 512);
  uint32_t* redo = (uint32_t*)((uint8_t*)full + 512);            // plain form: a byte per tile of this worker
  static_assert((2 * F::STAGES + 2 * F::NACC + F::NSUM + 1 + 2 * kRing) * 8 + 4 <= 512, "barrier area");

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint32_t wl = a.wait_limit ? a.wait_limit : ptx::kWaitLimit;
  int* err = a.err;
  // this CTA's place: worker `me` of `workers` (a worker is a CTA or a pair), rank in the pair
  constexpr uint32_t CT = F::PAIR ? 2 : 1;
  const uint32_t rank = F::PAIR ? ptx::cluster_rank() : 0;
  const uint32_t me = blockIdx.x / CT, workers = gridDim.x / CT;
  if (threadIdx.x == 0) {
    for (int s = 0; s < F::STAGES; ++s) {
      ptx::mbar_init(ptx::smem_u32(&full[s]), CT * kConvThreads / 32);
      ptx::mbar_init(ptx::smem_u32(&empty[s]), 1);
    }
    for (int q = 0; q < F::NACC; ++q) {
      ptx::mbar_init(ptx::smem_u32(&acc_full[q]), 1);
      ptx::mbar_init(ptx::smem_u32(&acc_empty[q]), CT * 8);
    }
    for (int q = 0; q < F::NSUM; ++q) ptx::mbar_init(ptx::smem_u32(&sum_empty[q]), CT * 8);
    ptx::mbar_init(ptx::smem_u32(drain), 1);
    if (GROUPED) {
      for (uint32_t q = 0; q < kRing; ++q) {
        ptx::mbar_init(ptx::smem_u32(&ring_full[q]), 1);
        ptx::mbar_init(ptx::smem_u32(&ring_empty[q]), 17);
      }
    }
    ptx::fence_mbar_init();
  }
  if constexpr (F::PROMOTE) {
    const uint32_t mine = (a.total - me + workers - 1) / workers;   // (a worker has a tile at least)
    for (uint32_t i = threadIdx.x; i < (mine + 3) / 4; i += kSplitThreads) redo[i] = 0;
  }
  if (warp == 16) {
    if constexpr (F::PAIR) {
      ptx::tmem_alloc_pair(ptx::smem_u32(tmem_slot), F::TMEM_COLS);
    } else {
      ptx::tmem_alloc(ptx::smem_u32(tmem_slot), F::TMEM_COLS);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (F::PAIR) ptx::cluster_sync();   // both CTAs' barriers and tensor memory are there
  ptx::tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);   // known to be warp-uniform
  // under a programmatic launch the set-up above overlaps the end of the kernel before
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const uint32_t nkc_all = (uint32_t)((a.k + kKC - 1) / kKC);   // chunks of every tile of a batched launch
  // a wait that all lanes of a warp pass or all give up, converged: what follows is the whole warp's
  // (tensor-memory loads, __syncwarp)
  auto wait_warp = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
    return __all_sync(0xffffffffu, ptx::mbar_wait(ptx::smem_u32(bar), parity, err, code, wl));
  };
  // the worker's i-th tile: whether there is one (grouped: once its record has arrived)
  auto tile_ready = [&](uint32_t i, int code) -> bool {
    if constexpr (GROUPED) {
      const uint32_t q = i % kRing;
      return wait_warp(&ring_full[q], (i / kRing) & 1, code) && ring[q].valid;
    } else {
      return me + i * workers < a.total;
    }
  };

  // a pair's `full` and `acc_empty` are the leader's, and collect both CTAs' arrivals
  auto arrive = [&](uint64_t* bar) {
    if constexpr (F::PAIR) ptx::mbar_arrive_at(ptx::smem_u32(bar), 0);
    else ptx::mbar_arrive(ptx::smem_u32(bar));
  };

  if (warp >= 8 && warp < 16) {
    // ------------------------------------------------------------------ converters --------
    if constexpr (F::CONV_REGS > 96) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F::CONV_REGS));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F::CONV_REGS));
    const int t = threadIdx.x - 256;
    const uint32_t stages0 = ptx::smem_u32(stages);
    const uint32_t raw0 = ptx::smem_u32(raw) + 16 * t;
    // next chunk to copy: tile, chunk of it, place
    uint32_t li = 0, lkc = 0, lr = 0;
    uint32_t lnkc = nkc_all;               // chunks of that tile
    bool more = true;                      // there is such a tile
    SplitOperand A, B;
    auto enter = [&]() {
      more = tile_ready(li, 88);
      if (!more) return;
      if constexpr (GROUPED) {
        const SplitItem& it = ring[li % kRing];
        A = split_operand<F::AR>(it.A, it.r.m, it.r.k, it.r.lda, it.r.a_mn != 0, it.r.m0, t);
        B = split_operand<F::BN>(it.B, it.r.n, it.r.k, it.r.ldb, it.r.b_mn != 0, it.r.n0, t);
        lnkc = (uint32_t)it.r.nkc;
      } else {
        const SplitTile ti = split_tile<F>(a, me + li * workers);
        A = split_operand<F::AR>(a.A[ti.b], a.m, a.k, a.lda, a.a_mn != 0, ti.m0 + rank * 128, t);
        B = split_operand<F::BN>(a.B[ti.b], a.n, a.k, a.ldb, a.b_mn != 0, ti.n0 + rank * F::BN, t);
      }
    };
    auto copy = [&]() {
      if (more) {
        const uint32_t dst = raw0 + lr * F::RAW_STAGE;
        split_copy<F::AR, F::UA, GROUPED>(A, t, dst);
        split_copy<F::BN, F::UB, GROUPED>(B, t, dst + F::UA * kUnitRow);
        if (++lkc == lnkc) {
          lkc = 0;
          ++li;
          enter();
        }
      }
      if (++lr == F::RAW) lr = 0;
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    enter();
#pragma unroll
    for (int d = 0; d < F::RAW; ++d) copy();
    uint32_t c = 0, s = 0, r = 0;
    bool ok = true;
    for (uint32_t i = 0; ok && (i < li || more); ++i) {   // the copies are at tile i or past it
      bool amn = a.a_mn != 0, bmn = a.b_mn != 0;
      uint32_t nkc = nkc_all;
      // a grouped call's tiles are often mostly outside their matrices: what stands in the rows past one
      // (any bits) reaches only results that are not stored
      int ua = F::UA, ub = F::UB;
      if constexpr (GROUPED) {
        const SplitItem& it = ring[i % kRing];
        ua = split_units<F::AR>(it.r.m - it.r.m0 - (it.r.a_mn ? 4 * (t % (F::AR / 4)) : t / 8), it.r.a_mn != 0);
        ub = split_units<F::BN>(it.r.n - it.r.n0 - (it.r.b_mn ? 4 * (t % (F::BN / 4)) : t / 8), it.r.b_mn != 0);
        amn = it.r.a_mn != 0;
        bmn = it.r.b_mn != 0;
        nkc = (uint32_t)it.r.nkc;
      }
      for (uint32_t kc = 0; kc < nkc; ++kc, ++c) {
        // the stage is waited for before the next copies are queued: behind them the answer would take
        // hundreds of cycles
        if (!wait_warp(&empty[s], ((c / F::STAGES) & 1) ^ 1, 81)) {
          ok = false;
          break;
        }
        if (c > 0) copy();                   // into the place of the chunk before, which this thread has read
        asm volatile("cp.async.wait_group %0;" ::"n"(F::RAW - 1) : "memory");   // (each thread reads its own units)
        const uint32_t st = stages0 + s * F::STAGE, rw = raw0 + r * F::RAW_STAGE;
        split_store<F::NP, F::AR, F::UA, GROUPED>(rw, st, amn, t, ua);
        split_store<F::NP, F::BN, F::UB, GROUPED>(rw + F::UA * kUnitRow, st + F::NP * F::A_PLANE, bmn, t, ub);
        ptx::fence_proxy_async_smem();   // generic-proxy writes -> the tensor core's reads
        __syncwarp();
        if (lane == 0 && !(a.skip && c == 0 && blockIdx.x == 0)) arrive(&full[s]);
        if (++s == F::STAGES) s = 0;
        if (++r == F::RAW) r = 0;
      }
      if constexpr (GROUPED) {
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&ring_empty[i % kRing]));
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // no copy is in flight when the CTA exits
  } else if (warp >= 16) {
    // ------------------------------------------------------------------ MMA ---------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F::ISSUE_REGS));
    if (warp == 16 && rank == 0) {
      // descriptors of stage 0's first part, and their step along K: 16 k are 32 bytes of a K-major
      // line, 16 lines of an MN-major block (addresses count 16 bytes). The whole warp runs the loop
      // and one lane's predicate is on the MMA itself, so descriptors stay in uniform registers:
      // under a branch on the lane each MMA cost four moves into them, 90 cycles a MMA.
      const uint32_t lead = ptx::elect_one();
      const uint32_t st0 = ptx::smem_u32(stages);
      static_assert(kKC == 32, "two K steps per chunk");
      uint32_t c = 0, q = 0, sq = 0;   // chunks, accumulators, accumulators of the smaller products
      bool ok = true;
      auto commit = [&](uint64_t* bar) {
        if constexpr (F::PAIR) ptx::mma_commit_pair_if(lead, ptx::smem_u32(bar));
        else ptx::mma_commit_if(lead, ptx::smem_u32(bar));
      };
      for (uint32_t i = 0; ok && tile_ready(i, 89); ++i) {
        bool amn = a.a_mn != 0, bmn = a.b_mn != 0;
        uint32_t nkc = nkc_all;
        if constexpr (GROUPED) {
          const SplitItem& it = ring[i % kRing];
          amn = __shfl_sync(0xffffffffu, it.r.a_mn, 0) != 0;
          bmn = __shfl_sync(0xffffffffu, it.r.b_mn, 0) != 0;
          nkc = (uint32_t)__shfl_sync(0xffffffffu, it.r.nkc, 0);
          if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&ring_empty[i % kRing]));
        }
        const uint32_t idesc = ptx::idesc_bf16(F::TM, F::TN, amn, bmn);
        const uint64_t a0 = amn ? ptx::smem_desc_mnmajor(st0, kKC * 128) : ptx::smem_desc_kmajor(st0, 64);
        const uint64_t b0 = bmn ? ptx::smem_desc_mnmajor(st0 + F::NP * F::A_PLANE, kKC * 128)
                                : ptx::smem_desc_kmajor(st0 + F::NP * F::A_PLANE, 64);
        const uint32_t ka = amn ? 128 : 2, kb = bmn ? 128 : 2;
        for (uint32_t kc = 0; kc < nkc; ++kc, ++c) {
          const uint32_t s = c % F::STAGES;
          // (plain: the smaller products have accumulators of their own, read once in kSumChunks; the one
          // accumulator of a pair for hi hi is waited for behind them)
          bool free = true;
          if (F::PROMOTE && kc % kSumChunks == 0)
            free = ptx::mbar_wait(ptx::smem_u32(&sum_empty[sq % F::SUMS]),
                                  ((sq / F::SUMS) & 1) ^ 1, err, 86, wl);
          if (F::PROMOTE ? F::NACC > 1 : kc == 0)
            free = free && ptx::mbar_wait(ptx::smem_u32(&acc_empty[q % F::NACC]), ((q / F::NACC) & 1) ^ 1, err, 82, wl);
          if (!free) {
            ok = false;
            break;
          }
          if (!ptx::mbar_wait(ptx::smem_u32(&full[s]), (c / F::STAGES) & 1, err, 83, wl)) {
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          // (the low words: the addresses in them do not carry into the high ones)
          const uint32_t sa = (uint32_t)a0 + s * (uint32_t)(F::STAGE >> 4), sb = (uint32_t)b0 + s * (uint32_t)(F::STAGE >> 4);
          auto word = [](uint32_t lo, uint64_t base) { return (base & 0xffffffff00000000ull) | lo; };
          const uint32_t d = tmem + (q % F::NACC) * F::TN;
          const uint32_t ds = F::PROMOTE ? tmem + (F::NACC + sq % F::SUMS) * F::TN : d;
          uint32_t acc = (F::PROMOTE ? kc % kSumChunks : kc) == 0 ? 0u : 1u;
          // smallest products first
#pragma unroll
          for (int sum = F::NP - 1; sum >= 0; --sum) {
            if (F::PROMOTE && sum == 0) {
              if constexpr (F::NACC == 1) {
                if (!ptx::mbar_wait(ptx::smem_u32(&acc_empty[0]), (q & 1) ^ 1, err, 82, wl)) ok = false;
                ptx::tc_fence_after();
              }
              acc = 0u;
            }
#pragma unroll
            for (int p = 0; p <= sum; ++p) {
              const uint32_t ad = sa + (uint32_t)(p * (F::A_PLANE >> 4)), bd = sb + (uint32_t)((sum - p) * (F::B_PLANE >> 4));
              if constexpr (F::PAIR) {
                ptx::mma_f16_pair_if(lead, sum ? ds : d, word(ad, a0), word(bd, b0), idesc, acc);
                ptx::mma_f16_pair_if(lead, sum ? ds : d, word(ad + ka, a0), word(bd + kb, b0), idesc, 1u);
              } else {
                ptx::mma_f16_if(lead, sum ? ds : d, word(ad, a0), word(bd, b0), idesc, acc);
                ptx::mma_f16_if(lead, sum ? ds : d, word(ad + ka, a0), word(bd + kb, b0), idesc, 1u);
              }
              acc = 1u;
            }
          }
          if (F::PROMOTE && (kc % kSumChunks == kSumChunks - 1 || kc + 1 == nkc)) ++sq;
          if (!ok) break;
          commit(&empty[s]);
          if (F::PROMOTE || kc + 1 == nkc) {
            commit(&acc_full[q % F::NACC]);
            ++q;
          }
        }
      }
      // every MMA issued has finished before the tensor memory is released
      commit(drain);
      ptx::mbar_wait(ptx::smem_u32(drain), 0, err, 84, wl);
    } else if (warp == 16) {
      ptx::mbar_wait(ptx::smem_u32(drain), 0, err, 84, wl);   // the leader's last arrival here
    } else if (GROUPED && warp == 17) {
      // ---------------------------------------------------------------- scheduler ---------
      constexpr uint32_t kBatch = kRing / 2;
      for (uint32_t i = 0;; i += kBatch) {
        const uint32_t rec = i + lane, q = rec % kRing, t = me + rec * workers;
        bool last = false;
        if (lane < kBatch) {
          last = !ptx::mbar_wait(ptx::smem_u32(&ring_empty[q]), ((rec / kRing) & 1) ^ 1, err, 80, wl) || t >= a.total;
          SplitItem& it = ring[q];
          if (!last) {
            it.r = a.recs[t];
            it.A = a.A[it.r.idx];
            it.B = a.B[it.r.idx];
            it.C = a.C[it.r.idx];
          }
          it.valid = last ? 0 : 1;
          ptx::mbar_arrive(ptx::smem_u32(&ring_full[q]));
        }
        if (__any_sync(0xffffffffu, last)) break;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue ----------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F::EPI_REGS));
    constexpr int HALF = F::TN / 2;
    const int quarter = warp % 4, half = warp / 4;
    const uint32_t t_row = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * HALF);
    const bool active = quarter * 32 < F::AR;      // rows past AR hold no results
    uint32_t q = 0, sq = 0;
    bool ok = true;
    for (uint32_t i = 0; ok && tile_ready(i, 90); ++i) {
      long gi = rank * 128 + quarter * 32 + lane, gj0 = half * HALF, m = a.m, n = a.n, ldc = a.ldc;
      float alpha = a.alpha, beta = a.beta;
      float* C;
      uint32_t b = 0;
      if constexpr (GROUPED) {
        const SplitItem& it = ring[i % kRing];
        gi += it.r.m0;
        gj0 += it.r.n0;
        m = it.r.m;
        n = it.r.n;
        ldc = it.r.ldc;
        alpha = it.r.alpha;
        beta = it.r.beta;
        C = it.C;
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&ring_empty[i % kRing]));
      } else {
        const SplitTile ti = split_tile<F>(a, me + i * workers);
        b = ti.b;
        gi += ti.m0;
        gj0 += ti.n0;
        C = a.C[b];
      }
      C += gi + gj0 * ldc;
      const bool row_ok = active && gi < m;
      const int cols = gj0 < n ? (n - gj0 < HALF ? (int)(n - gj0) : HALF) : 0;
      const bool read_c = beta != 0.0f;
      if constexpr (GROUPED) {
        // the next tile's C: short tiles leave the reads no other time to cross HBM
        if (tile_ready(i + 1, 91) && ring[(i + 1) % kRing].r.beta != 0.0f) {
          const SplitItem& nx = ring[(i + 1) % kRing];
          const int r0 = nx.r.m0 + quarter * 32, c0 = nx.r.n0 + half * HALF;
#pragma unroll
          for (int h = 0; h < HALF; h += 32)
            if (r0 < nx.r.m && c0 + h + lane < nx.r.n) ptx::prefetch_l2(nx.C + r0 + (c0 + h + lane) * nx.r.ldc);
        }
      }
      // narrow tiles, and those of one accumulator: C is in flight while the products run
      constexpr bool EARLY_C = HALF == 32;
      constexpr int G = EARLY_C || !F::PROMOTE ? 32 : 16;     // columns per group
      float cv[G];
      // (the walking pointers are opaque to the compiler: it would keep an address per column otherwise)
      // columns and rows past the matrix repeat its last ones: a predicate per column had made the reads of
      // ragged tiles most of their time (us: 500 x (60 x 60 x 140) 43 -> 34, 1000 x (48 x 48 x 128) 63 -> 48)
      const int back = gi < m ? 0 : (int)(gi - (m - 1));
      auto load_c = [&](int j0) {
        if (!active || j0 >= cols) return;
        const float* cp = C - back + (long)j0 * ldc;
        asm volatile("" : "+l"(cp));
        if (cols >= j0 + G) {
#pragma unroll
          for (int j = 0; j < G; ++j, cp += ldc) cv[j] = __ldcs(cp);
        } else {
#pragma unroll
          for (int j = 0; j < G; ++j) {
            cv[j] = __ldcs(cp);
            if (j0 + j + 1 < cols) cp += ldc;
          }
        }
      };
      if ((EARLY_C || !F::PROMOTE) && read_c) load_c(0);
      if constexpr (!F::PROMOTE) {
        // one accumulator per tile: groups of columns straight from it to C
        const uint32_t buf = q % F::NACC;
        if (!wait_warp(&acc_full[buf], (q / F::NACC) & 1, 85)) break;
        ptx::tc_fence_after();
        if (active && gi - lane < m) {
#pragma unroll 1
          for (int g = 0; g < cols; g += G) {
            uint32_t raw[G / 16][16];
#pragma unroll
            for (int h = 0; h < G / 16; ++h) ptx::tmem_ld16(t_row + buf * F::TN + g + 16 * h, raw[h]);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < G; ++j)
              raw[j / 16][j % 16] =
                  __float_as_uint(fmaf(__uint_as_float(raw[j / 16][j % 16]), alpha, read_c ? beta * cv[j] : 0.0f));
            if (read_c && g + G < cols) load_c(g + G);
            if (row_ok) {
              float* cp = C + (long)g * ldc;
              asm volatile("" : "+l"(cp));
              if (cols >= g + G) {
#pragma unroll
                for (int j = 0; j < G; ++j, cp += ldc) __stcs(cp, __uint_as_float(raw[j / 16][j % 16]));
              } else {
#pragma unroll
                for (int j = 0; j < G; ++j, cp += ldc)
                  if (g + j < cols) __stcs(cp, __uint_as_float(raw[j / 16][j % 16]));
              }
            }
            __syncwarp();   // the next group's tensor-memory loads are the whole warp's
          }
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive(&acc_empty[buf]);
        ++q;
        continue;
      }
      uint64_t sum[HALF / 2];                  // pairs of columns
#pragma unroll
      for (int j = 0; j < HALF / 2; ++j) sum[j] = 0;
      for (uint32_t p = 0; p < nkc_all; ++p, ++q) {
        const uint32_t buf = q % F::NACC;
        if (!wait_warp(&acc_full[buf], (q / F::NACC) & 1, 85)) {
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        // the smaller products' accumulator first, where it ends (the next chunk begins with them), then hi hi:
        // added to the sums, rounding to nearest
        const bool ends = p % kSumChunks == kSumChunks - 1 || p + 1 == nkc_all;
#pragma unroll 1
        for (int part = ends ? 0 : 1; part < 2; ++part) {
          const uint32_t d = part ? buf : F::NACC + sq % F::SUMS;
          if (active) {
#pragma unroll
            for (int g = 0; g < HALF; g += 16) {
              uint32_t raw[16];
              ptx::tmem_ld16(t_row + d * F::TN + g, raw);
              ptx::tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j)
                sum[g / 2 + j] = add2(sum[g / 2 + j], pack2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1])));
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive(part ? &acc_empty[buf] : &sum_empty[sq % F::SUMS]);
        }
        if (ends) ++sq;
      }
      if (!ok) break;
      float acc[HALF];
#pragma unroll
      for (int j = 0; j < HALF / 2; ++j)
        unpack2(mul2(sum[j], pack2(kUnscale, kUnscale)), acc[2 * j], acc[2 * j + 1]);
      float high = 0.f;
#pragma unroll
      for (int j = 0; j < HALF; ++j) asm("max.NaN.f32 %0, %0, %1;" : "+f"(high) : "f"(fabsf(acc[j])));
      if (__any_sync(0xffffffffu, row_ok && cols > 0 && !(high < INFINITY))) {
        if (lane == 0) atomicOr(&redo[i / 4], 1u << (8 * (i % 4) + warp));
        continue;
      }
#pragma unroll
      for (int g = 0; g < HALF; g += G) {
        if (!EARLY_C && read_c) load_c(g);
        float* cp = C + (long)g * ldc;
        asm volatile("" : "+l"(cp));
#pragma unroll
        for (int j = 0; j < G; ++j) acc[g + j] = fmaf(acc[g + j], alpha, read_c ? beta * cv[j] : 0.0f);
        if (!row_ok) continue;
        if (cols == HALF) {
#pragma unroll
          for (int j = 0; j < G; ++j, cp += ldc) __stcs(cp, acc[g + j]);
        } else {
#pragma unroll
          for (int j = 0; j < G; ++j, cp += ldc)
            if (g + j < cols) __stcs(cp, acc[g + j]);
        }
      }
    }
    if constexpr (F::PROMOTE) {
      // (inside this branch, whose registers the FFMA tiles need) every other warp has arrived here when no
      // copy or MMA is in flight in this CTA's shared memory any more, and none of them waits with a limit.
      // `again` is `a` once more: with one copy of the arguments for both, the compiler spent the pipeline's
      // registers on what this needs of them (128 x 64 tiles 5% slower)
      asm volatile("bar.sync 2, %0;" ::"n"(kSplitThreads) : "memory");
      for (uint32_t i = 0; me + i * workers < again.total; ++i) {
        const uint32_t flags = (redo[i / 4] >> (8 * (i % 4))) & 0xffu;
        if (!flags) continue;
        const SplitTile ti = split_tile<F>(again, me + i * workers);
        split_redo<F::AR, F::TN / 2>(again, ti.b, ti.m0 + rank * 128, ti.n0, flags, (float*)stages);
      }
    }
  }
  if constexpr (F::PROMOTE) {
    if (warp >= 8) {
      __syncwarp();
      asm volatile("bar.arrive 2, %0;" ::"n"(kSplitThreads) : "memory");
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  // neither CTA of a pair leaves, or gives up its tensor memory, while the other may still reach it
  if constexpr (F::PAIR) ptx::cluster_sync();
  if (warp == 16) {
    ptx::tc_fence_after();
    if constexpr (F::PAIR) ptx::tmem_dealloc_pair(tmem, F::TMEM_COLS);
    else ptx::tmem_dealloc(tmem, F::TMEM_COLS);
  }
}

// One launch over a.total tiles.
template <class F, bool GROUPED>
cudaError_t launch_tiles(SplitArgs a, const char* name, cudaStream_t st) {
  a.err = device_error_flag();
  if (!GROUPED && settings().fault == SSBLAS_FAULT_SKIP_COPY) {
    settings().fault = SSBLAS_FAULT_NONE;
    a.skip = 1;
    a.wait_limit = 1u << 10;
  }
  auto kern = f32_split_kernel<F, GROUPED>;
  constexpr int smem = F::SMEM + (GROUPED ? kRing * (int)sizeof(SplitItem) : F::PROMOTE ? (int)kRedoTiles : 0);
  static_assert(smem <= 232448, "shared memory");
  static bool attr[kMaxDevices] = {};
  if (cudaError_t e = smem_attr_once(attr, kern, smem)) return e;
  constexpr unsigned CT = F::PAIR ? 2 : 1;
  const unsigned workers = (unsigned)num_sms() / CT;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CT * (a.total < workers ? a.total : workers), 1, 1);
  cfg.blockDim = dim3(kSplitThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = CT;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = F::PAIR ? 2 : 1;
  ProfScope prof(name, st);
  note_launch();
  return cudaLaunchKernelEx(&cfg, kern, a, a);
}

template <class F>
cudaError_t launch_split(const BatchDesc& d, cudaStream_t st) {
  SplitArgs a{};
  a.m = d.m; a.n = d.n; a.k = d.k; a.lda = d.lda; a.ldb = d.ldb; a.ldc = d.ldc;
  a.A = (const float* const*)d.A;
  a.B = (const float* const*)d.B;
  a.C = (float* const*)d.C;
  a.alpha = d.alpha_f;
  a.beta = d.beta_f;
  a.a_mn = d.transa == SSBLAS_OP_N;
  a.b_mn = d.transb == SSBLAS_OP_T;
  const long tm = (d.m + F::TM - 1) / F::TM, tn = (d.n + F::TN - 1) / F::TN;
  a.tiles_m = (uint32_t)tm;
  a.tiles_mn = (uint32_t)(tm * tn);
  const long all = tm * tn * d.batch, most = F::PROMOTE ? (long)kRedoTiles * (num_sms() / (F::PAIR ? 2 : 1)) : all;
  for (long t = 0; t < all; t += most) {
    a.first = (uint32_t)t;
    a.total = (uint32_t)(all - t < most ? all - t : most);
    const cudaError_t e = launch_tiles<F, false>(a, F::NP == 3 ? "f32_split" : "bf16x3_split", st);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int NP>
cudaError_t launch_split_np(const BatchDesc& d, cudaStream_t st) {
  if (!tcgen05_available()) return cudaErrorNotSupported;
  if (d.k >= (1L << 31) || d.m >= (1L << 31) || d.n >= (1L << 31) || d.lda >= (1L << 25) || d.ldb >= (1L << 25))
    return cudaErrorNotSupported;
  if ((d.m + 127) / 128 * ((d.n + 63) / 64) * d.batch >= (1L << 31)) return cudaErrorNotSupported;
  switch (split_form(NP, d.m, d.n, d.k, d.batch, num_sms()).form) {
    case SPLIT_64: return launch_split<Split<NP, 64, 64>>(d, st);
    case SPLIT_128_64: return launch_split<Split<NP, 128, 64>>(d, st);
    case SPLIT_128_128: return launch_split<Split<NP, 128, 128>>(d, st);
    default: return launch_split<Split<NP, 128, 128, true>>(d, st);
  }
}

}  // namespace

using GroupedSplit = Split<2, 128, 128>;

bool f32_split_records(const GroupedInst& in, std::vector<SplitRec>& out) {
  if (in.k == 0 || in.m >= (1L << 31) || in.n >= (1L << 31) || in.k >= (1L << 31) || in.lda >= (1L << 25) || in.ldb >= (1L << 25) ||
      in.idx >= (1L << 31))
    return false;
  SplitRec r{};
  r.m = (int)in.m; r.n = (int)in.n; r.k = (int)in.k;
  r.idx = (int)in.idx;
  r.a_mn = in.transa == SSBLAS_OP_N;
  r.b_mn = in.transb == SSBLAS_OP_T;
  r.lda = (int)in.lda; r.ldb = (int)in.ldb; r.ldc = in.ldc;
  r.alpha = in.alpha_f; r.beta = in.beta_f;
  r.nkc = (int)((in.k + kKC - 1) / kKC);
  for (long m0 = 0; m0 < in.m; m0 += GroupedSplit::TM)
    for (long n0 = 0; n0 < in.n; n0 += GroupedSplit::TN) {
      r.m0 = (int)m0;
      r.n0 = (int)n0;
      out.push_back(r);
    }
  return true;
}

cudaError_t launch_f32_split_grouped(const SplitRec* recs, long tiles, const GroupedPtrs& p, cudaStream_t st) {
  if (!tcgen05_available()) return cudaErrorNotSupported;
  SplitArgs a{};
  a.A = (const float* const*)p.A;
  a.B = (const float* const*)p.B;
  a.C = (float* const*)p.C;
  a.recs = recs;
  a.total = (uint32_t)tiles;
  return launch_tiles<GroupedSplit, true>(a, "grouped_bf16x3_gemm", st);
}

cudaError_t launch_f32_split(const BatchDesc& d, int parts, cudaStream_t st) {
  return parts == 3 ? launch_split_np<3>(d, st) : launch_split_np<2>(d, st);
}

}  // namespace ssb
