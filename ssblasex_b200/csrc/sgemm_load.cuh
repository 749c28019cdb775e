// Copies of FP32 operand slabs into shared memory, staged [k][rows] whatever the operand's layout: the loads
// of the FFMA kernels (gemm_sgemm.cu) and of the tiles that the BF16-split kernel computes again
// (f32_split.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ssb {

static __device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
static __device__ __forceinline__ void cp16s(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
static __device__ __forceinline__ void cp4s(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
static __device__ __forceinline__ void commit_s() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
static __device__ __forceinline__ void wait_s() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Copies the (ROWS x BK) slab of one operand at (r0, k0) into a stage buffer staged [k][r]
// (pitch ROWS + 4 floats). MN: element (r, k) at X[r + k*ld]; otherwise at X[r*ld + k].
// Each thread's chunks keep one position along the contiguous dimension and step a fixed number
// of rows (or k) per iteration, so the source pointer advances by a constant: no per-element
// index arithmetic.
template <int ROWS, int BK, int NT, bool MN>
static __device__ __forceinline__ void sload(float* dst, const float* __restrict__ X, long nrows, long K, long ld, long r0,
                                      long k0, bool vec) {
  constexpr int P = ROWS + 4;
  const int t = threadIdx.x;
  if (MN) {
    if (vec) {
      // 16-byte chunks along r: thread t takes r = 4 (t % (ROWS/4)), k = t / (ROWS/4) + q KSTEP
      constexpr int CPR = ROWS / 4, KSTEP = NT / CPR, NQ = BK / KSTEP;
      static_assert(NT % CPR == 0 && BK % KSTEP == 0, "copy shape");
      const int rr = 4 * (t % CPR), kk0 = t / CPR;
      const long gr = r0 + rr;
      long nv = nrows - gr;
      nv = nv < 0 ? 0 : (nv > 4 ? 4 : nv);
      const float* src = X + gr + (k0 + kk0) * ld;
      const uint32_t d0 = saddr(dst + kk0 * P + rr);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool ok = nv > 0 && k0 + kk0 + q * KSTEP < K;
        cp16s(d0 + 4u * (uint32_t)(q * KSTEP * P), ok ? src + (long)q * KSTEP * ld : X, ok ? (int)(4 * nv) : 0);
      }
    } else {
      constexpr int KSTEP = NT / ROWS, NQ = BK / KSTEP;
      static_assert(NT % ROWS == 0 && BK % KSTEP == 0, "copy shape");
      const int rr = t % ROWS, kk0 = t / ROWS;
      const bool rok = r0 + rr < nrows;
      const float* src = X + (r0 + rr) + (k0 + kk0) * ld;
      const uint32_t d0 = saddr(dst + kk0 * P + rr);
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const bool ok = rok && k0 + kk0 + q * KSTEP < K;
        cp4s(d0 + 4u * (uint32_t)(q * KSTEP * P), ok ? src + (long)q * KSTEP * ld : X, ok ? 4 : 0);
      }
    }
  } else {
    // Transpose by the copy. A warp instruction covers 8 consecutive k of 4 consecutive rows
    // (lane = 4 * (k % 8) + r % 4): the reads are whole 32-byte sectors, and the [k][r] stores
    // land in banks (4 k + r) mod 32 (pitch = 4 mod 32), all 32 distinct. Instruction u = warp + W q
    // of the stage takes k group u % KG and row group u / KG, so each thread keeps its k and
    // steps RSTEP rows per iteration.
    constexpr int W = NT / 32, KG = BK / 8, RSTEP = 4 * (W / KG), NQ = ROWS / RSTEP;
    static_assert(BK % 8 == 0 && W % KG == 0 && ROWS % RSTEP == 0 && P % 32 == 4, "copy shape");
    const int lane = t % 32, warp = t / 32;
    const int kk = 8 * (warp % KG) + lane / 4, rr0 = 4 * (warp / KG) + lane % 4;
    const bool kok = k0 + kk < K;
    const float* src = X + (r0 + rr0) * ld + (k0 + kk);
    const uint32_t d0 = saddr(dst + kk * P + rr0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const bool ok = kok && r0 + rr0 + q * RSTEP < nrows;
      cp4s(d0 + 4u * (uint32_t)(q * RSTEP), ok ? src + (long)q * RSTEP * ld : X, ok ? 4 : 0);
    }
  }
}

}  // namespace ssb
