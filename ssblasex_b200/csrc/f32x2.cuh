// Packed FP32 arithmetic of sm_100: two values per instruction, each rounded as the single form rounds
// it. The pipe's rate is that of the single form (70 TFLOP/s measured for either); the packed form takes
// half the issue slots for it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ssb {

static __device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
static __device__ __forceinline__ void unpack2(uint64_t v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
static __device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
static __device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
static __device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// acc (TM x TN, pairs of rows) += a (TM values, k-th line of op(A) at pa) x b (TN values at pb); pa and pb
// are 16-byte aligned, TM and TN multiples of 4; the rows are groups of 4, STEP apart.
template <int TM, int TN, int STEP = 4>
static __device__ __forceinline__ void outer2(uint64_t (&acc)[TM / 2][TN], const float* pa, const float* pb) {
  uint64_t a[TM / 2];
#pragma unroll
  for (int i = 0; i < TM / 4; ++i) {
    const ulonglong2 x = *(const ulonglong2*)(pa + STEP * i);
    a[2 * i] = x.x;
    a[2 * i + 1] = x.y;
  }
#pragma unroll
  for (int j = 0; j < TN; j += 4) {
    const float4 x = *(const float4*)(pb + j);
    const uint64_t b[4] = {pack2(x.x, x.x), pack2(x.y, x.y), pack2(x.z, x.z), pack2(x.w, x.w)};
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int i = 0; i < TM / 2; ++i) acc[i][j + q] = fma2(a[i], b[q], acc[i][j + q]);
  }
}
template <int TM, int TN>
static __device__ __forceinline__ void unpack_acc(const uint64_t (&v)[TM / 2][TN], float (&acc)[TM][TN]) {
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) unpack2(v[i][j], acc[2 * i][j], acc[2 * i + 1][j]);
}

}  // namespace ssb
