// Copies of one operand of the FP64 tensor-core kernel (gemm_dmma.cu), slab by slab along K. Free of
// CUDA -- the copies themselves are the caller's -- so that its index arithmetic is unit-tested on the CPU.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define SSB_HD __host__ __device__ __forceinline__
#else
#define SSB_HD inline
#endif

namespace ssb {

// One operand's copies by thread t: chunk q (two doubles along the contiguous dimension) of the next
// K slab comes from src + q * step and goes to dst + q * DSTEP of the slab's buffer, so that a slab
// inside the matrix costs one copy and one addition per chunk (with the position of every chunk
// worked out again the copies took as many issue slots as the products' loads).
//   MN: rows contiguous in global memory (element (r, k) at X[r + k*ld]) -> staged [k][r];
//   otherwise element (r, k) at X[r*ld + k] -> staged [r][k].
// K has 64 bits (two thin operands of 2^31 k fit the device): what is left of it is held as a count of whole
// slabs and the k of the last, ragged one, each of 32 bits.
template <int ROWS, int BK, int NT, bool MN>
struct Slab {
  static constexpr int P = MN ? ROWS + 4 : BK + 4;
  static constexpr int CPL = (MN ? ROWS : BK) / 2;        // chunks per contiguous line
  static constexpr int NQ = ROWS * BK / 2 / NT;           // chunks per thread
  static constexpr int LSTEP = NT / CPL;                  // lines between a thread's chunks
  static constexpr int DSTEP = LSTEP * P;                 // doubles between their places
  static constexpr long KMAX = BK * 0x7ffffff0L;          // K below it (256 GB of one row)
  static_assert(NT % CPL == 0 && NQ * NT == ROWS * BK / 2 && NQ * LSTEP == (MN ? BK : ROWS), "slab/threads mismatch");
  const double* src;
  const double* X;
  long step, adv;            // doubles between chunks, between slabs
  int whole, rest;           // slabs left that lie inside K, and the valid k of the one after them
  int kk;                    // k of this thread's first chunk in a slab
  int lines, bytes;          // chunks of this thread inside the rows, and valid bytes of each (MN)
  uint32_t dst;              // byte offset of its place
  bool vec;
  SSB_HD void init(const double* X_, long nrows, long K, long ld, long r0, int t) {
    X = X_;
    vec = ((uintptr_t)X % 16 == 0) && (ld % 2 == 0);
    const int rr = MN ? 2 * (t % CPL) : t / CPL;
    kk = MN ? t / CPL : 2 * (t % CPL);
    src = X + (MN ? r0 + rr + kk * ld : (r0 + rr) * ld + kk);
    step = LSTEP * ld;
    adv = MN ? BK * ld : BK;
    const long left = nrows - r0 - rr;    // valid rows from this thread's first chunk on
    const int most = (int)((left + LSTEP - 1) / LSTEP < NQ ? (left + LSTEP - 1) / LSTEP : NQ);
    lines = MN ? NQ : left > 0 ? most : 0;
    bytes = MN ? (left >= 2 ? 16 : left == 1 ? 8 : 0) : 16;
    if (bytes == 0) lines = 0;
    whole = (int)(K / BK);
    rest = (int)(K % BK);
    dst = 8u * (uint32_t)(MN ? kk * P + rr : rr * P + kk);
  }
  SSB_HD int slabs() const { return whole + (rest != 0 ? 1 : 0); }
  // The next slab into `buf` (shared-space address) by cp.cp16 / cp.cp8(destination, source, valid bytes);
  // moves on to the one after it. A slab with all of its k inside the matrix asks for fixed lines and
  // bytes per thread; only the last one, where k runs out, looks at each chunk.
  template <class Copy>
  SSB_HD void copy(uint32_t buf, const Copy& cp) {
    const uint32_t d = buf + dst;
    const double* s = src;
    if (whole > 0) {
      if (vec && lines == NQ && bytes == 16) {
#pragma unroll
        for (int q = 0; q < NQ; ++q, s += step) cp.cp16(d + 8u * (uint32_t)(q * DSTEP), s, 16);
      } else if (vec) {
#pragma unroll
        for (int q = 0; q < NQ; ++q, s += step)
          cp.cp16(d + 8u * (uint32_t)(q * DSTEP), q < lines ? s : X, q < lines ? bytes : 0);
      } else {
        const int b0 = bytes < 8 ? bytes : 8, b1 = bytes - b0;
#pragma unroll
        for (int q = 0; q < NQ; ++q, s += step) {
          const bool ok = q < lines;
          cp.cp8(d + 8u * (uint32_t)(q * DSTEP), ok ? s : X, ok ? b0 : 0);
          cp.cp8(d + 8u * (uint32_t)(q * DSTEP + 1), ok && b1 ? s + 1 : X, ok ? b1 : 0);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < NQ; ++q, s += step) {
        // valid elements of the chunk, which runs along r (MN) or along k
        int nv = MN ? (kk + q * LSTEP < rest ? bytes / 8 : 0) : (q < lines ? rest - kk : 0);
        nv = nv < 0 ? 0 : (nv > 2 ? 2 : nv);
        const double* g = nv > 0 ? s : X;
        if (vec) {
          cp.cp16(d + 8u * (uint32_t)(q * DSTEP), g, 8 * nv);
        } else {
          cp.cp8(d + 8u * (uint32_t)(q * DSTEP), g, nv > 0 ? 8 : 0);
          cp.cp8(d + 8u * (uint32_t)(q * DSTEP + 1), nv > 1 ? g + 1 : X, nv > 1 ? 8 : 0);
        }
      }
      rest = 0;
    }
    src += adv;
    --whole;
  }
};

}  // namespace ssb
