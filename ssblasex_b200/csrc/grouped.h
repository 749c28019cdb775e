// Grouped batched GEMM: host-side description shared by api.cpp, grouped.cu and gemm_simt.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <vector>

#include "internal.h"

namespace ssb {

struct GroupedInst {
  Row row;
  int transa, transb;
  long m, n, k, lda, ldb, ldc;
  long idx;                  // position in the A/B/C pointer arrays
  double alpha_d, beta_d;
  float alpha_f, beta_f;
  int32_t alpha_i, beta_i;
};

struct GroupedDesc {
  std::vector<GroupedInst> inst;
};

// The shape arguments of a grouped call as the caller passes them (no pointer array), and the scalars
// of its groups by value (the bits of alpha, then beta, of each group).
struct GroupedArgs {
  const ssblasOperation_t *transa, *transb;
  const SSINT *m, *n, *k, *lda, *ldb, *ldc, *group_size;
  const ssblasDataType_t *atype, *btype, *ctype;
  SSINT groups;
  std::vector<uint64_t> scalars;
};
struct GroupedPlan;

// plain fp32/fp64 instances of a grouped call (64 x 64 tiles: FFMA / DMMA kernels, or the SIMT
// kernel where a forced configuration asks for it)
struct SimtGInst {
  int transa, transb;
  long m, n, k, lda, ldb, ldc, idx;
  double alpha_d, beta_d;
  float alpha_f, beta_f;
};
struct GroupedSimt {
  void *inst32 = nullptr, *tiles32 = nullptr, *inst64 = nullptr, *tiles64 = nullptr;
  long ntiles32 = 0, ntiles64 = 0;
  // fp64 tiles for the FP64 tensor cores (gemm_dmma.cu), one table per op(A) / op(B) layout
  // (2 * (op(A) rows contiguous) + (op(B) columns contiguous)), longest k first; their instances
  // are in inst64
  void* dmma_tiles[4] = {};
  long ndmma[4] = {};
  // fp32 tiles for the cp.async FFMA kernel (gemm_sgemm.cu), the same way; instances in inst32
  void* sg_tiles[4] = {};
  long nsg[4] = {};
  ~GroupedSimt();
};
cudaError_t plan_simt_grouped(const GroupedDesc& g, const std::vector<int>& members, GroupedSimt& out,
                              cudaStream_t st);
// the pointer arrays (device arrays of device pointers) of a grouped call
struct GroupedPtrs {
  const void* const* A;
  const void* const* B;
  void* const* C;
};
cudaError_t launch_simt_grouped(const GroupedSimt& s, const GroupedPtrs& p, cudaStream_t st);
// One launch per layout. The layouts' launches have nothing to do with each other, and run into each other:
// `follows` says that the launch before on the stream is one of this call's chain (grid_chain_end in ptx.cuh), and is set for the next.
cudaError_t launch_dmma_grouped(const GroupedSimt& s, const GroupedPtrs& p, cudaStream_t st, bool& follows);
cudaError_t launch_sgemm_grouped(const GroupedSimt& s, const GroupedPtrs& p, cudaStream_t st, bool& follows);
#ifdef __CUDACC__
template <class K, class... Args>
cudaError_t launch_chained(K kern, unsigned grid, unsigned block, int smem, cudaStream_t st, bool& follows, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = follows ? 1 : 0;   // the first of a chain waits for all before it
  follows = true;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}
#endif

// One 128 x 128 tile of an fp32 instance in the 3xBF16 mode (f32_split.cu).
struct SplitRec {
  int m, n, k, m0, n0, idx;  // the instance's shape, the tile's first row and column, place in the arrays
  int a_mn, b_mn;            // op(A) rows / op(B) columns contiguous in memory
  int lda, ldb;
  long ldc;
  float alpha, beta;
  int nkc, pad;              // K chunks
};
// appends the instance's tiles; false (none appended) where its sizes are beyond the records
bool f32_split_records(const GroupedInst& in, std::vector<SplitRec>& out);
cudaError_t launch_f32_split_grouped(const SplitRec* recs, long tiles, const GroupedPtrs& p, cudaStream_t st);

// A grouped call's device tables depend on its shapes, scalars and the settings only, so a plan serves
// every call that repeats those values, whatever matrices it points to. grouped_find: the cached plan of the
// current device for these arguments (compared value by value), nullptr if there is none; read_scalars fills
// a.scalars, and is asked once the shapes and types are known to be a plan's (false: they cannot be read).
// grouped_make: a new plan (the arguments were validated), cached in place of the least recently
// used one. grouped_launch: all instances with device-resident operands, one pre-pass and one
// persistent GEMM launch per kind. captured: the stream is being captured; the plan then stays until
// grouped_release and serves graphs only. grouped_has_f64: whether any instance is fp64.
GroupedPlan* grouped_find(const GroupedArgs& a, bool captured, const std::function<bool()>& read_scalars);
cudaError_t grouped_make(const GroupedDesc& g, const GroupedArgs& a, cudaStream_t st, GroupedPlan** out);
cudaError_t grouped_launch(GroupedPlan& plan, const GroupedPtrs& p, cudaStream_t st, bool captured);
bool grouped_has_f64(const GroupedPlan& plan);
void grouped_release();

}  // namespace ssb
