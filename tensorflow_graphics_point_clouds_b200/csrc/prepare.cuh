// What has to be done before a kernel's main work starts, in one launch.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace tfgpc {

// x [*, cols] fp32 -> hi, mid [rows, ld] bf16 (see prepare_kernel), rows `stride` (0: ld)
// values apart.
struct SplitJob {
  const float* x = nullptr;
  int64_t rows = 0;
  int cols = 0, ld = 0;
  const int32_t* order = nullptr;
  int k_src = 1, k_dst = 1;
  __nv_bfloat16 *hi = nullptr, *mid = nullptr;
  int64_t stride = 0;
};

// What a product or a projection needs before it starts: operands split into bf16 pairs
// and buffers cleared, all in one launch.  (As separate launches and memsets these were
// 11 of the 22 of a small layer's training step, 2 to 3 us each, more than the layer's
// arithmetic.)
struct Prepare {
  static constexpr int kSplits = 3, kClears = 5;
  SplitJob split[kSplits];
  struct Clear { void* p; int64_t words; } clear[kClears];
  int splits = 0, clears = 0;
  void add(const SplitJob& j) { split[splits++] = j; }
  // `bytes` (a multiple of 4) zeros at p (4-byte aligned)
  void zero(void* p, size_t bytes) { if (bytes) clear[clears++] = {p, (int64_t)(bytes / 4)}; }
};
int prepare(cudaStream_t stream, const Prepare& jobs);

// Features [n, C] as the tensor-core projections read them: fs [n, 2, C], the hi terms of
// a point and then its mid terms.
inline SplitJob feature_job(const float* features, int64_t n, int C, __nv_bfloat16* fs) {
  SplitJob j;
  j.x = features;
  j.rows = n;
  j.cols = j.ld = C;
  j.stride = 2 * (int64_t)C;
  j.hi = fs;
  j.mid = fs + C;
  return j;
}

}  // namespace tfgpc
