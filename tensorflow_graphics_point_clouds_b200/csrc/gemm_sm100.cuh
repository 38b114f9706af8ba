// fp32-accurate GEMM on the sm_100a tensor cores (tcgen05 + TMEM + TMA).
//
// C[M,N] (fp32) = A[M,K] * B[N,K]^T where both operands are given as two bf16
// arrays each, x ~= hi + mid (see split_bf16): three tensor-core passes
// (hi*hi + hi*mid + mid*hi) accumulate in fp32 in tensor memory and reproduce
// the fp32 product to about 2^-17 relative, well inside the 1e-4 parity bound,
// where a single bf16 or tf32 pass is not.
#pragma once

#include <cuda_bf16.h>

#include "prepare.cuh"

namespace tfgpc {

// How an operand lies in global memory.
enum class Major : int {
  K = 0,   // [rows, K] row-major: the reduction index is contiguous
  MN = 1,  // [K, rows] row-major: the M (or N) index is contiguous
};

struct GemmOperand {
  const __nv_bfloat16* hi;
  const __nv_bfloat16* mid;
  int64_t ld;  // elements between consecutive rows of the global array
  Major major;
  int64_t batch_stride = 0;  // elements between the matrices of consecutive batches
};

// C = A * B^T over k in [0, K), for every batch (the blocks of a block-diagonal weight
// matrix).  M, N, K are the logical sizes; edges are handled by TMA zero fill and
// masked stores.  transposed: c receives C^T [N, M] (MN-major A, K-major B) -- the form
// to use when the small matrix is the natural left operand: the tensor pipe reads an
// MN-major left operand faster than a K-major one (0.63 ms against 0.72 ms for 256 x
// 262144 x 2048).  bias, [N] (transposed: [M]), is added to every row of the result.
struct GemmProblem {
  int64_t M, N, K;
  GemmOperand a, b;
  float* c;
  int64_t ldc;
  bool transposed = false;
  int batches = 1;
  int64_t c_batch_stride = 0;
  const float* bias = nullptr;
  // The sums have a fixed order: more than two slices of the reduction go to `partials`
  // (partial_elems values, see gemm_partial_elems) and are added one after the other; two
  // are added into zeros, in either order the same.
  bool ordered = false;
  float* partials = nullptr;
  int64_t partial_elems = 0;
  bool cleared = false;      // c holds zeros already (see gemm_adds_slices)
};

// Values that an ordered product needs for the slices of its reduction (0: none).
int64_t gemm_partial_elems(int64_t M, int64_t N, int64_t K, bool b_mn);

// Whether the product adds the slices of its reduction into c, which then has to start
// from zero: a caller that clears all of c beforehand says so (cleared), else gemm_bf16x3
// does it with a launch of its own.
bool gemm_adds_slices(const GemmProblem& p);

// err_flag (device int, zero-initialised by the caller) is set to 1 if a bounded wait
// inside the kernel ran out.
int gemm_bf16x3(cudaStream_t stream, const GemmProblem& p, int* err_flag);

// C^T = (A * B^T)^T, A MN-major with M = channels * 16 rows, B K-major with one row per
// sample, written not as fp32 but as the bf16 hi/mid operand image of the tensor-core
// projection gradients: per group of `group` rows (1 to 4), [hi | mid][channel][128
// bytes], where the 16-byte chunk 2 * (row % group) + (k / 8) of a channel's line sits at
// position chunk ^ (channel % 8).  `image` holds ceil(N / group) groups.
int gemm_bf16x3_grad_image_tn(cudaStream_t stream, int channels, int64_t N, int64_t K,
                              const GemmOperand& a, const GemmOperand& b, void* image, int group,
                              int* err_flag);

// C^T[N, M] with row j of it written to row row_order[j] of `out` ([*, ld_out] fp32,
// 32-byte aligned rows): for right operands whose rows come in another sequence than the
// caller's.
int gemm_bf16x3_tn_scatter(cudaStream_t stream, int64_t M, int64_t N, int64_t K,
                           const GemmOperand& a, const GemmOperand& b, float* out, int64_t ld_out,
                           const int32_t* row_order, int* err_flag);

// x padded to [rows, cols] (see split_transpose_kernel) -> transposed bf16 pair.
int split_transpose_to_bf16(cudaStream_t stream, const float* x, int64_t rows, int64_t cols,
                            int cols_src, int k_src, int k_dst, __nv_bfloat16* hi_t,
                            __nv_bfloat16* mid_t);

}  // namespace tfgpc
