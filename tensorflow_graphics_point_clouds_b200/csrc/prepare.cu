// Operand splits and clears (prepare.cuh): bound by HBM where they are large (32 bytes
// in and 32 out per thread of a split), by the launch where they are small.
#include "prepare.cuh"
#include "basis_proj.cuh"

namespace tfgpc {
namespace {

// Row r of a split's output is the split of a row of its source, `ld` columns wide with
// zeros from `cols` on: row order[r], or, for a weight matrix whose basis functions are
// padded from k_src to k_dst, row (r / k_dst) * k_src + r % k_dst (none if r % k_dst
// reaches k_src).
struct PrepareJobs {
  Prepare jobs;
  int first_block[Prepare::kSplits + Prepare::kClears + 1];    // splits, then clears
};

constexpr int kSplitPer = 8;       // values per thread: 32 bytes in, 16 and 16 out
constexpr int kClearWords = 16;    // words per thread

__device__ __forceinline__ void split_block(const SplitJob& j, unsigned block) {
  const unsigned octets = (unsigned)j.ld / kSplitPer;
  const unsigned i = block * 256u + threadIdx.x;
  if (i >= (unsigned)j.rows * octets) return;
  const unsigned r = (octets & (octets - 1)) == 0 ? i >> (31 - __clz(octets)) : i / octets;
  const int c = (int)(i - r * octets) * kSplitPer;
  int64_t src = r;
  if (j.order) {
    src = ld_global(j.order + r);
  } else if (j.k_src != j.k_dst) {
    const unsigned ch = r / (unsigned)j.k_dst;
    const int k = (int)(r - ch * j.k_dst);
    src = k < j.k_src ? (int64_t)ch * j.k_src + k : -1;
  }
  float v[kSplitPer];
#pragma unroll
  for (int e = 0; e < kSplitPer; ++e) v[e] = 0.0f;
  if (src >= 0) {
    const float* p = j.x + src * j.cols + c;
    if (j.cols % 4 == 0 && (uintptr_t)j.x % 16 == 0) {
#pragma unroll
      for (int e = 0; e < kSplitPer; e += 4) {
        if (c + e < j.cols) {
          const float4 q = ld_global(reinterpret_cast<const float4*>(p + e));
          v[e] = q.x; v[e + 1] = q.y; v[e + 2] = q.z; v[e + 3] = q.w;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < kSplitPer; ++e)
        if (c + e < j.cols) v[e] = ld_global(p + e);
    }
  }
  uint4 h, m;
  split2_bf16(v[0], v[1], h.x, m.x);
  split2_bf16(v[2], v[3], h.y, m.y);
  split2_bf16(v[4], v[5], h.z, m.z);
  split2_bf16(v[6], v[7], h.w, m.w);
  *reinterpret_cast<uint4*>(j.hi + (int64_t)r * j.stride + c) = h;
  *reinterpret_cast<uint4*>(j.mid + (int64_t)r * j.stride + c) = m;
}

__device__ __forceinline__ void clear_block(const Prepare::Clear& j, int64_t block) {
  uint32_t* p = (uint32_t*)j.p;
  const int64_t w0 = block * (256 * kClearWords);
  if ((uintptr_t)p % 16 == 0) {
#pragma unroll
    for (int u = 0; u < kClearWords / 4; ++u) {
      const int64_t w = w0 + (u * 256 + (int)threadIdx.x) * 4;
      if (w + 4 <= j.words) {
        *reinterpret_cast<uint4*>(p + w) = make_uint4(0, 0, 0, 0);
      } else {
        for (int64_t e = w; e < j.words; ++e) p[e] = 0;
      }
    }
  } else {
#pragma unroll
    for (int u = 0; u < kClearWords; ++u) {
      const int64_t w = w0 + u * 256 + (int)threadIdx.x;
      if (w < j.words) p[w] = 0;
    }
  }
}

__global__ void __launch_bounds__(256) prepare_kernel(const __grid_constant__ PrepareJobs a) {
  chain_enter();
  const int block = (int)blockIdx.x;
#pragma unroll
  for (int i = 0; i < Prepare::kSplits; ++i)
    if (block >= a.first_block[i] && block < a.first_block[i + 1])
      split_block(a.jobs.split[i], (unsigned)(block - a.first_block[i]));
#pragma unroll
  for (int i = 0; i < Prepare::kClears; ++i) {
    const int f = Prepare::kSplits + i;
    if (block >= a.first_block[f] && block < a.first_block[f + 1])
      clear_block(a.jobs.clear[i], block - a.first_block[f]);
  }
}

}  // namespace

int prepare(cudaStream_t stream, const Prepare& jobs) {
  PrepareJobs a{};
  a.jobs = jobs;
  int64_t blocks = 0;
  for (int i = 0; i < Prepare::kSplits + Prepare::kClears; ++i) {
    a.first_block[i] = (int)blocks;
    if (i < Prepare::kSplits && i < jobs.splits) {
      SplitJob& j = a.jobs.split[i];
      if (j.stride == 0) j.stride = j.ld;
      TFGPC_REQUIRE(j.ld % kSplitPer == 0 && j.stride % kSplitPer == 0 &&
                    (uintptr_t)j.hi % 16 == 0 && (uintptr_t)j.mid % 16 == 0,
                    "prepare expects rows of a multiple of 8 values, 16-byte aligned");
      const int64_t items = j.rows * (j.ld / kSplitPer);
      TFGPC_REQUIRE(items < (int64_t)UINT32_MAX - 256, "prepare: too many values");
      blocks += (items + 255) / 256;
    } else if (i >= Prepare::kSplits && i - Prepare::kSplits < jobs.clears) {
      const Prepare::Clear& j = jobs.clear[i - Prepare::kSplits];
      blocks += (j.words + 256 * kClearWords - 1) / (256 * kClearWords);
    }
    TFGPC_REQUIRE(blocks < (int64_t)INT32_MAX, "prepare: too many values");
  }
  a.first_block[Prepare::kSplits + Prepare::kClears] = (int)blocks;
  if (blocks == 0) return TFGPC_OK;
  ProfScope prof(stream, "prepare");
  TFGPC_CUDA(launch_chained(stream, (unsigned)blocks, 256, 0, prepare_kernel, a));
  return TFGPC_OK;
}

}  // namespace tfgpc
