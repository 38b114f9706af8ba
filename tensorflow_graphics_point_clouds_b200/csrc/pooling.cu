// Pooling layers and the bias of the 1x1 convolution.
//
// The reference runs these as TensorFlow segment ops: a gather of the
// neighbors' feature rows into an [M, C] tensor followed by
// unsorted_segment_max / _mean over the sample index (Pooling.py:148-162), and
// unsorted_segment_max / _mean over the batch ids for the global variants
// (Pooling.py:51-57, 90-96).  Here the rows of a sample are read in place (its
// pairs are contiguous, ranges holds their end), one thread per (sample,
// channel), so the [M, C] tensor is never written; the global variants
// accumulate per cloud with atomics on the [B, C] result.
// An empty segment gives the lowest float for max (what TensorFlow's
// unsorted_segment_max writes) and 0 for mean.
#include <cfloat>

#include "common.cuh"

namespace tfgpc {
namespace {

constexpr int kPoolThreads = 256;

// A thread owns VEC channels of a sample: 4 where the rows are 16-byte aligned.  What
// bounds it is the number of row loads in flight out of L2: the 128-channel
// rows of 24 neighbors around the subsample of 16 x 8192 points took 36 us in 4-byte
// loads, 22 now.  Four rows are loaded before the first is used: left to the compiler they
// stayed one behind the other in the averages (64 channels around 333 000 samples of 1 000 000
// points, us: 169 so, 126 now; with read-only loads 155).
template <int VEC>
__global__ void __launch_bounds__(kPoolThreads)
neighborhood_pool_kernel(int mode, int C, int64_t ns, const float* features,
                         const int2* neigh, const int32_t* ranges,
                         float* __restrict__ out) {
  const int groups = C / VEC;
  const int64_t total = ns * groups;
  chain_enter(total, (int64_t)gridDim.x * kPoolThreads);
  for (int64_t i = (int64_t)blockIdx.x * kPoolThreads + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * kPoolThreads) {
    const int64_t s = i / groups;
    const int c = (int)(i - s * groups) * VEC;
    const int a = s ? ld_global(ranges + s - 1) : 0;
    const int e = ld_global(ranges + s);
    float acc[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = mode == 0 ? -FLT_MAX : 0.0f;
    auto load = [&](int m, float* v) {
      const float* row = features + (int64_t)ld_global(&neigh[m].x) * C + c;
      if (VEC == 4) {
        const float4 f = ld_global(reinterpret_cast<const float4*>(row));
        v[0] = f.x; v[VEC > 1] = f.y; v[VEC > 1 ? 2 : 0] = f.z; v[VEC - 1] = f.w;
      } else {
        v[0] = ld_global(row);
      }
    };
    auto add = [&](const float* v) {
#pragma unroll
      for (int k = 0; k < VEC; ++k) acc[k] = mode == 0 ? fmaxf(acc[k], v[k]) : acc[k] + v[k];
    };
    int m = a;
    for (; VEC == 4 && m + 4 <= e; m += 4) {
      float v[4][VEC];
#pragma unroll
      for (int u = 0; u < 4; ++u) load(m + u, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) add(v[u]);
    }
#pragma unroll 4
    for (; m < e; ++m) {
      float v[VEC];
      load(m, v);
      add(v);
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      if (mode == 1 && e > a) acc[k] /= (float)(e - a);
      if (VEC == 1) out[s * C + c] = acc[k];
    }
    if (VEC == 4)
      *reinterpret_cast<float4*>(out + s * C + c) =
          make_float4(acc[0], acc[VEC > 1], acc[VEC > 1 ? 2 : 0], acc[VEC - 1]);
  }
}

// Order-preserving map between floats and unsigned integers, so that the
// maximum of floats is an atomicMax of integers.
__device__ __forceinline__ unsigned float_key(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__global__ void pool_init_kernel(int mode, int64_t n, float* out, float* counts, int64_t b) {
  chain_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = mode == 0 ? __uint_as_float(float_key(-FLT_MAX)) : 0.0f;
  if (i < b) counts[i] = 0.0f;
}

// A thread owns one channel of kPoolRun consecutive points and folds them while the
// cloud stays the same, so that the atomics, all on the few values of the result, are
// one per run: 18.9 -> 6.6 us at the
// 16 subsampled clouds of 8192 points, 256 channels.  The maximum is one of keys throughout: it also keeps what is no number.
constexpr int kPoolRun = 16;

__global__ void __launch_bounds__(kPoolThreads)
global_pool_kernel(int mode, int C, int64_t n, int64_t batch_size,
                   const float* features, const int32_t* batch_ids,
                   float* out, float* counts) {
  const int64_t total = (n + kPoolRun - 1) / kPoolRun * C;
  chain_enter(total, (int64_t)gridDim.x * kPoolThreads);
  for (int64_t i = (int64_t)blockIdx.x * kPoolThreads + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * kPoolThreads) {
    const int64_t run = i / C;
    const int c = (int)(i - run * C);
    float v[kPoolRun];
    int b[kPoolRun];
#pragma unroll
    for (int k = 0; k < kPoolRun; ++k) {
      const int64_t p = run * kPoolRun + k;
      b[k] = p < n ? ld_global(batch_ids + p) : -1;
      v[k] = p < n ? ld_global(features + p * C + c) : 0.0f;
    }
    unsigned top = 0u;
    float sum = 0.0f, count = 0.0f;
#pragma unroll
    for (int k = 0; k < kPoolRun; ++k) {
      if (mode == 0) top = max(top, float_key(v[k]));
      sum += v[k];
      count += 1.0f;
      if (k + 1 < kPoolRun && b[k + 1] == b[k]) continue;
      if (b[k] >= 0 && b[k] < batch_size) {
        if (mode == 0) {
          atomicMax(reinterpret_cast<unsigned*>(out) + (int64_t)b[k] * C + c, top);
        } else {
          atomicAdd(out + (int64_t)b[k] * C + c, sum);
          if (c == 0) atomicAdd(counts + b[k], count);
        }
      }
      top = 0u;
      sum = count = 0.0f;
    }
  }
}

__global__ void pool_finish_kernel(int mode, int C, int64_t n, float* out,
                                   const float* counts) {
  chain_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (mode == 0) {
    out[i] = key_float(reinterpret_cast<unsigned*>(out)[i]);
  } else {
    const float cnt = counts[i / C];
    out[i] = cnt > 0.0f ? out[i] / cnt : 0.0f;
  }
}

__global__ void add_bias_kernel(int64_t n, int C, float* x, const float* bias) {
  chain_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n * C) x[i] += ld_global(bias + (i % C));
}

// x = act(x * scale + bias): inference batch normalisation with stored
// statistics folded into scale and bias, followed by the activation
// (modelnet40_small.py:236-243).  act 0: none, 1: leaky ReLU with slope alpha.
__global__ void scale_bias_act_kernel(int64_t total, int C, float* x, float scale,
                                      const float* bias, int act, float alpha) {
  chain_enter(total, (int64_t)gridDim.x * blockDim.x);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    float v = x[i] * scale;
    if (bias) v += ld_global(bias + (i % C));
    if (act == 1) v = v > 0.0f ? v : v * alpha;
    x[i] = v;
  }
}

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

extern "C" int tfgpc_neighborhood_pool(void* stream, int mode, int C, int64_t ns, int64_t n_in,
                                       int64_t M, const float* features,
                                       const int32_t* neighbors, const int32_t* ranges,
                                       float* out) {
  TFGPC_REQUIRE(mode == 0 || mode == 1, "Pooling expects mode 0 (max) or 1 (average)");
  TFGPC_REQUIRE(C > 0 && ns >= 0 && n_in >= 0 && M >= 0 && ns < (int64_t)INT32_MAX &&
                M <= (int64_t)INT32_MAX, "Pooling expects 0 <= ns, M < 2^31 and C > 0");
  if (ns == 0) return TFGPC_OK;
  TFGPC_REQUIRE(ranges && out && (M == 0 || (features && neighbors)),
                "Pooling got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope prof(st, "neighborhood_pool");
  const bool wide = C % 4 == 0 && (uintptr_t)features % 16 == 0 && (uintptr_t)out % 16 == 0;
  const unsigned grid = min(blocks_for(ns * (wide ? C / 4 : C), kPoolThreads),
                            (unsigned)(sm_count() * 32));
  auto kernel = wide ? neighborhood_pool_kernel<4> : neighborhood_pool_kernel<1>;
  TFGPC_CUDA(launch_chained(st, grid, kPoolThreads, 0, kernel, mode, C, ns, features,
      (const int2*)neighbors, ranges, out));
  return TFGPC_OK;
}

extern "C" size_t tfgpc_global_pool_workspace_bytes(int64_t batch_size) {
  return align_up((size_t)(batch_size > 0 ? batch_size : 0) * sizeof(float), 256) + 256;
}

extern "C" int tfgpc_global_pool(void* stream, int mode, int C, int64_t n, int64_t batch_size,
                                 const float* features, const int32_t* batch_ids, float* out,
                                 void* ws, size_t ws_bytes) {
  TFGPC_REQUIRE(mode == 0 || mode == 1, "Pooling expects mode 0 (max) or 1 (average)");
  TFGPC_REQUIRE(C > 0 && n >= 0 && batch_size > 0 && n < (int64_t)INT32_MAX,
                "Pooling expects C > 0, a positive batch size and 0 <= n < 2^31");
  TFGPC_REQUIRE(out && ws && (n == 0 || (features && batch_ids)), "Pooling got a null pointer");
  if (ws_bytes < tfgpc_global_pool_workspace_bytes(batch_size))
    return fail(TFGPC_ENOMEM, "Pooling workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope prof(st, "global_pool");
  float* counts = (float*)ws;
  const int64_t cells = batch_size * C;
  const int64_t init = cells > batch_size ? cells : batch_size;
  TFGPC_CUDA(launch_chained(st, blocks_for(init, 256), 256, 0, pool_init_kernel, mode, cells, out,
      counts, batch_size));
  if (n > 0) {
    const unsigned grid = min(blocks_for((n + kPoolRun - 1) / kPoolRun * C, kPoolThreads),
                              (unsigned)(sm_count() * 32));
    TFGPC_CUDA(launch_chained(st, grid, kPoolThreads, 0, global_pool_kernel, mode, C, n,
        batch_size, features, batch_ids, out, counts));
  }
  TFGPC_CUDA(launch_chained(st, blocks_for(cells, 256), 256, 0, pool_finish_kernel, mode, C, cells,
      out, counts));
  return TFGPC_OK;
}

extern "C" int tfgpc_add_bias(void* stream, int64_t n, int C, float* x, const float* bias) {
  TFGPC_REQUIRE(n >= 0 && C > 0, "AddBias expects n >= 0 and C > 0");
  if (n == 0) return TFGPC_OK;
  TFGPC_REQUIRE(x && bias, "AddBias got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope prof(st, "add_bias");
  TFGPC_CUDA(launch_chained(st, blocks_for(n * C, 256), 256, 0, add_bias_kernel, n, C, x, bias));
  return TFGPC_OK;
}

extern "C" int tfgpc_scale_bias_activation(void* stream, int64_t n, int C, float* x, float scale,
                                           const float* bias, int activation, float alpha) {
  TFGPC_REQUIRE(n >= 0 && C > 0, "ScaleBiasActivation expects n >= 0 and C > 0");
  TFGPC_REQUIRE(activation == 0 || activation == 1,
                "ScaleBiasActivation expects activation 0 (none) or 1 (leaky ReLU)");
  if (n == 0) return TFGPC_OK;
  TFGPC_REQUIRE(x, "ScaleBiasActivation got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope prof(st, "scale_bias_activation");
  unsigned grid = min(blocks_for(n * C, 256), (unsigned)(sm_count() * 16));
  TFGPC_CUDA(launch_chained(st, grid, 256, 0, scale_bias_act_kernel, n * C, C, x, scale, bias,
      activation, alpha));
  return TFGPC_OK;
}
