// Kernel-MLP basis of the Monte-Carlo convolution and its weight gradients.
//
// Forward, per neighbor pair m = (point j, sample s):
//   diff = (p_in[j] - p_out[s]) * inv_radius                (MCConv.py:264-269)
//   basis[m, k] = act(sum_d diff_d * w1[d, k] + b1[k]) / pdf[m]   (:163-171)
// which the reference runs as a chain of TensorFlow ops (two gathers, subtract,
// divide, tile, matmul, add, leaky_relu, transpose/reshape, divide), each a full
// pass over [M, K] memory.  Here one thread owns one pair and the only traffic
// is the pair's indices, two point gathers, its density and the 4*K-byte row
// it writes.
// Backward: dpre = dbasis / pdf * act'(pre); dw1[d, k] = sum_m diff_d * dpre_k,
// db1[k] = sum_m dpre_k, accumulated in registers over a grid-stride loop,
// reduced through shuffles and shared memory, one atomic per block and value.
#include "activation.cuh"
#include "basis_proj.cuh"
#include "prepare.cuh"

namespace tfgpc {
namespace {

constexpr int kKbThreads = 256;
// Basis functions handled per thread in the backward pass: (D + 1) accumulators each.
__host__ __device__ constexpr int k_tile(int D, int K) {
  return D <= 3 && K >= 16 ? 16 : 8;
}

// 256-bit accesses to global memory (sm_100): a thread that owns a 64-byte row
// then reads or writes whole 32-byte sectors instead of halves of them.
__device__ __forceinline__ void st_global_256(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
                 "f"(v[6]), "f"(v[7]) : "memory");
}

__device__ __forceinline__ void ld_global_256(const float* p, float* v) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7]) : "l"(p));
}

template <int D>
__device__ __forceinline__ void pair_diff(const float* p_in,
                                          const float* p_out, int2 nb,
                                          float inv_radius, float* diff) {
#pragma unroll
  for (int d = 0; d < D; ++d)
    diff[d] = (ld_global(p_in + (int64_t)nb.x * D + d) - ld_global(p_out + (int64_t)nb.y * D + d)) * inv_radius;
}

// diff and 1 / density of pair m.  pdf_mode 0: density per pair, 1: a table with
// one density per point of p_in, 2 (D == 3): p_in is the packed table of
// pack_points_density_kernel, (x, y, z, 1 / density) per point -- ONE 16-byte
// gather per pair in place of three coordinate loads and a density load, which
// matters because these kernels are bound by the number of scattered loads a warp
// issues, not by bytes.
template <int D>
__device__ __forceinline__ float pair_inputs(const float* p_in,
                                             const float* p_out,
                                             const float* pdf, int2 nb, int64_t m,
                                             float inv_radius, int pdf_mode, float* diff) {
  if (D == 3 && pdf_mode == 2) {
    const float4 pp = ld_global(reinterpret_cast<const float4*>(p_in) + nb.x);
    const float* q = p_out + (int64_t)nb.y * 3;
    diff[0] = (pp.x - ld_global(q)) * inv_radius;
    diff[1] = (pp.y - ld_global(q + 1)) * inv_radius;
    diff[2] = (pp.z - ld_global(q + 2)) * inv_radius;
    return pp.w;
  }
  pair_diff<D>(p_in, p_out, nb, inv_radius, diff);
  return 1.0f / ld_global(pdf + (pdf_mode ? (int64_t)nb.x : m));
}

__global__ void pack_points_density_kernel(int64_t n, const float* pts,
                                           const float* pdf,
                                           float4* __restrict__ out) {
  chain_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = make_float4(ld_global(pts + 3 * i), ld_global(pts + 3 * i + 1), ld_global(pts + 3 * i + 2),
                       1.0f / ld_global(pdf + i));
}

// Where the weight of dimension d and basis function k lies in [K / hidden, D, hidden]: the
// kernel MLPs one after the other, as a layer stores them; hidden = K is [D, K].
template <int D>
__device__ __forceinline__ int weight_at(int d, int k, int hidden) {
  const int g = k / hidden;
  return (g * D + d) * hidden + (k - g * hidden);
}

// WIDE: rows are 32-byte aligned, 256-bit accesses are allowed.
template <int D, int K, bool WIDE>
__global__ void __launch_bounds__(kKbThreads)
kernel_basis_kernel(int64_t M, const float* p_in, const float* p_out,
                    const int2* neigh, const float* pdf,
                    const float* w1, const float* b1, float inv_radius,
                    int act, float alpha, float* __restrict__ basis,
                    __nv_bfloat16* __restrict__ pair, int pdf_by_nbr, int hidden) {
  chain_enter(M, (int64_t)gridDim.x * kKbThreads);
  __shared__ float w_s[D * K + K];
  for (int i = threadIdx.x; i < D * K + K; i += kKbThreads)
    w_s[i] = i < D * K ? ld_global(w1 + weight_at<D>(i / K, i % K, hidden)) : ld_global(b1 + i - D * K);
  __syncthreads();
  for (int64_t m = (int64_t)blockIdx.x * kKbThreads + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * kKbThreads) {
    const int2 nb = ld_global(neigh + m);
    float diff[D];
    const float inv_pdf = pair_inputs<D>(p_in, p_out, pdf, nb, m, inv_radius, pdf_by_nbr, diff);
    float* dst = basis + m * K;
    uint4 pr[K / 4];   // hi chunks, then mid chunks, of the bf16 pair
#pragma unroll
    for (int q = 0; q < K / 8; ++q) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = 8 * q + i;
        float pre = w_s[D * K + k];
#pragma unroll
        for (int d = 0; d < D; ++d) pre = fmaf(diff[d], w_s[d * K + k], pre);
        v[i] = pre;
      }
      activate<8>(v, act, alpha);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] *= inv_pdf;
      if (!basis) {
      } else if (WIDE) {
        st_global_256(dst + 8 * q, v);
      } else {
        reinterpret_cast<float4*>(dst)[2 * q] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(dst)[2 * q + 1] = make_float4(v[4], v[5], v[6], v[7]);
      }
      if (pair) {
        // the same row as bf16 hi / mid terms: [m][hi K | mid K]
        split2_bf16(v[0], v[1], pr[q].x, pr[K / 8 + q].x);
        split2_bf16(v[2], v[3], pr[q].y, pr[K / 8 + q].y);
        split2_bf16(v[4], v[5], pr[q].z, pr[K / 8 + q].z);
        split2_bf16(v[6], v[7], pr[q].w, pr[K / 8 + q].w);
      }
    }
    if (pair) {
      // whole 32-byte sectors per store
      uint8_t* prow = reinterpret_cast<uint8_t*>(pair + m * (2 * K));
#pragma unroll
      for (int i = 0; i < K / 8; ++i)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(prow + 32 * i), "r"(pr[2 * i].x), "r"(pr[2 * i].y), "r"(pr[2 * i].z),
                       "r"(pr[2 * i].w), "r"(pr[2 * i + 1].x), "r"(pr[2 * i + 1].y),
                       "r"(pr[2 * i + 1].z), "r"(pr[2 * i + 1].w) : "memory");
    }
  }
}

// What a thread of the backward pass holds of a pair it has not worked on yet.
template <int D>
struct PairLoads { float in[D], out[D], density; };

template <int D>
__device__ __forceinline__ PairLoads<D> load_pair(const float* p_in,
                                                  const float* p_out,
                                                  const float* pdf, int2 nb,
                                                  int64_t m, int pdf_mode) {
  PairLoads<D> r;
  if (D == 3 && pdf_mode == 2) {
    const float4 pp = ld_global(reinterpret_cast<const float4*>(p_in) + nb.x);
    r.in[0] = pp.x; r.in[1] = pp.y; r.in[D - 1] = pp.z;
    r.density = pp.w;
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) r.in[d] = ld_global(p_in + (int64_t)nb.x * D + d);
    r.density = ld_global(pdf + (pdf_mode ? (int64_t)nb.x : m));
  }
#pragma unroll
  for (int d = 0; d < D; ++d) r.out[d] = ld_global(p_out + (int64_t)nb.y * D + d);
  return r;
}

// The 64 accumulators leave room for two blocks per SM, too few for three dependent
// loads per pair (indices, points, gradient row): a thread loads the points and the row
// of its next pair and the indices of the one after that while it works on this one.
// One wave of blocks: each ends with (D + 1) * KT warp reductions.
// 17.8 million pairs, K 16: 446 -> 313 us (1.43 GB: 4.6 TB/s); 250 000 pairs, K 32: 52 -> 24.
template <int D, int K, bool WIDE>
__global__ void __launch_bounds__(kKbThreads, 2)
kernel_basis_grads_kernel(int64_t M, const float* p_in,
                          const float* p_out, const int2* neigh,
                          const float* pdf, const float* w1,
                          const float* b1, float inv_radius, int act, float alpha,
                          const float* dbasis, float* __restrict__ dw1,
                          float* __restrict__ db1, int pdf_by_nbr, int hidden) {
  chain_enter(M, (int64_t)gridDim.x * kKbThreads);
  constexpr int KT = k_tile(D, K);
  __shared__ float w_s[D * K + K];
  __shared__ float red[(D + 1) * KT];
  const int64_t stride = (int64_t)gridDim.x * kKbThreads;
  int64_t m = (int64_t)blockIdx.x * kKbThreads + threadIdx.x;
  const int k0 = blockIdx.y * KT;
  auto load_row = [&](int64_t row, float* g) {
    const float* src = dbasis + row * K + k0;
#pragma unroll
    for (int q = 0; q < KT / 8; ++q) {
      if (WIDE) {
        ld_global_256(src + 8 * q, g + 8 * q);
      } else {
        const float4 g0 = ld_global(reinterpret_cast<const float4*>(src) + 2 * q);
        const float4 g1 = ld_global(reinterpret_cast<const float4*>(src) + 2 * q + 1);
        g[8 * q] = g0.x; g[8 * q + 1] = g0.y; g[8 * q + 2] = g0.z; g[8 * q + 3] = g0.w;
        g[8 * q + 4] = g1.x; g[8 * q + 5] = g1.y; g[8 * q + 6] = g1.z; g[8 * q + 7] = g1.w;
      }
    }
  };
  // (past the end the last pair is loaded again)
  int2 nb = ld_global(neigh + min(m, M - 1));
  int2 nb_next = ld_global(neigh + min(m + stride, M - 1));
  float g[KT];
  load_row(min(m, M - 1), g);
  PairLoads<D> cur = load_pair<D>(p_in, p_out, pdf, nb, min(m, M - 1), pdf_by_nbr);
  for (int i = threadIdx.x; i < D * K + K; i += kKbThreads)
    w_s[i] = i < D * K ? ld_global(w1 + weight_at<D>(i / K, i % K, hidden)) : ld_global(b1 + i - D * K);
  for (int i = threadIdx.x; i < (D + 1) * KT; i += kKbThreads) red[i] = 0.0f;
  __syncthreads();
  constexpr int kValues = ((D + 1) * KT + 31) / 32 * 32;
  float acc[kValues];                     // [D][KT] of the weights, [KT] of the biases
#pragma unroll
  for (int i = 0; i < kValues; ++i) acc[i] = 0.0f;
  for (; m < M; m += stride) {
    const int64_t next = min(m + stride, M - 1);
    const PairLoads<D> ahead = load_pair<D>(p_in, p_out, pdf, nb_next, next, pdf_by_nbr);
    float g_next[KT];
    load_row(next, g_next);
    nb_next = ld_global(neigh + min(m + 2 * stride, M - 1));
    float diff[D];
#pragma unroll
    for (int d = 0; d < D; ++d) diff[d] = (cur.in[d] - cur.out[d]) * inv_radius;
    const float inv_pdf = D == 3 && pdf_by_nbr == 2 ? cur.density : 1.0f / cur.density;
#pragma unroll
    for (int k = 0; k < KT; k += 4) {
      float pre[4], slope[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        pre[e] = w_s[D * K + k0 + k + e];
#pragma unroll
        for (int d = 0; d < D; ++d) pre[e] = fmaf(diff[d], w_s[d * K + k0 + k + e], pre[e]);
      }
      slopes<4>(pre, slope, act, alpha);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float dpre = g[k + e] * inv_pdf * slope[e];
        acc[D * KT + k + e] += dpre;
#pragma unroll
        for (int d = 0; d < D; ++d) acc[d * KT + k + e] = fmaf(diff[d], dpre, acc[d * KT + k + e]);
      }
    }
    cur = ahead;
#pragma unroll
    for (int k = 0; k < KT; ++k) g[k] = g_next[k];
  }
  // Sums over the warp by halving: at every step a lane hands half of its values to its
  // partner and keeps the other half, (D + 1) * KT shuffles in all in place of five per
  // value; then one shared-memory atomic per warp and value.  (20 000 pairs, K 16: 13.0 ->
  // 4.3 us; 250 000, K 32: 22.8 -> 18.7.)
  int first = 0;
#pragma unroll
  for (int step = 0; step < 5; ++step) {
    const int o = 16 >> step, width = kValues >> (step + 1);
    const bool upper = (lane_id() & o) != 0;
    if (upper) first += width;
#pragma unroll
    for (int i = 0; i < kValues / 2; ++i) {
      if (i < width) {
        const float send = upper ? acc[i] : acc[i + width];
        const float keep = upper ? acc[i + width] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kValues / 32; ++i)
    if (first + i < (D + 1) * KT) atomicAdd(&red[first + i], acc[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < (D + 1) * KT; i += kKbThreads) {
    const int d = i / KT, k = i % KT;
    if (d < D) atomicAdd(dw1 + weight_at<D>(d, k0 + k, hidden), red[i]);
    else atomicAdd(db1 + k0 + k, red[i]);
  }
}

// Kernel-point correlation of KPConv (KPConv.py:194-212): per neighbor pair
//   basis[m, k] = weighting(|diff - kp[k]|, sigma)   for k < num_kp, 0 above
// with weighting = max(0, 1 - dist / sigma) (linear, KPConv.py:28-40) or
// exp(-(dist / (sigma / 3))^2) (gaussian, :43-56).  The columns from num_kp up to
// K are the zero padding the reference adds with tf.pad to reach a basis count
// the projection accepts.
//
// Instructions bound it (1.15 million pairs of 16 values: 74 MB written, 12 us), and a division
// per value was most of them.  The divisor is known before the launch: dist times its inverse in
// two floats, inv + rest, by one multiplication and one fma is within an ulp of the quotient
// (Brisebarre, Muller, Raina: Accelerating correctly rounded floating-point division when the
// divisor is known in advance).  For most divisors that is the rounded quotient already, not for
// all (0.48: dist 0.426666617 came out an ulp high); one correction by the remainder rounds it
// for every one (Markstein: Computation of elementary functions on the IBM RISC System/6000
// processor, theorem on the last step of a division).  All 2^23 mantissas of dist over 600
// divisors: none differs from the division, 16 did without the correction.
// 1.15 million pairs, us, by division / now / without the correction: 15 points of 16, linear
// 28.1 / 25.2 / 24.4, Gaussian 31.8 / 29.1 / 28.5; 60 of 64 114 / 97 / 92.  (A point's coordinates
// by one 16-byte load, without the correction: 25.8, 29.4 and 118.)
constexpr int kMaxKernelPoints = 64;

struct Divisor {
  float value, inv, rest;
  bool by_inverse;            // (not where the inverse's parts could underflow or overflow)
};
inline Divisor divisor_of(float v) {
  const float inv = 1.0f / v;
  const double rest = (1.0 - (double)v * (double)inv) / (double)v;
  return Divisor{v, inv, (float)rest, v > 1e-12f && v < 1e12f};
}

template <int D, int K, bool WIDE>
__global__ void __launch_bounds__(kKbThreads)
kp_basis_kernel(int64_t M, int num_kp, const float* p_in,
                const float* p_out, const int2* neigh,
                const float* kernel_points, float inv_radius, Divisor by,
                int interpolation, float* __restrict__ basis) {
  chain_enter(M, (int64_t)gridDim.x * kKbThreads);
  __shared__ float kp_s[kMaxKernelPoints * D];
  for (int i = threadIdx.x; i < num_kp * D; i += kKbThreads) kp_s[i] = ld_global(kernel_points + i);
  __syncthreads();
  for (int64_t m = (int64_t)blockIdx.x * kKbThreads + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * kKbThreads) {
    const int2 nb = ld_global(neigh + m);
    float diff[D];
    pair_diff<D>(p_in, p_out, nb, inv_radius, diff);
    float* dst = basis + m * K;
#pragma unroll
    for (int q = 0; q < K / 8; ++q) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = 8 * q + i;
        float w = 0.0f;
        if (k < num_kp) {
          float d2 = 0.0f;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const float t = diff[d] - kp_s[k * D + d];
            d2 = fmaf(t, t, d2);
          }
          const float dist = sqrtf(d2);
          const float near = fmaf(dist, by.inv, dist * by.rest);
          const float r = by.by_inverse ? fmaf(fmaf(-near, by.value, dist), by.inv, near)
                                        : dist / by.value;
          if (interpolation == 0) {
            w = fmaxf(1.0f - r, 0.0f);
          } else {
            const float q = dist < INFINITY ? r : dist;      // (infinity times a rest of zero)
            w = expf(-(q * q));
          }
        }
        v[i] = w;
      }
      if (WIDE) {
        st_global_256(dst + 8 * q, v);
      } else {
        reinterpret_cast<float4*>(dst)[2 * q] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(dst)[2 * q + 1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
}

// Density transform of PointConv (PointConv.py:168-183): per sample the largest
// density among its neighbor pairs, then per pair
//   out[m] = sum_j relu(pdf[m] / max * w1[j] + b1[j]) * w2[j] + b2      (j < 16)
// One warp owns one sample; its pairs are contiguous (ranges holds their end).  neigh null:
// pdf holds a density per pair, else one per point, read at the pair's neighbor index.
constexpr int kPdfHidden = 16;

__global__ void __launch_bounds__(kKbThreads)
pointconv_pdf_kernel(int64_t ns, const int32_t* ranges,
                     const int2* neigh, const float* pdf, const float* w1,
                     const float* b1, const float* w2,
                     const float* b2, float* __restrict__ out) {
  chain_enter(ns * 32, (int64_t)gridDim.x * kKbThreads);
  __shared__ float par[3 * kPdfHidden + 1];
  for (int i = threadIdx.x; i < 3 * kPdfHidden + 1; i += kKbThreads)
    par[i] = i < kPdfHidden ? ld_global(w1 + i)
             : i < 2 * kPdfHidden ? ld_global(b1 + i - kPdfHidden)
             : i < 3 * kPdfHidden ? ld_global(w2 + i - 2 * kPdfHidden) : ld_global(b2);
  __syncthreads();
  const int lane = lane_id();
  const int64_t warps = ((int64_t)gridDim.x * kKbThreads) >> 5;
  for (int64_t s = ((int64_t)blockIdx.x * kKbThreads + threadIdx.x) >> 5; s < ns; s += warps) {
    const int a = s ? ld_global(ranges + s - 1) : 0;
    const int e = ld_global(ranges + s);
    float mx = -INFINITY;
    auto density = [&](int m) { return ld_global(pdf + (neigh ? ld_global(&neigh[m].x) : m)); };
    for (int m = a + lane; m < e; m += 32) mx = fmaxf(mx, density(m));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    for (int m = a + lane; m < e; m += 32) {
      const float x = density(m) / mx;
      float acc = 0.0f;
#pragma unroll
      for (int j = 0; j < kPdfHidden; ++j)
        acc = fmaf(fmaxf(fmaf(x, par[j], par[kPdfHidden + j]), 0.0f), par[2 * kPdfHidden + j], acc);
      out[m] = acc + par[3 * kPdfHidden];
    }
  }
}

int check_kb_args(const char* op, int D, int K, int64_t M, int act) {
  TFGPC_REQUIRE(valid_dims(D), "%s expects a valid number of dimension (got %d)", op, D);
  TFGPC_REQUIRE(K == 8 || K == 16 || K == 32 || K == 64,
                "%s expects a valid number of basis functions.", op);
  TFGPC_REQUIRE(M >= 0 && M <= (int64_t)INT32_MAX, "%s expects 0 <= M < 2^31", op);
  TFGPC_REQUIRE(act == 0 || act == 1, "%s expects activation 0 (leaky ReLU) or 1 (ELU)", op);
  return TFGPC_OK;
}

#define TFGPC_K_SWITCH(K, ...)                              \
  switch (K) {                                              \
    case 8: { constexpr int kK = 8; __VA_ARGS__; } break;   \
    case 16: { constexpr int kK = 16; __VA_ARGS__; } break; \
    case 32: { constexpr int kK = 32; __VA_ARGS__; } break; \
    default: { constexpr int kK = 64; __VA_ARGS__; } break; \
  }

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

static int check_pdf_mode(const char* op, int D, int mode, const float* points_in) {
  TFGPC_REQUIRE(mode >= 0 && mode <= 2, "%s expects pdf_by_neighbor 0, 1 or 2", op);
  TFGPC_REQUIRE(mode != 2 || (D == 3 && (uintptr_t)points_in % 16 == 0),
                "%s: the packed point table (pdf_by_neighbor 2) needs D == 3 and 16-byte alignment",
                op);
  return TFGPC_OK;
}

extern "C" int tfgpc_pack_points_density(void* stream, int64_t n, const float* points,
                                         const float* pdf, float* packed_out) {
  TFGPC_REQUIRE(n >= 0 && n < (int64_t)INT32_MAX, "PackPointsDensity expects 0 <= n < 2^31");
  if (n == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points && pdf && packed_out, "PackPointsDensity got a null pointer");
  TFGPC_REQUIRE((uintptr_t)packed_out % 16 == 0, "PackPointsDensity expects a 16-byte aligned output");
  cudaStream_t st = (cudaStream_t)stream;
  ProfScope prof(st, "pack_points_density");
  TFGPC_CUDA(launch_chained(st, blocks_for(n, 256), 256, 0, pack_points_density_kernel, n, points,
      pdf, (float4*)packed_out));
  return TFGPC_OK;
}

static int kernel_basis_impl(void* stream, int D, int K, int64_t M, const float* points_in,
                             const float* points_out, const int32_t* neighbors, const float* pdf,
                             const float* w1, const float* b1, float inv_radius, int activation,
                             float alpha, float* basis_out, __nv_bfloat16* pair_out,
                             int pdf_by_nbr, int num_mlps = 1) {
  int rc = check_kb_args("KernelBasis", D, K, M, activation);
  if (rc) return rc;
  TFGPC_REQUIRE(num_mlps >= 1 && K % num_mlps == 0,
                "KernelBasis expects as many basis functions from every kernel MLP");
  if (M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points_in && points_out && neighbors && (pdf || pdf_by_nbr == 2) && w1 && b1 &&
                (basis_out || pair_out), "KernelBasis got a null pointer");
  rc = check_pdf_mode("KernelBasis", D, pdf_by_nbr, points_in);
  if (rc) return rc;
  TFGPC_REQUIRE((uintptr_t)basis_out % 16 == 0 && (uintptr_t)pair_out % 32 == 0,
                "KernelBasis expects 16-byte aligned outputs (32 for the bf16 pair)");
  cudaStream_t st = (cudaStream_t)stream;
  unsigned grid = min(blocks_for(M, kKbThreads), (unsigned)(sm_count() * 16));
  ProfScope prof(st, "kernel_basis");
  if ((uintptr_t)basis_out % 32 == 0) {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kernel_basis_kernel<kD, kK, true>, M, points_in, points_out, (const int2*)neighbors, pdf,
        w1, b1, inv_radius, activation, alpha, basis_out, pair_out, pdf_by_nbr,
        K / num_mlps))));
  } else {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kernel_basis_kernel<kD, kK, false>, M, points_in, points_out, (const int2*)neighbors, pdf,
        w1, b1, inv_radius, activation, alpha, basis_out, pair_out, pdf_by_nbr,
        K / num_mlps))));
  }
  return TFGPC_OK;
}

extern "C" int tfgpc_kernel_basis(void* stream, int D, int K, int64_t M, const float* points_in,
                                  const float* points_out, const int32_t* neighbors,
                                  const float* pdf, const float* w1, const float* b1,
                                  float inv_radius, int activation, float alpha,
                                  int pdf_by_neighbor, float* basis_out) {
  return kernel_basis_impl(stream, D, K, M, points_in, points_out, neighbors, pdf, w1, b1,
                           inv_radius, activation, alpha, basis_out, nullptr, pdf_by_neighbor);
}

extern "C" int tfgpc_kernel_basis_split(void* stream, int D, int K, int64_t M,
                                        const float* points_in, const float* points_out,
                                        const int32_t* neighbors, const float* pdf,
                                        const float* w1, const float* b1, float inv_radius,
                                        int activation, float alpha, int pdf_by_neighbor,
                                        float* basis_out, void* basis_pair_out) {
  TFGPC_REQUIRE(M == 0 || basis_pair_out, "KernelBasis got a null pointer");
  return kernel_basis_impl(stream, D, K, M, points_in, points_out, neighbors, pdf, w1, b1,
                           inv_radius, activation, alpha, basis_out,
                           (__nv_bfloat16*)basis_pair_out, pdf_by_neighbor);
}

extern "C" int tfgpc_kernel_basis_mlps(void* stream, int D, int K, int num_mlps, int64_t M,
                                       const float* points_in, const float* points_out,
                                       const int32_t* neighbors, const float* pdf,
                                       const float* w1, const float* b1, float inv_radius,
                                       int activation, float alpha, int pdf_by_neighbor,
                                       float* basis_out, void* basis_pair_out) {
  return kernel_basis_impl(stream, D, K, M, points_in, points_out, neighbors, pdf, w1, b1,
                           inv_radius, activation, alpha, basis_out,
                           (__nv_bfloat16*)basis_pair_out, pdf_by_neighbor, num_mlps);
}

static int kernel_basis_grads_impl(void* stream, int D, int K, int num_mlps, int64_t M,
                                   const float* points_in, const float* points_out,
                                   const int32_t* neighbors, const float* pdf, const float* w1,
                                   const float* b1, float inv_radius, int activation, float alpha,
                                   int pdf_by_neighbor, const float* basis_grads, float* dw1_out,
                                   float* db1_out) {
  int rc = check_kb_args("KernelBasisGrads", D, K, M, activation);
  if (rc) return rc;
  TFGPC_REQUIRE(num_mlps >= 1 && K % num_mlps == 0,
                "KernelBasisGrads expects as many basis functions from every kernel MLP");
  TFGPC_REQUIRE(dw1_out && db1_out, "KernelBasisGrads got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  Prepare jobs;
  jobs.zero(dw1_out, sizeof(float) * (size_t)D * K);
  jobs.zero(db1_out, sizeof(float) * (size_t)K);
  rc = prepare(st, jobs);
  if (rc) return rc;
  if (M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points_in && points_out && neighbors && (pdf || pdf_by_neighbor == 2) && w1 &&
                b1 && basis_grads, "KernelBasisGrads got a null pointer");
  rc = check_pdf_mode("KernelBasisGrads", D, pdf_by_neighbor, points_in);
  if (rc) return rc;
  TFGPC_REQUIRE((uintptr_t)basis_grads % 16 == 0,
                "KernelBasisGrads expects 16-byte aligned gradients");
  const unsigned tiles = (unsigned)(K / k_tile(D, K));
  dim3 grid(min(blocks_for(M, kKbThreads), max(2u * sm_count() / tiles, 1u)), tiles);
  ProfScope prof(st, "kernel_basis_grads");
  if ((uintptr_t)basis_grads % 32 == 0) {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kernel_basis_grads_kernel<kD, kK, true>, M, points_in, points_out, (const int2*)neighbors,
        pdf, w1, b1, inv_radius, activation, alpha, basis_grads, dw1_out, db1_out,
        pdf_by_neighbor, K / num_mlps))));
  } else {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kernel_basis_grads_kernel<kD, kK, false>, M, points_in, points_out, (const int2*)neighbors,
        pdf, w1, b1, inv_radius, activation, alpha, basis_grads, dw1_out, db1_out,
        pdf_by_neighbor, K / num_mlps))));
  }
  return TFGPC_OK;
}

extern "C" int tfgpc_kernel_basis_grads(void* stream, int D, int K, int64_t M,
                                        const float* points_in, const float* points_out,
                                        const int32_t* neighbors, const float* pdf,
                                        const float* w1, const float* b1, float inv_radius,
                                        int activation, float alpha, int pdf_by_neighbor,
                                        const float* basis_grads, float* dw1_out,
                                        float* db1_out) {
  return kernel_basis_grads_impl(stream, D, K, 1, M, points_in, points_out, neighbors, pdf, w1, b1,
                                 inv_radius, activation, alpha, pdf_by_neighbor, basis_grads,
                                 dw1_out, db1_out);
}

extern "C" int tfgpc_kernel_basis_mlps_grads(
    void* stream, int D, int K, int num_mlps, int64_t M, const float* points_in,
    const float* points_out, const int32_t* neighbors, const float* pdf, const float* w1,
    const float* b1, float inv_radius, int activation, float alpha, int pdf_by_neighbor,
    const float* basis_grads, float* dw1_out, float* db1_out) {
  return kernel_basis_grads_impl(stream, D, K, num_mlps, M, points_in, points_out, neighbors, pdf,
                                 w1, b1, inv_radius, activation, alpha, pdf_by_neighbor,
                                 basis_grads, dw1_out, db1_out);
}

extern "C" int tfgpc_kp_basis(void* stream, int D, int K, int num_kernel_points, int64_t M,
                              const float* points_in, const float* points_out,
                              const int32_t* neighbors, const float* kernel_points,
                              float inv_radius, float sigma, int interpolation,
                              float* basis_out) {
  int rc = check_kb_args("KPBasis", D, K, M, 0);
  if (rc) return rc;
  TFGPC_REQUIRE(num_kernel_points >= 1 && num_kernel_points <= K,
                "KPBasis expects 1 <= kernel points <= basis functions");
  TFGPC_REQUIRE(interpolation == 0 || interpolation == 1,
                "KPBasis expects interpolation 0 (linear) or 1 (gaussian)");
  TFGPC_REQUIRE(sigma > 0.0f && inv_radius > 0.0f, "KPBasis expects a positive sigma and radius");
  if (M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points_in && points_out && neighbors && kernel_points && basis_out,
                "KPBasis got a null pointer");
  TFGPC_REQUIRE((uintptr_t)basis_out % 16 == 0, "KPBasis expects a 16-byte aligned output");
  cudaStream_t st = (cudaStream_t)stream;
  unsigned grid = min(blocks_for(M, kKbThreads), (unsigned)(sm_count() * 16));
  const Divisor by = divisor_of(interpolation == 0 ? sigma : sigma / 3.0f);
  ProfScope prof(st, "kp_basis");
  if ((uintptr_t)basis_out % 32 == 0) {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kp_basis_kernel<kD, kK, true>, M, num_kernel_points, points_in, points_out,
        (const int2*)neighbors, kernel_points, inv_radius, by, interpolation, basis_out))));
  } else {
    TFGPC_DIM_SWITCH(D, TFGPC_K_SWITCH(K, TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0,
        kp_basis_kernel<kD, kK, false>, M, num_kernel_points, points_in, points_out,
        (const int2*)neighbors, kernel_points, inv_radius, by, interpolation, basis_out))));
  }
  return TFGPC_OK;
}

static int pointconv_pdf(void* stream, int64_t ns, int64_t M, const int32_t* ranges,
                         const int32_t* neighbors, const float* pdf, const float* w1,
                         const float* b1, const float* w2, const float* b2, float* pdf_out) {
  TFGPC_REQUIRE(ns >= 0 && ns < (int64_t)INT32_MAX && M >= 0 && M <= (int64_t)INT32_MAX,
                "PointConvPdf expects 0 <= ns, M < 2^31");
  if (ns == 0 || M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(ranges && pdf && w1 && b1 && w2 && b2 && pdf_out,
                "PointConvPdf got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  unsigned grid = min(blocks_for(ns, kKbThreads / 32), (unsigned)(sm_count() * 16));
  ProfScope prof(st, "pointconv_pdf");
  TFGPC_CUDA(launch_chained(st, grid, kKbThreads, 0, pointconv_pdf_kernel, ns, ranges,
      (const int2*)neighbors, pdf, w1, b1, w2, b2, pdf_out));
  return TFGPC_OK;
}

extern "C" int tfgpc_pointconv_pdf(void* stream, int64_t ns, int64_t M, const int32_t* ranges,
                                   const float* pdf, const float* w1, const float* b1,
                                   const float* w2, const float* b2, float* pdf_out) {
  return pointconv_pdf(stream, ns, M, ranges, nullptr, pdf, w1, b1, w2, b2, pdf_out);
}

extern "C" int tfgpc_pointconv_pdf_by_neighbor(void* stream, int64_t ns, int64_t M,
                                               const int32_t* ranges, const int32_t* neighbors,
                                               const float* pdf, const float* w1, const float* b1,
                                               const float* w2, const float* b2, float* pdf_out) {
  TFGPC_REQUIRE(ns == 0 || M == 0 || neighbors, "PointConvPdf got a null pointer");
  return pointconv_pdf(stream, ns, M, ranges, neighbors, pdf, w1, b1, w2, b2, pdf_out);
}
