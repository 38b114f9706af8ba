// Kernel MLP of the Monte-Carlo convolution with any number of hidden layers,
// and ALL of its gradients (weights, biases, point coordinates, densities).
//
// MCConv.py:163-171 runs num_mlps independent MLPs on the relative neighbor
// position: layer l of MLP g maps H_{l-1} values to H_l values (H_0 = D), every
// layer is followed by the activation, the last layer's outputs of all MLPs are
// concatenated (column g * H_last + h) and divided by the pair's density:
//   diff = (p_in[j] - p_out[s]) * inv_radius                      (MCConv.py:264-269)
//   a_0 = diff, a_l = act(a_{l-1} W_l[g] + b_l[g]), basis[m, g H + h] = a_L[h] / pdf[m]
// kernel_basis.cu holds the fast path for one hidden layer and the weight gradients
// only; this file is the general path.  A block takes a tile of pairs, one per thread,
// whose activations stand in shared memory as [unit][pair]: a layer is eight outputs at
// a time in registers (one load of the pair's input and two broadcast loads of weights
// per eight FMAs), for any width.  (Activations in per-thread arrays indexed at run time
// lived in local memory: 83 us forward and 286 us backward on 360 000 pairs of an 8-16
// MLP, against a few us of arithmetic.)  The backward pass recomputes the
// activations, back-propagates dbasis, and adds
//   * the weight and bias gradients: every value belongs to one thread of the block, which
//     sums it over the tile's pairs, four per load, and over its tiles in shared memory
//     (a shuffle reduction per value and warp before); one global atomic per value and
//     block;
//   * the gradient of the point coordinates (MCConv's inputs are the positions:
//     monte_carlo_conv_test.py:182-219 checks this jacobian): +d_diff / radius to
//     the neighbor's row of points_in, -d_diff / radius to the sample's row of
//     points_out, by atomics;
//   * the gradient of the density, d_pdf[m] = -sum_k dbasis[m,k] basis[m,k] / pdf[m],
//     which the caller carries on through ComputePdfPtGrads.
#include "activation.cuh"
#include "prepare.cuh"

namespace tfgpc {
namespace {

constexpr int kMaxLayers = 4;
constexpr int kMaxWidth = 64;
constexpr int kMaxParams = 8192;     // floats of all weights and biases
constexpr size_t kMaxMlpSmem = 227 * 1024;

struct MlpShape {
  int D, G, L;
  int h[kMaxLayers + 1];       // h[0] = D, h[l] = width of layer l
  int hp[kMaxLayers + 1];      // the same rounded up to 8 (l > 0) if wide, else as they are
  bool wide;                   // parameters are read eight at a time
  int w_off[kMaxLayers];       // layer l's weights [G][h[l-1]][hp[l]] in the padded parameter block
  int b_off[kMaxLayers];       // layer l's biases [G][hp[l]]
  int params;                  // floats in the padded block
  int rows;                    // of [pair] that the backward pass keeps: the inputs, and the
                               // activations and their slopes of every layer but the last
  int widest;                  // max h[l]
  const float* w[kMaxLayers];  // [G][h[l-1]][h[l]]
  const float* b[kMaxLayers];  // [G][h[l]]
};

__device__ __forceinline__ void load_params(const MlpShape& s, float* par) {
  for (int l = 0; l < s.L; ++l) {
    const int ho = s.h[l + 1], hp = s.hp[l + 1];
    for (int i = threadIdx.x; i < s.G * s.h[l] * hp; i += blockDim.x) {
      const int r = i / hp, c = i - r * hp;
      par[s.w_off[l] + i] = c < ho ? ld_global(s.w[l] + r * ho + c) : 0.0f;
    }
    for (int i = threadIdx.x; i < s.G * hp; i += blockDim.x) {
      const int r = i / hp, c = i - r * hp;
      par[s.b_off[l] + i] = c < ho ? ld_global(s.b[l] + r * ho + c) : 0.0f;
    }
  }
}

// Outputs 8q .. 8q+7 (before the activation) of layer l + 1 of MLP g for this thread's
// pair, whose inputs are the column `in` (`stride` floats apart).
__device__ __forceinline__ void layer8(const MlpShape& s, const float* par, int l, int g, int q,
                                       const float* in, int stride, float* acc) {
  const int hi = s.h[l], hp = s.hp[l + 1];
  if (!s.wide) {
    const float* w = par + s.w_off[l] + g * hi * hp + 8 * q;
    const float* b = par + s.b_off[l] + g * hp + 8 * q;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      acc[e] = 8 * q + e < hp ? b[e] : 0.0f;
      for (int i = 0; i < hi && 8 * q + e < hp; ++i) acc[e] = fmaf(in[i * stride], w[i * hp + e], acc[e]);
    }
    return;
  }
  const float4* bb = reinterpret_cast<const float4*>(par + s.b_off[l] + g * hp) + 2 * q;
  const float4* ww = reinterpret_cast<const float4*>(par + s.w_off[l] + g * hi * hp) + 2 * q;
  float4 b0 = bb[0], b1 = bb[1];
  acc[0] = b0.x; acc[1] = b0.y; acc[2] = b0.z; acc[3] = b0.w;
  acc[4] = b1.x; acc[5] = b1.y; acc[6] = b1.z; acc[7] = b1.w;
#pragma unroll 4
  for (int i = 0; i < hi; ++i) {
    const float a = in[i * stride];
    const float4 w0 = ww[i * (hp / 4)], w1 = ww[i * (hp / 4) + 1];
    acc[0] = fmaf(a, w0.x, acc[0]); acc[1] = fmaf(a, w0.y, acc[1]);
    acc[2] = fmaf(a, w0.z, acc[2]); acc[3] = fmaf(a, w0.w, acc[3]);
    acc[4] = fmaf(a, w1.x, acc[4]); acc[5] = fmaf(a, w1.y, acc[5]);
    acc[6] = fmaf(a, w1.z, acc[6]); acc[7] = fmaf(a, w1.w, acc[7]);
  }
}

__device__ __forceinline__ void load_diff(const MlpShape& s, int2 nb, const float* p_in,
                                          const float* p_out, float inv_radius,
                                          float* col, int stride) {
  for (int d = 0; d < s.D; ++d)
    col[d * stride] = (ld_global(p_in + (int64_t)nb.x * s.D + d) - ld_global(p_out + (int64_t)nb.y * s.D + d)) *
                      inv_radius;
}

__global__ void __launch_bounds__(128)
kernel_mlp_basis_kernel(MlpShape s, int64_t M, const float* p_in,
                        const float* p_out, const int2* neigh,
                        const float* pdf, float inv_radius, int act, float alpha,
                        int pdf_by_nbr, float* __restrict__ basis) {
  chain_wait();
  extern __shared__ __align__(16) float par[];
  const int stride = blockDim.x;
  float* diff = par + s.params + threadIdx.x;        // [D][pair]
  float* buf0 = diff + s.D * stride;                 // [widest][pair], twice
  float* buf1 = buf0 + s.widest * stride;
  load_params(s, par);
  __syncthreads();
  const int hl = s.h[s.L], k_total = s.G * hl;
  const bool quads = hl % 4 == 0 && (uintptr_t)basis % 16 == 0;
  for (int64_t m = (int64_t)blockIdx.x * stride + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * stride) {
    const int2 nb = ld_global(neigh + m);
    load_diff(s, nb, p_in, p_out, inv_radius, diff, stride);
    const float inv_pdf = 1.0f / ld_global(pdf + (pdf_by_nbr ? (int64_t)nb.x : m));
    for (int g = 0; g < s.G; ++g) {
      const float* in = diff;
      for (int l = 0; l < s.L; ++l) {
        const bool last = l == s.L - 1;
        float* out = (l & 1) ? buf1 : buf0;
        float* dst = basis + m * k_total + g * hl;
        for (int q = 0; q * 8 < s.h[l + 1]; ++q) {
          float acc[8];
          layer8(s, par, l, g, q, in, stride, acc);
          const int cnt = min(8, s.h[l + 1] - 8 * q);
          activate<8>(acc, act, alpha);
          if (!last) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < cnt) out[(8 * q + e) * stride] = acc[e];
          } else if (quads) {
#pragma unroll
            for (int e = 0; e < 8; e += 4)
              if (e < cnt)
                *reinterpret_cast<float4*>(dst + 8 * q + e) =
                    make_float4(acc[e] * inv_pdf, acc[e + 1] * inv_pdf, acc[e + 2] * inv_pdf,
                                acc[e + 3] * inv_pdf);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < cnt) dst[8 * q + e] = acc[e] * inv_pdf;
          }
        }
        in = out;
      }
    }
  }
}

__global__ void __launch_bounds__(128)
kernel_mlp_grads_kernel(MlpShape s, int64_t M, const float* p_in,
                        const float* p_out, const int2* neigh,
                        const float* pdf, float inv_radius, int act, float alpha,
                        int pdf_by_nbr, const float* dbasis,
                        float* __restrict__ dweights, float* __restrict__ dbiases,
                        float* __restrict__ dp_in, float* __restrict__ dp_out,
                        float* __restrict__ dpdf) {
  chain_wait();
  extern __shared__ __align__(16) float par[];       // parameters
  const int tile = blockDim.x;
  const int stride = tile + 4;                       // rows of [unit][pair], banks shifted by 4
  float* acc = par + s.params;                       // their gradients, summed over the tiles
  float* units = acc + s.params;                     // inputs, then activations and slopes
  float* grads = units + s.rows * stride;            // [2][widest][pair]
  load_params(s, par);
  for (int i = threadIdx.x; i < s.params; i += tile) acc[i] = 0.0f;
  __syncthreads();
  const int hl = s.h[s.L], k_total = s.G * hl;
  float* my_units = units + threadIdx.x;
  for (int64_t m0 = (int64_t)blockIdx.x * tile; m0 < M; m0 += (int64_t)gridDim.x * tile) {
    const int64_t m = m0 + threadIdx.x;
    const bool live = m < M;     // other threads' pairs contribute zeros
    int2 nb = make_int2(0, 0);
    float inv_pdf = 0.0f, dpdf_m = 0.0f;
    float ddiff[TFGPC_MAX_DIMS];
#pragma unroll
    for (int d = 0; d < TFGPC_MAX_DIMS; ++d) ddiff[d] = 0.0f;
    if (live) {
      nb = ld_global(neigh + m);
      inv_pdf = 1.0f / ld_global(pdf + (pdf_by_nbr ? (int64_t)nb.x : m));
      load_diff(s, nb, p_in, p_out, inv_radius, my_units, stride);
    } else {
      for (int d = 0; d < s.D; ++d) my_units[d * stride] = 0.0f;
    }
    for (int g = 0; g < s.G; ++g) {
      // rows of a layer's inputs: D coordinates, else its activations and then their slopes
      int row = 0;
      for (int l = 0; l < s.L; ++l) {
        const bool last = l == s.L - 1;
        const int ho = s.h[l + 1], next = row + (l == 0 ? s.D : 2 * s.h[l]);
        for (int q = 0; q * 8 < ho; ++q) {
          float v[8];
          layer8(s, par, l, g, q, my_units + row * stride, stride, v);
          const int cnt = min(8, ho - 8 * q);
          float slope[8];
          if (cnt < 8) {      // unit by unit: eight exponentials for one or two units cost more
            if (!last) {
#pragma unroll
              for (int e = 0; e < 7; ++e)
                if (e < cnt) {
                  my_units[(next + 8 * q + e) * stride] = activation_of(v[e], act, alpha);
                  my_units[(next + ho + 8 * q + e) * stride] = slope_of(v[e], act, alpha);
                }
            } else {
              const float* gb = dbasis + m * k_total + g * hl + 8 * q;
#pragma unroll
              for (int e = 0; e < 7; ++e)
                if (e < cnt) {
                  const float b = live ? ld_global(gb + e) : 0.0f;
                  grads[(8 * q + e) * stride + threadIdx.x] = b * inv_pdf * slope_of(v[e], act, alpha);
                  if (dpdf) dpdf_m -= b * activation_of(v[e], act, alpha) * inv_pdf * inv_pdf;
                }
            }
            continue;
          }
          slopes<8>(v, slope, act, alpha);
          if (!last || dpdf) activate<8>(v, act, alpha);
          if (!last) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < cnt) {
                my_units[(next + 8 * q + e) * stride] = v[e];
                my_units[(next + ho + 8 * q + e) * stride] = slope[e];
              }
          } else {
            // gradient of the last layer's pre-activations: dbasis / pdf * slope; the
            // density's own gradient: basis = a_L / pdf  ->  d/dpdf = -a_L / pdf^2
            const float* gb = dbasis + m * k_total + g * hl + 8 * q;
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < cnt) {
                const float b = live ? ld_global(gb + e) : 0.0f;
                grads[(8 * q + e) * stride + threadIdx.x] = b * inv_pdf * slope[e];
                if (dpdf) dpdf_m -= b * v[e] * inv_pdf * inv_pdf;
              }
          }
        }
        if (!last) row = next;
      }
      int cur = 0;
      for (int l = s.L - 1; l >= 0; --l) {
        const int hi = s.h[l], ho = s.h[l + 1], hp = s.hp[l + 1];
        const float* gl = grads + cur * s.widest * stride;
        float* gp = grads + (cur ^ 1) * s.widest * stride;
        __syncthreads();      // the tile's gradients of this layer are complete
        // weights and biases: thread o owns the o-th value
        for (int o = threadIdx.x; o < (hi + 1) * hp; o += tile) {
          const int i = o / hp, j = o - i * hp;
          if (j >= ho) continue;
          const float4* gq = reinterpret_cast<const float4*>(gl + j * stride);
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
          if (i < hi) {
            const float4* aq = reinterpret_cast<const float4*>(units + (row + i) * stride);
#pragma unroll 4
            for (int p = 0; p < tile / 4; ++p) {
              const float4 a = aq[p], b = gq[p];
              sum.x = fmaf(a.x, b.x, sum.x); sum.y = fmaf(a.y, b.y, sum.y);
              sum.z = fmaf(a.z, b.z, sum.z); sum.w = fmaf(a.w, b.w, sum.w);
            }
            acc[s.w_off[l] + (g * hi + i) * hp + j] += (sum.x + sum.y) + (sum.z + sum.w);
          } else {
#pragma unroll 4
            for (int p = 0; p < tile / 4; ++p) {
              const float4 b = gq[p];
              sum.x += b.x; sum.y += b.y; sum.z += b.z; sum.w += b.w;
            }
            acc[s.b_off[l] + g * hp + j] += (sum.x + sum.y) + (sum.z + sum.w);
          }
        }
        // back to the layer's inputs
        const float* w = par + s.w_off[l] + g * hi * hp;
        for (int i = 0; i < hi; ++i) {
          float back = 0.0f;
          const float* col = gl + threadIdx.x;
          for (int j = 0; j < ho && !s.wide; ++j) back = fmaf(col[j * stride], w[i * hp + j], back);
          for (int j = 0; j < ho && s.wide; j += 8) {
            const float4 w0 = *reinterpret_cast<const float4*>(w + i * hp + j);
            const float4 w1 = *reinterpret_cast<const float4*>(w + i * hp + j + 4);
            const float* c = col + j * stride;
            const float wj[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (j + e < ho) back = fmaf(c[e * stride], wj[e], back);
          }
          if (l > 0) {
            gp[i * stride + threadIdx.x] = back * my_units[(row + hi + i) * stride];
          } else {
#pragma unroll
            for (int d = 0; d < TFGPC_MAX_DIMS; ++d)
              if (d == i) ddiff[d] += back;
          }
        }
        cur ^= 1;
        if (l > 0) row -= l == 1 ? s.D : 2 * s.h[l - 1];
      }
      __syncthreads();        // before the next MLP or tile overwrites the activations
    }
    if (live && dpdf) dpdf[m] = dpdf_m;
    if (dp_in || dp_out) {
      // a sample's pairs follow one another: its first lane in the warp adds them up
      const int lane = threadIdx.x & 31;
      const int who = live ? nb.y : -1;
      const int prev = __shfl_up_sync(0xffffffffu, who, 1);
      const bool head = lane == 0 || prev != who;
#pragma unroll
      for (int d = 0; d < TFGPC_MAX_DIMS; ++d) {
        if (d < s.D) {
          float v = ddiff[d] * inv_radius;
          if (live && dp_in) atomicAdd(dp_in + (int64_t)nb.x * s.D + d, v);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_down_sync(0xffffffffu, v, o);
            const int id = __shfl_down_sync(0xffffffffu, who, o);
            if (lane + o < 32 && id == who) v += y;
          }
          if (live && head && dp_out) atomicAdd(dp_out + (int64_t)nb.y * s.D + d, -v);
        }
      }
    }
  }
  __syncthreads();
  int w_base = 0, b_base = 0;
  for (int l = 0; l < s.L; ++l) {
    const int ho = s.h[l + 1], hp = s.hp[l + 1], wr = s.G * s.h[l];
    for (int i = threadIdx.x; i < wr * ho; i += tile) {
      const int r = i / ho;
      atomicAdd(dweights + w_base + i, acc[s.w_off[l] + r * hp + (i - r * ho)]);
    }
    for (int i = threadIdx.x; i < s.G * ho; i += tile) {
      const int r = i / ho;
      atomicAdd(dbiases + b_base + i, acc[s.b_off[l] + r * hp + (i - r * ho)]);
    }
    w_base += wr * ho;
    b_base += s.G * ho;
  }
}

// ---- two hidden layers of at most 8 and 16 units, three dimensions --------------------------
//
// The layers' usual sizes fit registers: no activation passes through shared memory, which
// bounded the general kernels (355 000 pairs, ELU, 8-16: forward 34 us and 78 warp
// instructions per pair, gradients 131 and 224; now 24 and 81 us).  Units are padded to
// H1 = 8 and H2 = 8 or 16 with zero weights.  A padded unit is zero, and nothing comes back
// through it, only where its inputs and what reaches it are finite (infinity times its zero
// weights is no number): it is set to zero.
constexpr int kH1 = 8;

bool small_mlp(const MlpShape& s) {
  return s.D == 3 && s.L == 2 && s.h[1] <= kH1 && s.h[2] <= 16;
}

// Parameters of MLP g in shared memory: [3][8] and [8], then [8][H2] and [H2].
template <int H2>
struct SmallParams {
  float4 w1[3][kH1 / 4], b1[kH1 / 4], w2[kH1][H2 / 4], b2[H2 / 4];
  __device__ __forceinline__ void load(const MlpShape& s, int g, int threads) {
    float* p = reinterpret_cast<float*>(this);
    constexpr int kFirst = 4 * kH1, kAll = kFirst + (kH1 + 1) * H2;
    for (int i = threadIdx.x; i < kAll; i += threads) {
      const bool second = i >= kFirst;
      const int h = second ? H2 : kH1, l = second;
      const int r = (second ? i - kFirst : i) / h, c = (second ? i - kFirst : i) % h;
      const int rows = second ? kH1 : 3, in = s.h[l], out = s.h[l + 1];
      float v = 0.0f;
      if (c < out) {
        if (r == rows) v = ld_global(s.b[l] + g * out + c);
        else if (r < in) v = ld_global(s.w[l] + (g * in + r) * out + c);
      }
      p[i] = v;
    }
  }
};

__device__ __forceinline__ void fma4(float* acc, float a, float4 w) {
  acc[0] = fmaf(a, w.x, acc[0]); acc[1] = fmaf(a, w.y, acc[1]);
  acc[2] = fmaf(a, w.z, acc[2]); acc[3] = fmaf(a, w.w, acc[3]);
}
__device__ __forceinline__ void set4(float* acc, float4 b) {
  acc[0] = b.x; acc[1] = b.y; acc[2] = b.z; acc[3] = b.w;
}

// One pair per thread, MLP after MLP: its gathers are made once, and its row of the basis is
// written by one thread.  (With the pairs inside the loop over the MLPs, two of 4-8 on 890 000
// pairs took 41 us, the general kernel 38; 31 so.)  Up to rows of 32 values: longer ones the
// general kernel, whose smaller blocks have more of them under way, writes faster (four MLPs of
// 8-16, leaky ReLU, 890 000 pairs: 164 us here and 133, though 23 and 28 on 160 000).
template <int H2>
__global__ void __launch_bounds__(256, 5)
small_mlp_basis_kernel(MlpShape s, int64_t M, const float* p_in,
                       const float* p_out, const int2* neigh,
                       const float* pdf, float inv_radius, int act, float alpha,
                       int pdf_by_nbr, float* __restrict__ basis) {
  chain_enter(M, (int64_t)gridDim.x * 256);
  extern __shared__ __align__(16) float par_s[];
  SmallParams<H2>* const par = reinterpret_cast<SmallParams<H2>*>(par_s);
  const int hl = s.h[2], k_total = s.G * hl;
  const bool quads = hl % 4 == 0 && (uintptr_t)basis % 16 == 0;
  for (int g = 0; g < s.G; ++g) par[g].load(s, g, 256);
  __syncthreads();
  for (int64_t m = (int64_t)blockIdx.x * 256 + threadIdx.x; m < M; m += (int64_t)gridDim.x * 256) {
    const int2 nb = ld_global(neigh + m);
    const float inv_pdf = 1.0f / ld_global(pdf + (pdf_by_nbr ? (int64_t)nb.x : m));
    float diff[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      diff[d] = (ld_global(p_in + (int64_t)nb.x * 3 + d) - ld_global(p_out + (int64_t)nb.y * 3 + d)) *
                inv_radius;
    for (int g = 0; g < s.G; ++g) {
      // the weights are read anew for each pair: kept over the loop they take 174 registers, and
      // the few warps left wait out the gathers (355 000 pairs: 56 us)
      asm volatile("" ::: "memory");
      const SmallParams<H2>& w = par[g];
      float h[kH1];
#pragma unroll
      for (int q = 0; q < kH1 / 4; ++q) set4(h + 4 * q, w.b1[q]);
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int q = 0; q < kH1 / 4; ++q) fma4(h + 4 * q, diff[d], w.w1[d][q]);
      activate<kH1>(h, act, alpha);
      if (s.h[1] < kH1) {
#pragma unroll
        for (int i = 0; i < kH1; ++i) h[i] = i < s.h[1] ? h[i] : 0.0f;
      }
      float* dst = basis + m * k_total + g * hl;
#pragma unroll
      for (int q = 0; q < H2 / 4; ++q) {
        float v[4];
        set4(v, w.b2[q]);
#pragma unroll
        for (int i = 0; i < kH1; ++i) fma4(v, h[i], w.w2[i][q]);
        activate<4>(v, act, alpha);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] *= inv_pdf;
        if (quads) {
          if (4 * q < hl) *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (4 * q + e < hl) dst[4 * q + e] = v[e];
        }
      }
    }
  }
}

// Two lanes per pair, each with half of the last layer's units and, of what comes before
// them, half of the hidden ones: the gradients of all parameters are sums over pairs in
// (9 H2 + 32) / 2 registers per lane, 88 at H2 = 16, folded over the warp once at the end.
// blockIdx.y: the MLP.  PADDED: 0 for 8 and H2 units, 1 for fewer in the first layer, 2 for fewer
// in the last or in both; instances of their own, since what keeps the padding at zero costs a
// tenth to a fifth (890 000 pairs, leaky ReLU, us without and with: 8-16 58 and 68; two MLPs of
// 4-8 77 and 87).
template <int H2, int PADDED>
__global__ void __launch_bounds__(128, 3)
small_mlp_grads_kernel(MlpShape s, int64_t M, const float* p_in,
                       const float* p_out, const int2* neigh,
                       const float* pdf, float inv_radius, int act, float alpha,
                       int pdf_by_nbr, const float* dbasis,
                       float* __restrict__ dweights, float* __restrict__ dbiases,
                       float* __restrict__ dp_in, float* __restrict__ dp_out,
                       float* __restrict__ dpdf) {
  constexpr int HJ = H2 / 2, HI = kH1 / 2;             // units of a lane
  constexpr int kB2 = kH1 * HJ, kW1 = kB2 + HJ, kB1 = kW1 + 3 * HI;
  constexpr int kValues = kB1 + HI, kPadded = (kValues + 15) / 16 * 16;
  chain_enter(M * 2, (int64_t)gridDim.x * 128);
  __shared__ SmallParams<H2> par;
  __shared__ float red[2][kPadded];
  const int g = blockIdx.y;
  par.load(s, g, 128);
  for (int i = threadIdx.x; i < 2 * kPadded; i += 128) red[0][i] = 0.0f;
  __syncthreads();
  const int lane = threadIdx.x & 31, half = lane & 1;
  const int h1 = s.h[1], hl = s.h[2], k_total = s.G * hl;
  const bool quads = hl == H2 && k_total % 4 == 0 && (uintptr_t)dbasis % 16 == 0;
  // acc: [8][HJ] and [HJ] of the second layer, [3][HI] and [HI] of the first
  float acc[kPadded];
#pragma unroll
  for (int i = 0; i < kPadded; ++i) acc[i] = 0.0f;
  const int64_t stride = (int64_t)gridDim.x * 64;
  // (the whole warp goes on until its first pair is beyond the end)
  for (int64_t m0 = (int64_t)blockIdx.x * 64 + (threadIdx.x >> 5) * 16; m0 < M; m0 += stride) {
    const int64_t m = m0 + (lane >> 1);
    const bool live = m < M;
    const int2 nb = ld_global(neigh + (live ? m : M - 1));
    float diff[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
      diff[d] = (ld_global(p_in + (int64_t)nb.x * 3 + d) - ld_global(p_out + (int64_t)nb.y * 3 + d)) * inv_radius;
    float inv_pdf = 1.0f / ld_global(pdf + (pdf_by_nbr ? (int64_t)nb.x : live ? m : M - 1));
    if (!live) {      // (a lane without a pair adds zeros)
      diff[0] = diff[1] = diff[2] = 0.0f;
      inv_pdf = 0.0f;
    }
    float up[HJ];
    const float* gb = dbasis + m * k_total + g * hl + half * HJ;
#pragma unroll
    for (int j = 0; j < HJ; j += 4) {
      if (quads) {
        const float4 q = live ? ld_global(reinterpret_cast<const float4*>(gb + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
        set4(up + j, q);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) up[j + e] = live && half * HJ + j + e < hl ? ld_global(gb + j + e) : 0.0f;
      }
    }
    // own hidden units, the partner's by a shuffle
    float own[HI], slope1[HI], a1[kH1];
    set4(own, par.b1[half]);
#pragma unroll
    for (int d = 0; d < 3; ++d) fma4(own, diff[d], par.w1[d][half]);
    slopes<HI>(own, slope1, act, alpha);
    activate<HI>(own, act, alpha);
    if (PADDED && !(fabsf((diff[0] + diff[1]) + diff[2]) < INFINITY)) {
#pragma unroll
      for (int i = 0; i < HI; ++i) own[i] = half * HI + i < h1 ? own[i] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < HI; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, own[i], 1);
      a1[i] = half ? other : own[i];
      a1[HI + i] = half ? own[i] : other;
    }
    float back[kH1], dpdf_m = 0.0f;
#pragma unroll
    for (int i = 0; i < kH1; ++i) back[i] = 0.0f;
#pragma unroll
    for (int q = 0; q < HJ / 4; ++q) {
      float v[4];
      set4(v, par.b2[half * (HJ / 4) + q]);
#pragma unroll
      for (int i = 0; i < kH1; ++i) fma4(v, a1[i], par.w2[i][half * (HJ / 4) + q]);
      // d/dpre of the last layer; the density's own gradient: basis = a / pdf -> -a / pdf^2
      float slope[4];
      slopes<4>(v, slope, act, alpha);
      if (dpdf) activate<4>(v, act, alpha);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float b = up[4 * q + e];
        const bool used = PADDED < 2 || half * HJ + 4 * q + e < hl;
        if (dpdf && used) dpdf_m -= b * v[e] * inv_pdf * inv_pdf;
        v[e] = used ? b * inv_pdf * slope[e] : 0.0f;
        acc[kB2 + 4 * q + e] += v[e];
      }
#pragma unroll
      for (int i = 0; i < kH1; ++i) {
        const float4 w = par.w2[i][half * (HJ / 4) + q];
        back[i] = fmaf(v[3], w.w, fmaf(v[2], w.z, fmaf(v[1], w.y, fmaf(v[0], w.x, back[i]))));
#pragma unroll
        for (int e = 0; e < 4; ++e)
          acc[i * HJ + 4 * q + e] = fmaf(a1[i], v[e], acc[i * HJ + 4 * q + e]);
      }
    }
    // both halves' sums for the own hidden units
    float g1[HI];
#pragma unroll
    for (int i = 0; i < HI; ++i) {
      const float send = half ? back[i] : back[HI + i], keep = half ? back[HI + i] : back[i];
      g1[i] = (keep + __shfl_xor_sync(0xffffffffu, send, 1)) * slope1[i];
      acc[kB1 + i] += g1[i];
#pragma unroll
      for (int d = 0; d < 3; ++d) acc[kW1 + d * HI + i] = fmaf(diff[d], g1[i], acc[kW1 + d * HI + i]);
    }
    if (dpdf) {
      dpdf_m += __shfl_xor_sync(0xffffffffu, dpdf_m, 1);
      if (live && half == 0) dpdf[m] = dpdf_m;
    }
    if (dp_in || dp_out) {
      // a sample's pairs follow one another: its first lane in the warp adds them up
      const int who = live ? nb.y : -1;
      const int prev = __shfl_up_sync(0xffffffffu, who, 2);
      const bool head = lane < 2 || prev != who;
      // (found once for the three coordinates: ELU, 8-16, 8 clouds of up to 16 384 points with 24
      // neighbors 340 -> 334 us)
      bool joined[4];      // with the pair that many lanes on
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int id = __shfl_down_sync(0xffffffffu, who, 2 << t);
        joined[t] = lane + (2 << t) < 32 && id == who;
      }
#pragma unroll
      for (int i = 0; PADDED && i < HI; ++i) g1[i] = half * HI + i < h1 ? g1[i] : 0.0f;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float4 w = par.w1[d][half];
        const float mine = g1[0] * w.x + g1[1] * w.y + g1[2] * w.z + g1[3] * w.w;
        float v = (mine + __shfl_xor_sync(0xffffffffu, mine, 1)) * inv_radius;
        if (live && half == 0 && dp_in) atomicAdd(dp_in + (int64_t)nb.x * 3 + d, v);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float y = __shfl_down_sync(0xffffffffu, v, 2 << t);
          if (joined[t]) v += y;
        }
        if (live && half == 1 && head && dp_out) atomicAdd(dp_out + (int64_t)nb.y * 3 + d, -v);
      }
    }
  }
  // ---- sums over the lanes of the same half by halving (see kernel_basis_grads_kernel)
  int first = 0;
#pragma unroll
  for (int step = 0; step < 4; ++step) {
    const int o = 16 >> step, width = kPadded >> (step + 1);
    const bool upper = (lane & o) != 0;
    if (upper) first += width;
#pragma unroll
    for (int i = 0; i < kPadded / 2; ++i) {
      if (i < width) {
        const float send = upper ? acc[i] : acc[i + width];
        const float keep = upper ? acc[i + width] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kPadded / 16; ++i) atomicAdd(&red[half][first + i], acc[i]);
  __syncthreads();
  float* const dw1 = dweights + g * 3 * h1;
  float* const dw2 = dweights + s.G * 3 * h1 + g * h1 * hl;
  float* const db1 = dbiases + g * h1;
  float* const db2 = dbiases + s.G * h1 + g * hl;
  for (int i = threadIdx.x; i < 2 * kValues; i += 128) {
    const int side = i >= kValues, v = side ? i - kValues : i;
    const float x = red[side][v];
    if (v < kW1) {
      const int r = v / HJ, c = side * HJ + v % HJ;       // r = 8: the bias
      if (c < hl && r < h1) atomicAdd(dw2 + r * hl + c, x);
      else if (c < hl && r == kH1) atomicAdd(db2 + c, x);
    } else {
      const int d = (v - kW1) / HI, c = side * HI + (v - kW1) % HI;
      if (c < h1) atomicAdd(d < 3 ? dw1 + d * h1 + c : db1 + c, x);
    }
  }
}

// Shared memory of a tile of `pairs` pairs.
size_t mlp_smem(const MlpShape& s, int pairs, bool backward) {
  const size_t f = backward ? 2 * (size_t)s.params + (size_t)(s.rows + 2 * s.widest) * (pairs + 4)
                            : (size_t)s.params + (size_t)(s.D + 2 * s.widest) * pairs;
  return f * sizeof(float);
}

// Where the parameters of the layers lie in shared memory.
void place_params(MlpShape* s, bool wide) {
  s->wide = wide;
  int off = 0;
  for (int l = 0; l < s->L; ++l) {
    s->hp[l + 1] = wide ? (s->h[l + 1] + 7) / 8 * 8 : s->h[l + 1];
    s->w_off[l] = off;
    off += s->G * s->h[l] * s->hp[l + 1];
  }
  for (int l = 0; l < s->L; ++l) {
    s->b_off[l] = off;
    off += s->G * s->hp[l + 1];
  }
  s->params = wide ? off : (off + 3) / 4 * 4;   // (what follows is read in quads)
}

int make_shape(const char* op, int D, int G, int L, const int32_t* layer_sizes,
               const float* const* weights, const float* const* biases, MlpShape* out,
               int* num_weights, int* num_biases) {
  TFGPC_REQUIRE(valid_dims(D), "%s expects a valid number of dimension (got %d)", op, D);
  TFGPC_REQUIRE(G >= 1 && L >= 1 && L <= kMaxLayers && layer_sizes,
                "%s expects 1 to %d hidden layers and at least one MLP", op, kMaxLayers);
  MlpShape s{};
  s.D = D; s.G = G; s.L = L; s.h[0] = s.hp[0] = D;
  s.rows = s.widest = D;
  int nw = 0, nb = 0;
  for (int l = 0; l < L; ++l) {
    TFGPC_REQUIRE(layer_sizes[l] >= 1 && layer_sizes[l] <= kMaxWidth,
                  "%s expects hidden layers of 1 to %d units", op, kMaxWidth);
    s.h[l + 1] = layer_sizes[l];
    if (l + 1 < L) s.rows += 2 * layer_sizes[l];
    if (layer_sizes[l] > s.widest) s.widest = layer_sizes[l];
    nw += G * s.h[l] * s.h[l + 1];
    nb += G * s.h[l + 1];
    s.w[l] = weights ? weights[l] : nullptr;
    s.b[l] = biases ? biases[l] : nullptr;
  }
  TFGPC_REQUIRE(nw + nb <= kMaxParams, "%s: the kernel MLPs hold %d parameters, at most %d are supported",
                op, nw + nb, kMaxParams);
  // a thousand MLPs of a unit or two do not fit with their rows padded to eight
  place_params(&s, true);
  if (mlp_smem(s, 32, true) > kMaxMlpSmem) place_params(&s, false);
  *out = s;
  *num_weights = nw;
  *num_biases = nb;
  return TFGPC_OK;
}

// Pairs per tile: 128, fewer for MLPs so wide that they would not fit.
int mlp_tile(const MlpShape& s, bool backward) {
  int pairs = 128;
  while (pairs > 32 && mlp_smem(s, pairs, backward) > kMaxMlpSmem) pairs /= 2;
  return pairs;
}

// Per-layer pointers into flat parameter arrays.
struct LayerPointers {
  const float *w[kMaxLayers], *b[kMaxLayers];
};
LayerPointers layer_pointers(int D, int G, int L, const int32_t* sizes, const float* w,
                             const float* b) {
  LayerPointers p{};
  int prev = D;
  for (int l = 0; l < L && l < kMaxLayers && sizes; ++l) {
    p.w[l] = w;
    p.b[l] = b;
    w += (int64_t)G * prev * sizes[l];
    b += (int64_t)G * sizes[l];
    prev = sizes[l];
  }
  return p;
}

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

extern "C" int tfgpc_kernel_mlp_basis(void* stream, int D, int num_mlps, int num_layers,
                                      const int32_t* layer_sizes, int64_t M,
                                      const float* points_in, const float* points_out,
                                      const int32_t* neighbors, const float* pdf,
                                      const float* weights, const float* biases, float inv_radius,
                                      int activation, float alpha, int pdf_by_neighbor,
                                      float* basis_out) {
  TFGPC_REQUIRE(M == 0 || (weights && biases), "KernelMlpBasis got a null pointer");
  const LayerPointers p = layer_pointers(D, num_mlps, num_layers, layer_sizes, weights, biases);
  return tfgpc_kernel_mlp_basis_layers(stream, D, num_mlps, num_layers, layer_sizes, M, points_in,
                                       points_out, neighbors, pdf, p.w, p.b, inv_radius, activation,
                                       alpha, pdf_by_neighbor, basis_out);
}

extern "C" int tfgpc_kernel_mlp_basis_layers(
    void* stream, int D, int num_mlps, int num_layers, const int32_t* layer_sizes, int64_t M,
    const float* points_in, const float* points_out, const int32_t* neighbors, const float* pdf,
    const float* const* weights, const float* const* biases, float inv_radius, int activation,
    float alpha, int pdf_by_neighbor, float* basis_out) {
  MlpShape s;
  int nw, nb;
  int rc = make_shape("KernelMlpBasis", D, num_mlps, num_layers, layer_sizes, weights, biases, &s,
                      &nw, &nb);
  if (rc) return rc;
  TFGPC_REQUIRE(M >= 0 && M <= (int64_t)INT32_MAX, "KernelMlpBasis expects 0 <= M < 2^31");
  TFGPC_REQUIRE(activation == 0 || activation == 1,
                "KernelMlpBasis expects activation 0 (leaky ReLU) or 1 (ELU)");
  if (M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points_in && points_out && neighbors && pdf && weights && biases && basis_out,
                "KernelMlpBasis got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (small_mlp(s) && s.G * s.h[2] <= 32) {
    const unsigned blocks = min(blocks_for(M, 256), (unsigned)(sm_count() * 8));
    const size_t smem = s.G * (s.h[2] <= 8 ? sizeof(SmallParams<8>) : sizeof(SmallParams<16>));
    ProfScope prof(st, "kernel_mlp_basis");
    TFGPC_CUDA(launch_chained(st, blocks, 256, smem,
        s.h[2] <= 8 ? small_mlp_basis_kernel<8> : small_mlp_basis_kernel<16>, s, M, points_in,
        points_out, (const int2*)neighbors, pdf, inv_radius, activation, alpha, pdf_by_neighbor,
        basis_out));
    return TFGPC_OK;
  }
  const int tile = mlp_tile(s, false);
  const size_t smem = mlp_smem(s, tile, false);
  TFGPC_CUDA(cudaFuncSetAttribute(kernel_mlp_basis_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  unsigned grid = min(blocks_for(M, tile), (unsigned)(sm_count() * 16));
  ProfScope prof(st, "kernel_mlp_basis");
  TFGPC_CUDA(launch_chained(st, grid, tile, smem, kernel_mlp_basis_kernel, s, M, points_in,
      points_out, (const int2*)neighbors, pdf, inv_radius, activation, alpha, pdf_by_neighbor,
      basis_out));
  return TFGPC_OK;
}

extern "C" int tfgpc_kernel_mlp_grads(void* stream, int D, int num_mlps, int num_layers,
                                      const int32_t* layer_sizes, int64_t M, int64_t n_in,
                                      int64_t ns, const float* points_in, const float* points_out,
                                      const int32_t* neighbors, const float* pdf,
                                      const float* weights, const float* biases, float inv_radius,
                                      int activation, float alpha, int pdf_by_neighbor,
                                      const float* basis_grads, float* dweights_out,
                                      float* dbiases_out,
                                      float* dpoints_in_out, float* dpoints_out_out,
                                      float* dpdf_out) {
  TFGPC_REQUIRE(M == 0 || (weights && biases), "KernelMlpGrads got a null pointer");
  const LayerPointers p = layer_pointers(D, num_mlps, num_layers, layer_sizes, weights, biases);
  return tfgpc_kernel_mlp_grads_layers(stream, D, num_mlps, num_layers, layer_sizes, M, n_in, ns,
                                       points_in, points_out, neighbors, pdf, p.w, p.b, inv_radius,
                                       activation, alpha, pdf_by_neighbor, basis_grads,
                                       dweights_out, dbiases_out, dpoints_in_out, dpoints_out_out,
                                       dpdf_out);
}

extern "C" int tfgpc_kernel_mlp_grads_layers(
    void* stream, int D, int num_mlps, int num_layers, const int32_t* layer_sizes, int64_t M,
    int64_t n_in, int64_t ns, const float* points_in, const float* points_out,
    const int32_t* neighbors, const float* pdf, const float* const* weights,
    const float* const* biases, float inv_radius, int activation, float alpha,
    int pdf_by_neighbor, const float* basis_grads, float* dweights_out, float* dbiases_out,
    float* dpoints_in_out, float* dpoints_out_out, float* dpdf_out) {
  MlpShape s;
  int nw, nb;
  int rc = make_shape("KernelMlpGrads", D, num_mlps, num_layers, layer_sizes, weights, biases, &s,
                      &nw, &nb);
  if (rc) return rc;
  TFGPC_REQUIRE(M >= 0 && M <= (int64_t)INT32_MAX && n_in >= 0 && ns >= 0,
                "KernelMlpGrads expects 0 <= M < 2^31 and non-negative point counts");
  TFGPC_REQUIRE(activation == 0 || activation == 1,
                "KernelMlpGrads expects activation 0 (leaky ReLU) or 1 (ELU)");
  TFGPC_REQUIRE(dweights_out && dbiases_out, "KernelMlpGrads got a null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  Prepare jobs;
  jobs.zero(dweights_out, sizeof(float) * (size_t)nw);
  jobs.zero(dbiases_out, sizeof(float) * (size_t)nb);
  // points_in and points_out may be one cloud: its gradient is then one array
  // that both roles add into
  if (dpoints_in_out) jobs.zero(dpoints_in_out, sizeof(float) * (size_t)n_in * D);
  if (dpoints_out_out && dpoints_out_out != dpoints_in_out)
    jobs.zero(dpoints_out_out, sizeof(float) * (size_t)ns * D);
  rc = prepare(st, jobs);
  if (rc) return rc;
  if (M == 0) return TFGPC_OK;
  TFGPC_REQUIRE(points_in && points_out && neighbors && pdf && weights && biases && basis_grads,
                "KernelMlpGrads got a null pointer");
  // (the gradient of a density is the sum over its MLPs: written by one block row only)
  if (small_mlp(s) && (s.G == 1 || !dpdf_out)) {
    const unsigned most = max(3u * sm_count() / (unsigned)s.G, 1u);
    dim3 blocks(min(blocks_for(M, 64), most), (unsigned)s.G);
    ProfScope prof(st, "kernel_mlp_grads");
    const int padded = s.h[2] % 8 != 0 ? 2 : s.h[1] < kH1 ? 1 : 0;
    auto kernel = s.h[2] <= 8 ? small_mlp_grads_kernel<8, 0> : small_mlp_grads_kernel<16, 0>;
    if (padded == 1)
      kernel = s.h[2] <= 8 ? small_mlp_grads_kernel<8, 1> : small_mlp_grads_kernel<16, 1>;
    if (padded == 2)
      kernel = s.h[2] <= 8 ? small_mlp_grads_kernel<8, 2> : small_mlp_grads_kernel<16, 2>;
    TFGPC_CUDA(launch_chained(st, blocks, 128, 0, kernel,
        s, M, points_in,
        points_out, (const int2*)neighbors, pdf, inv_radius, activation, alpha, pdf_by_neighbor,
        basis_grads, dweights_out, dbiases_out, dpoints_in_out, dpoints_out_out, dpdf_out));
    return TFGPC_OK;
  }
  const int tile = mlp_tile(s, true);
  const size_t smem = mlp_smem(s, tile, true);
  TFGPC_CUDA(cudaFuncSetAttribute(kernel_mlp_grads_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  unsigned grid = min(blocks_for(M, tile), (unsigned)(sm_count() * 8));
  ProfScope prof(st, "kernel_mlp_grads");
  TFGPC_CUDA(launch_chained(st, grid, tile, smem, kernel_mlp_grads_kernel, s, M, points_in,
      points_out, (const int2*)neighbors, pdf, inv_radius, activation, alpha, pdf_by_neighbor,
      basis_grads, dweights_out, dbiases_out, dpoints_in_out, dpoints_out_out, dpdf_out));
  return TFGPC_OK;
}
