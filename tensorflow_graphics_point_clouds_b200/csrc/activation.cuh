// Activations of the kernel MLPs: 0 leaky ReLU with slope alpha (0: ReLU), 1 ELU.
#pragma once

namespace tfgpc {

// N values at a time: one branch on the activation for all of them, and none on the sign.
// (With `x > 0 ? x : expm1f(x)` every unit was a divergent branch of its own, which kept
// the exponentials of a pair's units from overlapping.  131 072 pairs and one layer of 32
// units: basis 12.1 -> 9.1 us, gradients 18.7 -> 14.4; 355 000 pairs, layers of 8 and 16:
// gradients 95 -> 81.)
template <int N>
__device__ __forceinline__ void activate(float* x, int act, float alpha) {
  if (act == 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float e = expm1f(x[i] > 0.0f ? 0.0f : x[i]);
      x[i] = x[i] > 0.0f ? x[i] : e;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = x[i] > 0.0f ? x[i] : x[i] * alpha;
  }
}

// Slopes at the pre-activations x.  (From the activation's value they would be wrong for a
// negative alpha, whose values below zero are positive, and value + 1 loses the digits of
// ELU's exp(x).)
template <int N>
__device__ __forceinline__ void slopes(const float* x, float* s, int act, float alpha) {
  if (act == 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float e = expf(x[i] > 0.0f ? 0.0f : x[i]);
      s[i] = x[i] > 0.0f ? 1.0f : e;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = x[i] > 0.0f ? 1.0f : alpha;
  }
}

// One unit: a branch on its sign in place of an exponential that nobody needs.
__device__ __forceinline__ float activation_of(float x, int act, float alpha) {
  if (act == 1) return x > 0.0f ? x : expm1f(x);
  return x > 0.0f ? x : x * alpha;
}
__device__ __forceinline__ float slope_of(float x, int act, float alpha) {
  if (x > 0.0f) return 1.0f;
  return act == 1 ? expf(x) : alpha;
}

}  // namespace tfgpc
