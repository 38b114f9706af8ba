// Host side of the tensor-core basis projection (basis_proj_mma.cuh).
#include "basis_proj_mma.cuh"

namespace tfgpc {

namespace {

// Blocks of one SM each, and the samples a warp (or team) takes at a time: enough work
// items per warp (eight) to even out lists of unequal length, up to the 32 that one load of
// range ends covers.  (With 32 always, 41 000 samples left 1036 warps one or two blocks
// each; with four items, gradients of 33 000 ragged samples at C = 64, K = 32 took 183 us,
// with eight 165, with sixteen 167.)
struct Shape { int grid, bs; };

Shape walk_shape(int64_t items, int warps) {
  Shape s;
  int64_t bs = items / ((int64_t)sm_count() * warps * 8);
  s.bs = (int)(bs < 1 ? 1 : bs > 32 ? 32 : bs);
  int64_t grid = ((items + s.bs - 1) / s.bs + warps - 1) / warps;
  s.grid = (int)(grid < 1 ? 1 : grid > sm_count() ? sm_count() : grid);
  return s;
}

template <int K, int CC, int OUT, bool BLOCKS>
int launch_fwd(cudaStream_t st, int C, int64_t ns, const float* basis, const __nv_bfloat16* fs,
               const int2* neigh, const int32_t* ranges, float* out, __nv_bfloat16* hi,
               __nv_bfloat16* mid, int hidden) {
  typedef bpm::Cfg<K, CC> cfg;
  auto kern = bpm::basis_proj_mma_kernel<K, CC, OUT, BLOCKS>;
  constexpr int smem = cfg::kFwdWarps * cfg::kFwdWarpBytes;
  TFGPC_CUDA((allow_shared<bpm::basis_proj_mma_kernel<K, CC, OUT, BLOCKS>>(smem)));
  Shape s = walk_shape(ns, cfg::kFwdWarps);
  // few samples: the channel passes run side by side
  const int passes = (C + CC - 1) / CC;
  int rows = sm_count() / s.grid;
  rows = rows < 1 ? 1 : rows > passes ? passes : rows;
  ProfScope prof(st, OUT == 0 ? "basis_proj_mma" : "basis_proj_split_mma");
  TFGPC_CUDA(launch_chained(st, dim3(s.grid, rows), cfg::kFwdWarps * 32, smem, kern, s.bs,
      hidden_shift(hidden), C, ns, basis, fs, neigh, ranges, out, hi, mid));
  return TFGPC_OK;
}

template <int K, int CC, bool BASIS>
int launch_grads(cudaStream_t st, int C, int64_t ns, int64_t M, const float* basis,
                 const __nv_bfloat16* fs, const int2* neigh, const int32_t* ranges,
                 const float* in_grads, float* dbasis, float* dfeat, int hidden) {
  typedef bpm::GradCfg<K, CC, BASIS> cfg;
  auto kern = bpm::basis_proj_grads_mma_kernel<K, CC, BASIS>;
  constexpr int smem = cfg::kTeams * cfg::kTeamBytes;
  TFGPC_CUDA((allow_shared<bpm::basis_proj_grads_mma_kernel<K, CC, BASIS>>(smem)));
  // few samples with long lists: several teams share a sample's chunks
  const int64_t teams = (int64_t)sm_count() * cfg::kTeams;
  int64_t parts = ns > 0 ? 2 * teams / ns : 1;
  const int64_t most = ns > 0 ? M / ns / (2 * bpm::kChunk) : 1;
  if (parts > most) parts = most;
  if (parts < 1) parts = 1;
  Shape s = walk_shape(ns * parts, cfg::kTeams);
  ProfScope prof(st, BASIS ? "basis_proj_grads_mma" : "basis_proj_feature_grads_mma");
  TFGPC_CUDA(launch_chained(st, s.grid, cfg::kThreads, smem, kern, s.bs, (int)parts,
      hidden_shift(hidden), C, ns, M, basis, fs, neigh, ranges, in_grads, dbasis, dfeat));
  return TFGPC_OK;
}

// Channels per pass: the smallest that takes the layer in one, else the widest.
#define TFGPC_CC_SWITCH(K, C, ...)                                                    \
  if (K == 16) {                                                                      \
    constexpr int kK = 16;                                                            \
    if (C <= 32) { constexpr int kCC = 32; __VA_ARGS__; }                             \
    if (C <= 64) { constexpr int kCC = 64; __VA_ARGS__; }                             \
    { constexpr int kCC = 128; __VA_ARGS__; }                                         \
  }                                                                                   \
  if (K == 32) {                                                                      \
    constexpr int kK = 32;                                                            \
    if (C <= 32) { constexpr int kCC = 32; __VA_ARGS__; }                             \
    { constexpr int kCC = 64; __VA_ARGS__; }                                          \
  }                                                                                   \
  if (K == 64) { constexpr int kK = 64; constexpr int kCC = 32; __VA_ARGS__; }

}  // namespace

bool basis_proj_mma_supported(int K, int C) {
  return (K == 16 || K == 32 || K == 64) && C >= 16 && C % 16 == 0;
}

int basis_proj_mma_split(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                         const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                         __nv_bfloat16* hi, __nv_bfloat16* mid, int hidden) {
  TFGPC_CC_SWITCH(K, C, return hidden == kK
      ? launch_fwd<kK, kCC, 1, false>(st, C, ns, basis, fs, (const int2*)neigh, ranges, nullptr, hi,
                                      mid, hidden)
      : launch_fwd<kK, kCC, 1, true>(st, C, ns, basis, fs, (const int2*)neigh, ranges, nullptr, hi,
                                     mid, hidden))
  return fail(TFGPC_EINVAL, "tensor-core projection expects 16, 32 or 64 basis functions");
}

// The same projection as fp32 [ns, C, K] (the drop-in op's output).
int basis_proj_mma_f32(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                       const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                       float* out) {
  TFGPC_CC_SWITCH(K, C, return launch_fwd<kK, kCC, 0, false>(st, C, ns, basis, fs, (const int2*)neigh,
                                                      ranges, out, nullptr, nullptr, kK))
  return fail(TFGPC_EINVAL, "tensor-core projection expects 16, 32 or 64 basis functions");
}

// dbasis null: the gradient of the features alone.
int basis_proj_grads_mma(cudaStream_t st, int K, int C, int64_t ns, int64_t M, const float* basis,
                         const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                         const float* in_grads, float* dbasis, float* dfeat, int hidden) {
  // (at K = 16 wide layers take two passes: a team could not share their fragments)
  TFGPC_CC_SWITCH(K, C, constexpr int kPass = kK == 16 && kCC > 64 ? 64 : kCC;
                  return dbasis ? launch_grads<kK, kPass, true>(st, C, ns, M, basis, fs, (const int2*)neigh,
                                                                ranges, in_grads, dbasis, dfeat, hidden)
                                : launch_grads<kK, kPass, false>(st, C, ns, M, basis, fs, (const int2*)neigh,
                                                                 ranges, in_grads, nullptr, dfeat, hidden))
  return fail(TFGPC_EINVAL, "tensor-core projection expects 16, 32 or 64 basis functions");
}

}  // namespace tfgpc
