// Monte-Carlo convolution forward and backward: the basis projection followed
// by (forward) or preceded by (backward) the weight GEMMs on the tensor cores.
//
// Forward:  X[s, c*K+k] = sum_m basis[m,k] * feat[nbr(m), c]   (basis_proj.cu,
//           written directly as the bf16 hi/mid pair the GEMM consumes)
//           out = X * W                                        (gemm_sm100.cu)
// Backward: dX = dOut * W^T, (dbasis, dfeat) = BasisProjGrads(dX),
//           dW = X^T * dOut  (split over the sample range, slices summed).
// This is the pair BasisProj -> tf.matmul of pylib/pc/layers/MCConv.py:174-191
// and its autodiff, without the fp32 [Ns, C, K] tensor between the two.
#include "basis_proj.cuh"
#include "gemm_sm100.cuh"

namespace tfgpc {

int basis_proj_split(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                     const float* feat, const int32_t* neigh, const int32_t* ranges,
                     __nv_bfloat16* hi, __nv_bfloat16* mid, int hidden);
// (adds into dfeat, and into dbasis where basis_proj_grads_adds_dbasis says so: the caller
// clears them)
bool basis_proj_grads_adds_dbasis(int K, int C, const float* feat);
int basis_proj_grads_blocks(cudaStream_t st, int K, int C, int64_t ns, int64_t M,
                            const float* basis, const float* feat, const int32_t* neigh,
                            const int32_t* ranges, const float* in_grads, float* dbasis,
                            float* dfeat, int hidden);
// basis_proj_tile.cu: the gradients of narrow layers (dbasis may be null)
bool basis_proj_grads_tile_takes(int K, int C, const float* feat);
int basis_proj_grads_tile(cudaStream_t st, int K, int C, int64_t ns, int64_t M, const float* basis,
                          const float* feat, const int2* neigh, const int32_t* ranges,
                          const float* in_grads, float* dbasis, float* dfeat, int hidden);
// basis_proj_mma.cu: the projection on warp-level tensor-core MMAs
bool basis_proj_mma_supported(int K, int C);
int basis_proj_mma_split(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                         const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                         __nv_bfloat16* hi, __nv_bfloat16* mid, int hidden);
int basis_proj_grads_mma(cudaStream_t st, int K, int C, int64_t ns, int64_t M, const float* basis,
                         const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                         const float* in_grads, float* dbasis, float* dfeat, int hidden);

// basis_proj_grads_tc.cu: the gradients on tcgen05 tensor cores
bool basis_proj_grads_tc_supported(int K, int C);
int basis_proj_grads_tc_group(int64_t ns, int64_t M);
int basis_proj_grads_tc(cudaStream_t st, int group, int64_t ns, int64_t M, const float* basis,
                        const __nv_bfloat16* fs, const int32_t* neigh, const int32_t* ranges,
                        const void* image, float* dbasis, float* dfeat, int* err_flag);

// basis_proj_grads_tcu.cu: the gradients on the rows of a group plan
int basis_proj_grads_tcu(cudaStream_t st, int64_t ns, int64_t M, const void* plan,
                         const __nv_bfloat16* basis_pair, const __nv_bfloat16* fs,
                         const int32_t* ranges, const void* image, float* dbasis, float* dfeat,
                         int* err_flag);

// basis_proj_fwd_tcu.cu: the projection on the rows of a group plan
int basis_proj_fwd_tcu(cudaStream_t st, int64_t ns, int64_t M, const void* plan,
                       const __nv_bfloat16* basis_pair, const __nv_bfloat16* fs,
                       __nv_bfloat16* x_hi, __nv_bfloat16* x_mid, int* err_flag);

namespace {

struct McWs {
  int* err;                  // [0] set by a GEMM whose bounded wait ran out
  __nv_bfloat16 *x_hi, *x_mid;      // [ns, C*K]
  __nv_bfloat16 *w_hi, *w_mid;      // [C*K, Cout]
  __nv_bfloat16 *g_hi, *g_mid;      // [ns, Cout]   (backward)
  float* dx;                        // [ns, C*K]    (backward)
  __nv_bfloat16* fs;                // [n_in, 2, C] split features (tensor-core projection)
  float* partials;                  // slices of the forward product, where it has several
  int64_t partial_elems;
  __nv_bfloat16 *wt_hi, *wt_mid;    // [Cout, C*K]: W transposed (backward)
  float* dw_pad;                    // [C*K, Cout]: gradient of padded weights (backward)
  size_t bytes;
};

// With at least one full tile of output features the roles of the forward product are
// swapped, out^T = W^T * X^T with W as the (MN-major) left operand, and the tiles are
// transposed on their way out.
inline bool forward_swapped(int64_t cout) { return cout >= 128; }

McWs carve(void* ws, int K, int C, int Cout, int64_t ns, int64_t n_in, bool backward) {
  McWs w;
  char* p = (char*)ws;
  auto take = [&](size_t b) { char* r = p; p += align_up(b, 1024); return r; };
  const size_t ck = (size_t)C * K;
  w.err = (int*)take(256);
  w.x_hi = (__nv_bfloat16*)take((size_t)ns * ck * 2);
  w.x_mid = (__nv_bfloat16*)take((size_t)ns * ck * 2);
  w.w_hi = (__nv_bfloat16*)take(ck * Cout * 2);
  w.w_mid = (__nv_bfloat16*)take(ck * Cout * 2);
  // ahead of the backward-only buffers, so that a forward and a backward carve
  // of the same workspace agree on where it lies
  w.fs = nullptr;
  if (basis_proj_mma_supported(K, C)) w.fs = (__nv_bfloat16*)take((size_t)n_in * C * 4);
  w.partial_elems = forward_swapped(Cout) ? gemm_partial_elems(Cout, ns, ck, false)
                                          : gemm_partial_elems(ns, Cout, ck, true);
  w.partials = (float*)take((size_t)w.partial_elems * 4);
  w.g_hi = w.g_mid = nullptr; w.dx = nullptr; w.wt_hi = w.wt_mid = nullptr; w.dw_pad = nullptr;
  if (backward) {
    w.g_hi = (__nv_bfloat16*)take((size_t)ns * Cout * 2);
    w.g_mid = (__nv_bfloat16*)take((size_t)ns * Cout * 2);
    // as operand image of the tensor-core gradient kernel: one slot of 4*ck floats
    // per group of three (or four) samples
    w.dx = (float*)take((size_t)((ns + 2) / 3) * 4 * ck * 4);
    w.wt_hi = (__nv_bfloat16*)take(ck * Cout * 2);
    w.wt_mid = (__nv_bfloat16*)take(ck * Cout * 2);
    w.dw_pad = (float*)take(ck * Cout * 4);
  }
  w.bytes = (size_t)(p - (char*)ws);
  return w;
}

int check_mc_args(const char* op, int K, int C, int Cout, int64_t ns, int64_t n_in, int64_t M) {
  TFGPC_REQUIRE(valid_basis(K), "%s expects a valid number of basis functions.", op);
  TFGPC_REQUIRE(valid_features(C), "%s expects a valid number of input features, between 1 and 8 "
                "or multiple of 8", op);
  TFGPC_REQUIRE(Cout > 0 && Cout % 8 == 0, "%s expects a number of output features that is a "
                "multiple of 8", op);
  TFGPC_REQUIRE(ns >= 0 && ns < (int64_t)INT32_MAX && n_in >= 0 && n_in < (int64_t)INT32_MAX &&
                M >= 0 && M <= (int64_t)INT32_MAX, "%s expects 0 <= ns, n_in, M < 2^31", op);
  return TFGPC_OK;
}

// How the weights lie in memory.  groups > 1: `groups` kernel MLPs with K / groups
// outputs each, whose blocks [C * K/groups, Cout/groups] lie one after the other: the
// products run block by block (a dense matrix would be zero but for its diagonal
// blocks), X and dX with their columns in the order (group, channel, output).
// groups == 1: [C * k_src, cout_src], zero-padded to K basis functions and Cout columns.
struct Blocks {
  int groups, k_src, cout_src;
};

// out[(c * k_src + k), o] = padded[(c * k_dst + k), o]
__global__ void crop_weights_kernel(int64_t n, int cols, int ld, int k_src, int k_dst,
                                    const float* padded, float* __restrict__ out) {
  chain_enter();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t r = i / cols, c = r / k_src;
  out[i] = ld_global(padded + (c * k_dst + (r - c * k_src)) * ld + (i - r * cols));
}

int check_blocks(const char* op, int K, int C, int Cout, const Blocks& b) {
  TFGPC_REQUIRE(b.groups >= 1 && K % b.groups == 0 && Cout % b.groups == 0 &&
                b.k_src >= 1 && b.k_src <= K && b.cout_src >= 1 && b.cout_src <= Cout &&
                (b.groups == 1 || (b.k_src == K && b.cout_src == Cout &&
                                   tfgpc_mcconv_blocks_supported(K, C, Cout, b.groups))),
                "%s: weight blocks of this shape are not supported", op);
  return TFGPC_OK;
}

SplitJob weight_job(const McWs& w, const float* weights, int64_t ck, int K, int Cout,
                    const Blocks& b) {
  SplitJob j;
  j.x = weights;
  j.rows = ck;
  j.ld = Cout / b.groups;
  j.cols = b.groups > 1 ? j.ld : b.cout_src;
  j.k_src = b.k_src;
  j.k_dst = K;
  j.hi = w.w_hi;
  j.mid = w.w_mid;
  return j;
}

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

// Block-diagonal products need 16-byte aligned block columns, and the projection hands
// over four basis functions of one block at a time.
extern "C" int tfgpc_mcconv_blocks_supported(int K, int C, int Cout, int groups) {
  if (K <= 0 || C <= 0 || Cout <= 0 || groups < 1) return 0;
  if (groups == 1) return 1;
  if (K % groups || Cout % groups) return 0;
  const int h = K / groups, co = Cout / groups;
  return h % 4 == 0 && ((int64_t)C * h) % 8 == 0 && co % 8 == 0;
}

extern "C" size_t tfgpc_mcconv_workspace_bytes(int K, int C, int Cout, int64_t ns, int64_t n_in,
                                               int backward) {
  if (K <= 0 || C <= 0 || Cout <= 0 || ns < 0 || n_in < 0) return 0;
  return carve(nullptr, K, C, Cout, ns, n_in, backward != 0).bytes + 1024;
}

// The projection, written as the GEMM's bf16 operand pair: on tensor-core MMAs
// where the shape allows it (prepare_projection then splits the features), else on the
// SIMT kernels.
static bool on_mma(const McWs& w, const float* features) {
  return w.fs && (uintptr_t)features % 16 == 0;
}

static void prepare_projection(Prepare* jobs, const McWs& w, const float* features, int64_t n_in,
                               int C) {
  jobs->zero(w.err, sizeof(int));
  if (on_mma(w, features)) jobs->add(feature_job(features, n_in, C, w.fs));
}

static int project(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                   const float* features, const int32_t* neighbors, const int32_t* ranges,
                   const McWs& w, int hidden) {
  if (on_mma(w, features))
    return basis_proj_mma_split(st, K, C, ns, basis, w.fs, neighbors, ranges, w.x_hi, w.x_mid,
                                hidden);
  return basis_proj_split(st, K, C, ns, basis, features, neighbors, ranges, w.x_hi, w.x_mid, hidden);
}

extern "C" int tfgpc_mcconv_forward(void* stream, int K, int C, int Cout, int64_t ns, int64_t n_in,
                                    int64_t M, const float* basis, const float* features,
                                    const int32_t* neighbors, const int32_t* ranges,
                                    const float* weights, float* out, void* ws, size_t ws_bytes) {
  return tfgpc_mcconv_forward_blocks(stream, K, C, Cout, 1, K, Cout, ns, n_in, M, basis, features,
                                     neighbors, ranges, weights, out, ws, ws_bytes);
}

extern "C" int tfgpc_mcconv_forward_blocks(void* stream, int K, int C, int Cout, int groups,
                                           int k_src, int cout_src, int64_t ns, int64_t n_in,
                                           int64_t M, const float* basis, const float* features,
                                           const int32_t* neighbors, const int32_t* ranges,
                                           const float* weights, float* out, void* ws,
                                           size_t ws_bytes) {
  int rc = check_mc_args("MCConvForward", K, C, Cout, ns, n_in, M);
  if (rc) return rc;
  const Blocks blocks{groups, k_src, cout_src};
  rc = check_blocks("MCConvForward", K, C, Cout, blocks);
  if (rc) return rc;
  if (ns == 0) return TFGPC_OK;
  TFGPC_REQUIRE(ranges && weights && out && ws && (M == 0 || (basis && features && neighbors)),
                "MCConvForward got a null pointer");
  TFGPC_REQUIRE((uintptr_t)basis % 16 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)ws % 256 == 0,
                "MCConvForward expects 16-byte aligned buffers and a 256-byte aligned workspace");
  if (ws_bytes < tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 0))
    return fail(TFGPC_ENOMEM, "MCConvForward workspace too small: %zu < %zu", ws_bytes,
                tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 0));
  cudaStream_t st = (cudaStream_t)stream;
  McWs w = carve(ws, K, C, Cout, ns, n_in, false);
  const int64_t ck = (int64_t)C * K, ch = ck / groups, co = Cout / groups;
  GemmProblem p{};
  const GemmOperand x{w.x_hi, w.x_mid, ck, Major::K, ch};
  const GemmOperand wt{w.w_hi, w.w_mid, co, Major::MN, ch * co};  // [C*K, Cout]: N contiguous
  p.K = ch;
  p.c = out;
  p.ldc = Cout;
  p.batches = groups;
  p.c_batch_stride = co;
  p.transposed = forward_swapped(co);
  p.M = p.transposed ? co : ns;
  p.N = p.transposed ? ns : co;
  p.a = p.transposed ? wt : x;
  p.b = p.transposed ? x : wt;
  p.ordered = true;
  p.partials = w.partials;
  p.partial_elems = w.partial_elems;
  Prepare jobs;
  prepare_projection(&jobs, w, features, n_in, C);
  jobs.add(weight_job(w, weights, ck, K, Cout, blocks));
  p.cleared = gemm_adds_slices(p);
  if (p.cleared) jobs.zero(out, (size_t)ns * Cout * sizeof(float));
  rc = prepare(st, jobs);
  if (rc) return rc;
  rc = project(st, K, C, ns, basis, features, neighbors, ranges, w, K / groups);
  if (rc) return rc;
  return gemm_bf16x3(st, p, w.err);
}

extern "C" int tfgpc_mcconv_backward(void* stream, int K, int C, int Cout, int64_t ns,
                                     int64_t n_in, int64_t M, const float* basis,
                                     const float* features, const int32_t* neighbors,
                                     const int32_t* ranges, const float* weights,
                                     const float* out_grads, int x_in_workspace, float* dbasis_out,
                                     float* dfeat_out, float* dweights_out, void* ws,
                                     size_t ws_bytes) {
  return tfgpc_mcconv_backward_blocks(stream, K, C, Cout, 1, K, Cout, ns, n_in, M, basis, features,
                                      neighbors, ranges, weights, out_grads, x_in_workspace,
                                      dbasis_out, dfeat_out, dweights_out, ws, ws_bytes);
}

// want_basis false: without the gradient of the basis (dbasis_out is null).
static int backward_blocks(
    void* stream, int K, int C, int Cout, int groups, int k_src, int cout_src, int64_t ns,
    int64_t n_in, int64_t M, const float* basis, const float* features, const int32_t* neighbors,
    const int32_t* ranges, const float* weights, const float* out_grads, int x_in_workspace,
    bool want_basis, float* dbasis_out, float* dfeat_out, float* dweights_out, void* ws,
    size_t ws_bytes) {
  int rc = check_mc_args("MCConvBackward", K, C, Cout, ns, n_in, M);
  if (rc) return rc;
  const Blocks blocks{groups, k_src, cout_src};
  rc = check_blocks("MCConvBackward", K, C, Cout, blocks);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ck = (int64_t)C * K, ch = ck / groups, co = Cout / groups;
  const bool padded = k_src != K || cout_src != Cout;
  const int64_t weight_elems = groups > 1 ? ck * co : (int64_t)C * k_src * cout_src;
  TFGPC_REQUIRE(dweights_out && weights, "MCConvBackward got a null pointer");
  if (ns == 0 || M == 0) {
    TFGPC_CUDA(cudaMemsetAsync(dweights_out, 0, sizeof(float) * (size_t)weight_elems, st));
    if (M > 0 && dbasis_out) TFGPC_CUDA(cudaMemsetAsync(dbasis_out, 0, sizeof(float) * (size_t)M * K, st));
    if (n_in > 0 && dfeat_out) TFGPC_CUDA(cudaMemsetAsync(dfeat_out, 0, sizeof(float) * (size_t)n_in * C, st));
    return TFGPC_OK;
  }
  TFGPC_REQUIRE(basis && features && neighbors && ranges && out_grads &&
                (dbasis_out || !want_basis) && dfeat_out && ws, "MCConvBackward got a null pointer");
  TFGPC_REQUIRE((uintptr_t)basis % 16 == 0 && (uintptr_t)out_grads % 16 == 0 &&
                (uintptr_t)ws % 256 == 0,
                "MCConvBackward expects 16-byte aligned buffers and a 256-byte aligned workspace");
  if (ws_bytes < tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 1))
    return fail(TFGPC_ENOMEM, "MCConvBackward workspace too small: %zu < %zu", ws_bytes,
                tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 1));
  McWs w = carve(ws, K, C, Cout, ns, n_in, true);
  const int hidden = K / groups;
  const bool fs_ok = on_mma(w, features) && (uintptr_t)dbasis_out % 32 == 0 &&
                     (uintptr_t)dfeat_out % 16 == 0;
  TFGPC_REQUIRE(want_basis || fs_ok || basis_proj_grads_tile_takes(K, C, features),
                "MCConvBackwardFeatures expects 16-byte aligned features and feature gradients of a "
                "supported layer");
  // (Without the gradient of the basis two passes of the warp MMAs are faster than the tcgen05
  // kernel, which works that one out as well.  The whole backward at K = 16, C = Cout = 128, us,
  // tcgen05 / warp MMA, on 1024, 4096, 16 384 and 65 536 samples of 25 to 33 pairs: 44 / 37,
  // 68 / 54, 191 / 155, 759 / 603; at Cout = 256 49 / 43, 80 / 63, 222 / 188, 912 / 770.)
  const bool image = want_basis && fs_ok && groups == 1 && basis_proj_grads_tc_supported(K, C);
  // dX[ns, C*K] = dOut[ns, Cout] * W^T: B rows are W's rows, reduction over Cout
  GemmProblem px{};
  px.M = ns;
  px.N = ch;
  px.K = co;
  px.a = GemmOperand{w.g_hi, w.g_mid, (int64_t)Cout, Major::K, co};
  px.b = GemmOperand{w.w_hi, w.w_mid, co, Major::K, ch * co};
  px.c = w.dx;
  px.ldc = ck;
  px.batches = groups;
  px.c_batch_stride = ch;
  px.ordered = true;
  // dW[C*K, Cout] = X^T * dOut: both operands have the reduction (sample) index
  // as their row index, i.e. they are MN-major
  GemmProblem pw{};
  pw.M = ch;
  pw.N = co;
  pw.K = ns;
  pw.a = GemmOperand{w.x_hi, w.x_mid, ck, Major::MN, ch};
  pw.b = GemmOperand{w.g_hi, w.g_mid, (int64_t)Cout, Major::MN, co};
  pw.c = padded ? w.dw_pad : dweights_out;
  pw.ldc = co;
  pw.batches = groups;
  pw.c_batch_stride = ch * co;
  Prepare jobs;
  // (with x_in_workspace the word keeps what the forward call left: a timeout
  // there means that the projection this call is about to read is incomplete)
  if (!x_in_workspace) prepare_projection(&jobs, w, features, n_in, C);
  SplitJob gj;
  gj.x = out_grads;
  gj.rows = ns;
  gj.cols = cout_src;
  gj.ld = Cout;
  gj.hi = w.g_hi;
  gj.mid = w.g_mid;
  jobs.add(gj);
  // The weights are split again on every call (2 MB): the products below then work on
  // the values of this call's `weights`, whatever the forward call saw.
  if (!image) {
    jobs.add(weight_job(w, weights, ck, K, Cout, blocks));
    px.cleared = gemm_adds_slices(px);
    if (px.cleared) jobs.zero(w.dx, (size_t)ns * ck * sizeof(float));
  }
  pw.cleared = gemm_adds_slices(pw);
  if (pw.cleared) jobs.zero(pw.c, (size_t)ck * co * sizeof(float));
  jobs.zero(dfeat_out, (size_t)n_in * C * sizeof(float));
  if (want_basis && !fs_ok && basis_proj_grads_adds_dbasis(K, C, features))
    jobs.zero(dbasis_out, (size_t)M * K * sizeof(float));
  rc = prepare(st, jobs);
  if (rc) return rc;
  if (!x_in_workspace) {
    rc = project(st, K, C, ns, basis, features, neighbors, ranges, w, hidden);
    if (rc) return rc;
  }
  if (image) {
    // dX goes straight into the operand image of the tcgen05 gradient kernel
    const int group = basis_proj_grads_tc_group(ns, M);
    if (ns % group != 0) {
      // columns of the samples that do not exist must read as finite values
      char* last = (char*)w.dx + (size_t)(ns / group) * 4 * ck * 4;
      TFGPC_CUDA(cudaMemsetAsync(last, 0, (size_t)4 * ck * 4, st));
    }
    // dX^T = W * dOut^T with W^T [Cout, C*K] as the MN-major left operand (the
    // tensor pipe reads it faster than a K-major one; transposing 2 MB is free),
    // tiles transposed back on their way into the image
    rc = split_transpose_to_bf16(st, weights, ck, Cout, cout_src, k_src, K, w.wt_hi, w.wt_mid);
    if (rc) return rc;
    const GemmOperand wt_mn{w.wt_hi, w.wt_mid, ck, Major::MN};
    const GemmOperand g_k{w.g_hi, w.g_mid, (int64_t)Cout, Major::K};
    rc = gemm_bf16x3_grad_image_tn(st, C, ns, Cout, wt_mn, g_k, w.dx, group, w.err);
    if (rc) return rc;
    rc = basis_proj_grads_tc(st, group, ns, M, basis, w.fs, neighbors, ranges, w.dx, dbasis_out,
                             dfeat_out, w.err);
  } else {
    rc = gemm_bf16x3(st, px, w.err);
    if (rc) return rc;
    if (fs_ok)
      rc = basis_proj_grads_mma(st, K, C, ns, M, basis, w.fs, neighbors, ranges, w.dx, dbasis_out,
                                dfeat_out, hidden);
    else if (want_basis)
      rc = basis_proj_grads_blocks(st, K, C, ns, M, basis, features, neighbors, ranges, w.dx,
                                   dbasis_out, dfeat_out, hidden);
    else
      rc = basis_proj_grads_tile(st, K, C, ns, M, basis, features, (const int2*)neighbors, ranges,
                                 w.dx, nullptr, dfeat_out, hidden);
  }
  if (rc) return rc;
  rc = gemm_bf16x3(st, pw, w.err);
  if (rc || !padded) return rc;
  TFGPC_CUDA(launch_chained(st, blocks_for(weight_elems, 256), 256, 0, crop_weights_kernel,
      weight_elems, cout_src, Cout, k_src, K, w.dw_pad, dweights_out));
  return TFGPC_OK;
}

extern "C" int tfgpc_mcconv_backward_blocks(
    void* stream, int K, int C, int Cout, int groups, int k_src, int cout_src, int64_t ns,
    int64_t n_in, int64_t M, const float* basis, const float* features, const int32_t* neighbors,
    const int32_t* ranges, const float* weights, const float* out_grads, int x_in_workspace,
    float* dbasis_out, float* dfeat_out, float* dweights_out, void* ws, size_t ws_bytes) {
  return backward_blocks(stream, K, C, Cout, groups, k_src, cout_src, ns, n_in, M, basis, features,
                         neighbors, ranges, weights, out_grads, x_in_workspace, true, dbasis_out,
                         dfeat_out, dweights_out, ws, ws_bytes);
}

// (the kernels that leave out the basis read and reduce 16-byte pieces beyond eight channels)
extern "C" int tfgpc_mcconv_feature_grads_supported(int K, int C, const float* features,
                                                    const float* dfeat) {
  if (!valid_basis(K) || !valid_features(C)) return 0;
  if (basis_proj_grads_tile_takes(K, C, features)) return 1;
  return basis_proj_mma_supported(K, C) && (uintptr_t)features % 16 == 0 &&
                 (uintptr_t)dfeat % 16 == 0 ? 1 : 0;
}

extern "C" int tfgpc_mcconv_backward_features(
    void* stream, int K, int C, int Cout, int groups, int k_src, int cout_src, int64_t ns,
    int64_t n_in, int64_t M, const float* basis, const float* features, const int32_t* neighbors,
    const int32_t* ranges, const float* weights, const float* out_grads, int x_in_workspace,
    float* dfeat_out, float* dweights_out, void* ws, size_t ws_bytes) {
  return backward_blocks(stream, K, C, Cout, groups, k_src, cout_src, ns, n_in, M, basis, features,
                         neighbors, ranges, weights, out_grads, x_in_workspace, false, nullptr,
                         dfeat_out, dweights_out, ws, ws_bytes);
}

extern "C" int tfgpc_mcconv_grouped_supported(int K, int C) {
  return basis_proj_grads_tc_supported(K, C) ? 1 : 0;
}

namespace {

int check_grouped_args(const char* op, int K, int C, int Cout, const void* features,
                       const void* basis_pair, const void* ws, const void* plan) {
  TFGPC_REQUIRE(basis_proj_grads_tc_supported(K, C),
                "%s on a group plan expects K = 16 basis functions and C = 128 features", op);
  TFGPC_REQUIRE(Cout >= 128, "%s on a group plan expects at least 128 output features", op);
  TFGPC_REQUIRE((uintptr_t)features % 16 == 0 && (uintptr_t)basis_pair % 32 == 0 &&
                (uintptr_t)ws % 256 == 0 && (uintptr_t)plan % 256 == 0,
                "%s on a group plan expects 16-byte aligned features, a 32-byte aligned basis pair "
                "and 256-byte aligned workspace and plan", op);
  return TFGPC_OK;
}

}  // namespace

// Forward pass on the rows of a group plan: the projection is computed once per
// distinct neighbor of a group and written in the plan's visiting order; the
// weight GEMM puts its output rows back into the sample order.
extern "C" int tfgpc_mcconv_forward_grouped(
    void* stream, int K, int C, int Cout, int64_t ns, int64_t n_in, int64_t M,
    const void* basis_pair, const float* features, const float* weights, const int32_t* order,
    const void* plan, float* out, void* ws, size_t ws_bytes) {
  int rc = check_mc_args("MCConvForward", K, C, Cout, ns, n_in, M);
  if (rc) return rc;
  if (ns == 0) return TFGPC_OK;
  TFGPC_REQUIRE(weights && out && ws && order && plan && (M == 0 || (basis_pair && features)),
                "MCConvForward got a null pointer");
  rc = check_grouped_args("MCConvForward", K, C, Cout, features, basis_pair, ws, plan);
  if (rc) return rc;
  TFGPC_REQUIRE((uintptr_t)out % 32 == 0, "MCConvForward on a group plan expects a 32-byte aligned output");
  if (ws_bytes < tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 0))
    return fail(TFGPC_ENOMEM, "MCConvForward workspace too small: %zu < %zu", ws_bytes,
                tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 0));
  cudaStream_t st = (cudaStream_t)stream;
  McWs w = carve(ws, K, C, Cout, ns, n_in, false);
  const int64_t ck = (int64_t)C * K;
  Prepare jobs;
  jobs.zero(w.err, sizeof(int));
  jobs.add(feature_job(features, n_in, C, w.fs));
  jobs.add(weight_job(w, weights, ck, K, Cout, Blocks{1, K, Cout}));
  rc = prepare(st, jobs);
  if (rc) return rc;
  rc = basis_proj_fwd_tcu(st, ns, M, plan, (const __nv_bfloat16*)basis_pair, w.fs, w.x_hi, w.x_mid,
                          w.err);
  if (rc) return rc;
  GemmOperand a{w.x_hi, w.x_mid, ck, Major::K};
  GemmOperand b{w.w_hi, w.w_mid, (int64_t)Cout, Major::MN};
  // out^T = W^T * X^T; column v of out^T is the sample order[v]
  return gemm_bf16x3_tn_scatter(st, Cout, ns, ck, b, a, out, Cout, order, w.err);
}

// The backward pass on the rows of a group plan: dX is produced in the plan's
// visiting order (the rows of out_grads are gathered while they are split), the
// projection gradients run per distinct neighbor of a group instead of per
// pair, dW is unchanged.
extern "C" int tfgpc_mcconv_backward_grouped(
    void* stream, int K, int C, int Cout, int64_t ns, int64_t n_in, int64_t M,
    const void* basis_pair, const float* features, const int32_t* ranges, const float* weights,
    const float* out_grads, int x_in_workspace, const int32_t* order, const void* plan,
    float* dbasis_out, float* dfeat_out, float* dweights_out, void* ws, size_t ws_bytes) {
  int rc = check_mc_args("MCConvBackward", K, C, Cout, ns, n_in, M);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ck = (int64_t)C * K;
  TFGPC_REQUIRE(dweights_out && weights, "MCConvBackward got a null pointer");
  if (ns == 0 || M == 0) {
    TFGPC_CUDA(cudaMemsetAsync(dweights_out, 0, sizeof(float) * (size_t)ck * Cout, st));
    if (M > 0 && dbasis_out) TFGPC_CUDA(cudaMemsetAsync(dbasis_out, 0, sizeof(float) * (size_t)M * K, st));
    if (n_in > 0 && dfeat_out) TFGPC_CUDA(cudaMemsetAsync(dfeat_out, 0, sizeof(float) * (size_t)n_in * C, st));
    return TFGPC_OK;
  }
  TFGPC_REQUIRE(basis_pair && features && ranges && out_grads && order && plan && dbasis_out &&
                dfeat_out && ws, "MCConvBackward got a null pointer");
  rc = check_grouped_args("MCConvBackward", K, C, Cout, features, basis_pair, ws, plan);
  if (rc) return rc;
  TFGPC_REQUIRE((uintptr_t)out_grads % 16 == 0 && (uintptr_t)dbasis_out % 32 == 0 &&
                (uintptr_t)dfeat_out % 16 == 0,
                "MCConvBackward on a group plan expects 16-byte aligned gradients (dbasis 32)");
  if (ws_bytes < tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 1))
    return fail(TFGPC_ENOMEM, "MCConvBackward workspace too small: %zu < %zu", ws_bytes,
                tfgpc_mcconv_workspace_bytes(K, C, Cout, ns, n_in, 1));
  McWs w = carve(ws, K, C, Cout, ns, n_in, true);
  Prepare jobs;
  if (!x_in_workspace) {
    jobs.zero(w.err, sizeof(int));
    jobs.add(feature_job(features, n_in, C, w.fs));
  }
  // X lies in the visiting order (tfgpc_mcconv_forward_grouped wrote it so): the
  // rows of out_grads are brought into the same order while they are split, for
  // both products
  SplitJob gj;
  gj.x = out_grads;
  gj.rows = ns;
  gj.cols = gj.ld = Cout;
  gj.order = order;
  gj.hi = w.g_hi;
  gj.mid = w.g_mid;
  jobs.add(gj);
  constexpr int group = 4;
  if (ns % group != 0)
    jobs.zero((char*)w.dx + (size_t)(ns / group) * 4 * ck * 4, (size_t)4 * ck * 4);
  GemmProblem p{};
  p.M = ck;
  p.N = Cout;
  p.K = ns;
  p.a = GemmOperand{w.x_hi, w.x_mid, ck, Major::MN};
  p.b = GemmOperand{w.g_hi, w.g_mid, (int64_t)Cout, Major::MN};
  p.c = dweights_out;
  p.ldc = Cout;
  p.cleared = gemm_adds_slices(p);
  if (p.cleared) jobs.zero(dweights_out, (size_t)ck * Cout * sizeof(float));
  jobs.zero(dfeat_out, (size_t)n_in * C * sizeof(float));
  rc = prepare(st, jobs);
  if (rc) return rc;
  if (!x_in_workspace) {
    rc = basis_proj_fwd_tcu(st, ns, M, plan, (const __nv_bfloat16*)basis_pair, w.fs, w.x_hi,
                            w.x_mid, w.err);
    if (rc) return rc;
  }
  rc = split_transpose_to_bf16(st, weights, ck, Cout, Cout, K, K, w.wt_hi, w.wt_mid);
  if (rc) return rc;
  GemmOperand wt_mn{w.wt_hi, w.wt_mid, ck, Major::MN};
  GemmOperand gv_k{w.g_hi, w.g_mid, (int64_t)Cout, Major::K};
  rc = gemm_bf16x3_grad_image_tn(st, C, ns, Cout, wt_mn, gv_k, w.dx, group, w.err);
  if (rc) return rc;
  rc = basis_proj_grads_tcu(st, ns, M, plan, (const __nv_bfloat16*)basis_pair, w.fs, ranges, w.dx,
                            dbasis_out, dfeat_out, w.err);
  if (rc) return rc;
  return gemm_bf16x3(st, p, w.err);
}

extern "C" int tfgpc_mcconv_status(void* stream, const void* ws, int* status_out) {
  TFGPC_REQUIRE(ws && status_out, "mcconv_status got a null pointer");
  int flag = 0;
  int rc = read_small((cudaStream_t)stream, ws, sizeof(int), &flag);
  if (rc) return rc;
  *status_out = flag ? TFGPC_ETIMEOUT : TFGPC_OK;
  if (flag) return fail(TFGPC_ETIMEOUT, "a bounded wait inside the tensor-core GEMM ran out");
  return TFGPC_OK;
}

// ---- plain fp32 matrix product on the same GEMM -------------------------------

extern "C" size_t tfgpc_matmul_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return 1024;
  return 1024 + 2 * align_up((size_t)M * K * 2, 1024) + 2 * align_up((size_t)N * K * 2, 1024) +
         1024;
}

extern "C" int tfgpc_matmul_f32(void* stream, int64_t M, int64_t N, int64_t K, const float* a,
                                int a_transposed, const float* b, int b_transposed, float* c,
                                void* ws, size_t ws_bytes) {
  TFGPC_REQUIRE(M > 0 && N > 0 && K > 0, "matmul expects positive sizes");
  TFGPC_REQUIRE(a && b && c && ws, "matmul got a null pointer");
  TFGPC_REQUIRE((uintptr_t)ws % 256 == 0, "matmul expects a 256-byte aligned workspace");
  TFGPC_REQUIRE((a_transposed ? M : K) % 8 == 0 && (b_transposed ? K : N) % 8 == 0,
                "matmul expects row lengths that are multiples of 8");
  if (ws_bytes < tfgpc_matmul_workspace_bytes(M, N, K))
    return fail(TFGPC_ENOMEM, "matmul workspace too small: %zu < %zu", ws_bytes,
                tfgpc_matmul_workspace_bytes(M, N, K));
  cudaStream_t st = (cudaStream_t)stream;
  char* p = (char*)ws;
  int* err = (int*)p; p += 1024;
  __nv_bfloat16* a_hi = (__nv_bfloat16*)p; p += align_up((size_t)M * K * 2, 1024);
  __nv_bfloat16* a_mid = (__nv_bfloat16*)p; p += align_up((size_t)M * K * 2, 1024);
  __nv_bfloat16* b_hi = (__nv_bfloat16*)p; p += align_up((size_t)N * K * 2, 1024);
  __nv_bfloat16* b_mid = (__nv_bfloat16*)p; p += align_up((size_t)N * K * 2, 1024);
  SplitJob ja, jb;
  ja.x = a;
  ja.rows = a_transposed ? K : M;
  ja.cols = ja.ld = (int)(a_transposed ? M : K);
  ja.hi = a_hi;
  ja.mid = a_mid;
  jb.x = b;
  jb.rows = b_transposed ? N : K;
  jb.cols = jb.ld = (int)(b_transposed ? K : N);
  jb.hi = b_hi;
  jb.mid = b_mid;
  // a is [M,K] (K-major) or, transposed, [K,M] (MN-major); b is [K,N] (MN-major)
  // or, transposed, [N,K] (K-major)
  GemmProblem g{};
  g.M = M;
  g.N = N;
  g.K = K;
  g.a = GemmOperand{a_hi, a_mid, a_transposed ? M : K, a_transposed ? Major::MN : Major::K};
  g.b = GemmOperand{b_hi, b_mid, b_transposed ? K : N, b_transposed ? Major::K : Major::MN};
  g.c = c;
  g.ldc = N;
  Prepare jobs;
  jobs.zero(err, sizeof(int));
  jobs.add(ja);
  jobs.add(jb);
  g.cleared = gemm_adds_slices(g);
  if (g.cleared) jobs.zero(c, (size_t)M * N * sizeof(float));
  int rc = prepare(st, jobs);
  if (rc) return rc;
  return gemm_bf16x3(st, g, err);
}

// ---- Conv1x1 ------------------------------------------------------------------------

namespace {
inline int64_t up8(int64_t v) { return (v + 7) / 8 * 8; }
}  // namespace

extern "C" size_t tfgpc_linear_workspace_bytes(int64_t n, int64_t cin, int64_t cout) {
  if (n <= 0 || cin <= 0 || cout <= 0) return 1024;
  return 2 * align_up((size_t)n * up8(cin) * 2, 1024) +
         2 * align_up((size_t)cin * up8(cout) * 2, 1024);
}

extern "C" int tfgpc_linear_f32(void* stream, int64_t n, int64_t cin, int64_t cout, const float* x,
                                const float* weights, const float* bias, float* out, int* status,
                                void* ws, size_t ws_bytes) {
  TFGPC_REQUIRE(n > 0 && cin > 0 && cout > 0 && cin < (1 << 30) && cout < (1 << 30),
                "Conv1x1 expects positive sizes");
  TFGPC_REQUIRE(x && weights && out && status && ws, "Conv1x1 got a null pointer");
  TFGPC_REQUIRE((uintptr_t)ws % 256 == 0 && (uintptr_t)out % 16 == 0,
                "Conv1x1 expects a 256-byte aligned workspace and a 16-byte aligned output");
  if (ws_bytes < tfgpc_linear_workspace_bytes(n, cin, cout))
    return fail(TFGPC_ENOMEM, "Conv1x1 workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  char* p = (char*)ws;
  auto take = [&](size_t b) { char* r = p; p += align_up(b, 1024); return (__nv_bfloat16*)r; };
  SplitJob jx, jw;
  jx.x = x;
  jx.rows = n;
  jx.cols = (int)cin;
  jx.ld = (int)up8(cin);
  jx.hi = take((size_t)n * jx.ld * 2);
  jx.mid = take((size_t)n * jx.ld * 2);
  jw.x = weights;
  jw.rows = cin;
  jw.cols = (int)cout;
  jw.ld = (int)up8(cout);
  jw.hi = take((size_t)cin * jw.ld * 2);
  jw.mid = take((size_t)cin * jw.ld * 2);
  const GemmOperand xo{jx.hi, jx.mid, jx.ld, Major::K}, wo{jw.hi, jw.mid, jw.ld, Major::MN};
  GemmProblem g{};
  g.K = cin;
  g.transposed = cout >= 128;    // (see gemm_bf16x3)
  g.M = g.transposed ? cout : n;
  g.N = g.transposed ? n : cout;
  g.a = g.transposed ? wo : xo;
  g.b = g.transposed ? xo : wo;
  g.c = out;
  g.ldc = up8(cout);
  g.bias = bias;
  Prepare jobs;
  jobs.add(jx);
  jobs.add(jw);
  g.cleared = g.ldc == cout && gemm_adds_slices(g);
  if (g.cleared) jobs.zero(out, (size_t)n * cout * sizeof(float));
  int rc = prepare(st, jobs);
  if (rc) return rc;
  return gemm_bf16x3(st, g, status);
}
