// Kernel bases, projection and weight products, pooling and the 1x1 convolution.
#include "host.h"

namespace tfgpc_host {
namespace {

const float* maybe(const OptTensor& t, Tensor* keep) {
  if (!t) return nullptr;
  *keep = f32(*t);
  return fp(*keep);
}

// ---- kernel bases ------------------------------------------------------------------

Tensor pack_points_density(const Tensor& points_, const Tensor& pdf_) {
  Tensor points = f32(points_), pdf = f32(pdf_);
  const int64_t n = points.size(0);
  require(points.size(1) == 3 && pdf.numel() == n,
          "PackPointsDensity expects [n, 3] points and [n] densities");
  Tensor out = empty({n, 4}, at::kFloat, points);
  check(tfgpc_pack_points_density(stream(), n, fp(points), fp(pdf), fpm(out)));
  return out;
}

// Weights of one-layer kernel MLPs: [D, K], or [G, D, K / G] as a layer holds G of them.
struct OneLayer {
  int d, k, g;
  explicit OneLayer(const Tensor& w1) {
    require(w1.dim() == 2 || w1.dim() == 3, "KernelBasis expects weights [D, K] or [G, D, K / G]");
    g = w1.dim() == 3 ? (int)w1.size(0) : 1;
    d = (int)w1.size(-2);
    k = g * (int)w1.size(-1);
  }
};

// (basis [M, K] float32 or None, pair [M, 2, K] bf16 or None)
py::tuple kernel_basis(const Tensor& p_in_, const Tensor& p_out_, const Tensor& neigh_,
                       const OptTensor& pdf_, const Tensor& w1_, const Tensor& b1_,
                       double radius, int act, double alpha, int pdf_mode, bool want_f32,
                       bool want_pair) {
  Tensor p_in = f32(p_in_), p_out = f32(p_out_), neigh = i32(neigh_), w1 = f32(w1_), b1 = f32(b1_);
  Tensor pdf_keep;
  const float* pdf = maybe(pdf_, &pdf_keep);
  const OneLayer mlp(w1);
  const int64_t m = neigh.size(0);
  OptTensor basis, pair;
  if (want_f32) basis = empty({m, mlp.k}, at::kFloat, p_in);
  if (want_pair) pair = empty({m, 2, mlp.k}, at::kBFloat16, p_in);
  check(tfgpc_kernel_basis_mlps(stream(), mlp.d, mlp.k, mlp.g, m, fp(p_in), fp(p_out), ip(neigh),
                                pdf, fp(w1), fp(b1), (float)(1.0 / radius), act, (float)alpha,
                                pdf_mode, basis ? fpm(*basis) : nullptr,
                                pair ? pair->data_ptr() : nullptr));
  return py::make_tuple(basis, pair);
}

// (gradient of the weights in their layout, of the biases [K])
py::tuple kernel_basis_grads(const Tensor& p_in_, const Tensor& p_out_, const Tensor& neigh_,
                             const OptTensor& pdf_, const Tensor& w1_, const Tensor& b1_,
                             double radius, const Tensor& dbasis_, int act, double alpha,
                             int pdf_mode) {
  Tensor p_in = f32(p_in_), p_out = f32(p_out_), neigh = i32(neigh_), w1 = f32(w1_), b1 = f32(b1_),
         dbasis = f32(dbasis_);
  Tensor pdf_keep;
  const float* pdf = maybe(pdf_, &pdf_keep);
  const OneLayer mlp(w1);
  Tensor dw = empty(w1.sizes(), at::kFloat, p_in), db = empty({mlp.k}, at::kFloat, p_in);
  check(tfgpc_kernel_basis_mlps_grads(stream(), mlp.d, mlp.k, mlp.g, neigh.size(0), fp(p_in),
                                      fp(p_out), ip(neigh), pdf, fp(w1), fp(b1),
                                      (float)(1.0 / radius), act, (float)alpha, pdf_mode,
                                      fp(dbasis), fpm(dw), fpm(db)));
  return py::make_tuple(dw, db);
}

// Parameters of a kernel MLP, one tensor per layer: weights [G, H_{l-1}, H_l], biases
// [G, 1, H_l].
struct Mlp {
  std::vector<Tensor> w, b;
  std::vector<const float*> wp, bp;
  std::vector<int32_t> sizes;
  int d, g;
  Mlp(const std::vector<Tensor>& weights, const std::vector<Tensor>& biases) {
    require(!weights.empty() && weights.size() == biases.size(),
            "KernelMlp expects one bias per layer");
    for (size_t l = 0; l < weights.size(); ++l) {
      w.push_back(f32(weights[l]));
      b.push_back(f32(biases[l]));
      wp.push_back(fp(w[l]));
      bp.push_back(fp(b[l]));
      sizes.push_back((int32_t)w[l].size(2));
    }
    g = (int)w[0].size(0);
    d = (int)w[0].size(1);
  }
  int layers() const { return (int)sizes.size(); }
};

Tensor kernel_mlp_basis(const Tensor& p_in_, const Tensor& p_out_, const Tensor& neigh_,
                        const Tensor& pdf_, const std::vector<Tensor>& weights,
                        const std::vector<Tensor>& biases, double radius, int act, double alpha,
                        bool pdf_by_nbr) {
  Tensor p_in = f32(p_in_), p_out = f32(p_out_), neigh = i32(neigh_), pdf = f32(pdf_);
  Mlp mlp(weights, biases);
  const int64_t m = neigh.size(0);
  Tensor basis = empty({m, (int64_t)mlp.g * mlp.sizes.back()}, at::kFloat, p_in);
  check(tfgpc_kernel_mlp_basis_layers(stream(), mlp.d, mlp.g, mlp.layers(), mlp.sizes.data(), m,
                                      fp(p_in), fp(p_out), ip(neigh), fp(pdf), mlp.wp.data(),
                                      mlp.bp.data(), (float)(1.0 / radius), act, (float)alpha,
                                      pdf_by_nbr, fpm(basis)));
  return basis;
}

// (d_weights, d_biases[, d_points_in, d_points_out, d_pdf])
py::tuple kernel_mlp_grads(const Tensor& p_in_, const Tensor& p_out_, const Tensor& neigh_,
                           const Tensor& pdf_, const std::vector<Tensor>& weights,
                           const std::vector<Tensor>& biases, double radius,
                           const Tensor& dbasis_, int act, double alpha, bool point_grads,
                           bool pdf_by_nbr) {
  Tensor p_in = f32(p_in_), p_out = f32(p_out_), neigh = i32(neigh_), pdf = f32(pdf_),
         dbasis = f32(dbasis_);
  Mlp mlp(weights, biases);
  int64_t nw = 0, nb = 0;
  for (int l = 0; l < mlp.layers(); ++l) {
    nw += mlp.w[l].numel();
    nb += mlp.b[l].numel();
  }
  Tensor flat = empty({nw + nb}, at::kFloat, p_in);
  const int64_t m = neigh.size(0);
  OptTensor dpin, dpout, dpdf;
  if (point_grads) {
    dpin = at::empty_like(p_in);
    dpout = p_out.data_ptr() == p_in.data_ptr() ? *dpin : at::empty_like(p_out);
    dpdf = empty({m}, at::kFloat, pdf);
  }
  check(tfgpc_kernel_mlp_grads_layers(
      stream(), mlp.d, mlp.g, mlp.layers(), mlp.sizes.data(), m, p_in.size(0), p_out.size(0),
      fp(p_in), fp(p_out), ip(neigh), fp(pdf), mlp.wp.data(), mlp.bp.data(),
      (float)(1.0 / radius), act, (float)alpha, pdf_by_nbr, fp(dbasis), fpm(flat), fpm(flat) + nw,
      dpin ? fpm(*dpin) : nullptr, dpout ? fpm(*dpout) : nullptr, dpdf ? fpm(*dpdf) : nullptr));
  py::list dw, db;
  int64_t ow = 0, ob = nw;
  for (int l = 0; l < mlp.layers(); ++l) {
    dw.append(flat.narrow(0, ow, mlp.w[l].numel()).view(mlp.w[l].sizes()));
    db.append(flat.narrow(0, ob, mlp.b[l].numel()).view(mlp.b[l].sizes()));
    ow += mlp.w[l].numel();
    ob += mlp.b[l].numel();
  }
  if (!point_grads) return py::make_tuple(dw, db);
  py::object a = py::cast(*dpin);      // one cloud: one gradient, the same object twice
  py::object b = dpout->data_ptr() == dpin->data_ptr() ? a : py::cast(*dpout);
  return py::make_tuple(dw, db, a, b, *dpdf);
}

// [n] sums of values [M] over the pairs of every point (first index)
Tensor add_by_neighbor(const Tensor& neigh_, const Tensor& values_, int64_t n) {
  on_gpu(neigh_);
  require(values_.device() == neigh_.device(),
          "AddByNeighbor expects the values on the device of the neighbor list");
  require(neigh_.dim() == 2 && neigh_.size(1) == 2 && values_.dim() == 1 &&
              values_.size(0) == neigh_.size(0),
          "AddByNeighbor expects one value and two indices per pair");
  Tensor neigh = i32(neigh_), values = f32(values_);
  Tensor out = empty({n}, at::kFloat, values);
  check(tfgpc_add_by_neighbor(stream(), neigh.size(0), ip(neigh), fp(values), n, fpm(out)));
  return out;
}

Tensor kp_basis(const Tensor& p_in_, const Tensor& p_out_, const Tensor& neigh_,
                const Tensor& kernel_points_, double radius, double sigma, int64_t k_pad,
                int interpolation) {
  Tensor p_in = f32(p_in_), p_out = f32(p_out_), neigh = i32(neigh_), kp = f32(kernel_points_);
  const int64_t m = neigh.size(0);
  Tensor basis = empty({m, k_pad}, at::kFloat, p_in);
  check(tfgpc_kp_basis(stream(), (int)kp.size(1), (int)k_pad, (int)kp.size(0), m, fp(p_in),
                       fp(p_out), ip(neigh), fp(kp), (float)(1.0 / radius), (float)sigma,
                       interpolation, fpm(basis)));
  return basis;
}

Tensor pointconv_pdf(const Tensor& pdf_, const Tensor& ranges_, const Tensor& w1_,
                     const Tensor& b1_, const Tensor& w2_, const Tensor& b2_,
                     const OptTensor& neigh_) {
  Tensor pdf = f32(pdf_), ranges = i32(ranges_), w1 = f32(w1_), b1 = f32(b1_), w2 = f32(w2_),
         b2 = f32(b2_);
  require(w1.numel() == 16 && b1.numel() == 16 && w2.numel() == 16 && b2.numel() == 1,
          "PointConv's density transform has 16 hidden units");
  if (neigh_) {
    Tensor neigh = i32(*neigh_);
    require(neigh.dim() == 2 && neigh.size(1) == 2, "PointConvPdf expects two indices per pair");
    Tensor out = empty({neigh.size(0)}, at::kFloat, pdf);
    check(tfgpc_pointconv_pdf_by_neighbor(stream(), ranges.size(0), neigh.size(0), ip(ranges),
                                          ip(neigh), fp(pdf), fp(w1), fp(b1), fp(w2), fp(b2),
                                          fpm(out)));
    return out;
  }
  Tensor out = at::empty_like(pdf);
  check(tfgpc_pointconv_pdf(stream(), ranges.size(0), pdf.numel(), ip(ranges), fp(pdf), fp(w1),
                            fp(b1), fp(w2), fp(b2), fpm(out)));
  return out;
}

// ---- projection + weight product ------------------------------------------------------

Tensor group_plan(const Tensor& order_, const Tensor& ranges_, const Tensor& sorted_pairs_,
                  const Tensor& original_pairs_) {
  Tensor order = i32(order_), ranges = i32(ranges_), a = i32(sorted_pairs_),
         b = i32(original_pairs_);
  const int64_t ns = ranges.size(0), m = a.size(0);
  const size_t need = tfgpc_mcconv_group_plan_bytes(ns, m);
  Tensor plan = bytes(need, ranges);
  check(tfgpc_mcconv_group_plan(stream(), ns, m, ip(order), ip(ranges), ip(a), ip(b),
                                plan.data_ptr(), need));
  return plan;
}

// The kernels index with the layer's sizes: what they are given has to match them.
// (weights and gradients by their number of values: they come in several shapes)
void check_projection(int k, int c, int64_t rows, int64_t pairs, int64_t weight_elems,
                      int64_t weight_expected, const Tensor& features) {
  require(k > 0 && c > 0 && rows == pairs, "MCConv expects one basis row per neighbor pair");
  require(features.dim() == 2 && features.size(1) == c,
          "MCConv expects features with the layer's number of channels");
  require(weight_elems == weight_expected,
          "MCConv expects weights of the layer's basis functions, input and output features");
}

int64_t weight_elems(int k, int c, int cout, int groups, int k_src, int cout_src) {
  return groups > 1 ? (int64_t)k * c * (cout / groups) : (int64_t)c * k_src * cout_src;
}

void check_pairs(int k, const Tensor& basis, const Tensor& neigh) {
  require(basis.dim() == 2 && basis.size(1) == k, "MCConv expects a basis row of the layer's width");
  require(neigh.dim() == 2 && neigh.size(1) == 2, "MCConv expects two indices per neighbor pair");
}

// groups, k_src, cout_src: how the weights lie (tfgpc_mcconv_forward_blocks)
Tensor project_forward(int k, int c, int cout, int groups, int k_src, int cout_src,
                       const Tensor& ws, const Tensor& basis_, const Tensor& features_,
                       const Tensor& neigh_, const Tensor& ranges_, const Tensor& weights_) {
  Tensor basis = f32(basis_), features = f32(features_), neigh = i32(neigh_), ranges = i32(ranges_),
         weights = f32(weights_);
  const int64_t ns = ranges.size(0);
  check_pairs(k, basis, neigh);
  check_projection(k, c, basis.size(0), neigh.size(0), weights.numel(),
                   weight_elems(k, c, cout, groups, k_src, cout_src), features);
  Tensor out = empty({ns, cout}, at::kFloat, basis);
  check(tfgpc_mcconv_forward_blocks(stream(), k, c, cout, groups, k_src, cout_src, ns,
                                    features.size(0), basis.size(0), fp(basis), fp(features),
                                    ip(neigh), ip(ranges), fp(weights), fpm(out), ws.data_ptr(),
                                    (size_t)ws.numel()));
  return out;
}

py::tuple project_backward(int k, int c, int cout, int groups, int k_src, int cout_src,
                           const Tensor& ws, const Tensor& basis_, const Tensor& features_,
                           const Tensor& neigh_, const Tensor& ranges_, const Tensor& weights_,
                           const Tensor& out_grads_, bool reuse, bool want_basis) {
  Tensor basis = f32(basis_), features = f32(features_), neigh = i32(neigh_), ranges = i32(ranges_),
         weights = f32(weights_), g = f32(out_grads_);
  check_pairs(k, basis, neigh);
  check_projection(k, c, basis.size(0), neigh.size(0), weights.numel(),
                   weight_elems(k, c, cout, groups, k_src, cout_src), features);
  require(g.numel() == ranges.size(0) * (groups > 1 ? cout : cout_src),
          "MCConv expects one gradient per output feature of every sample");
  Tensor dfeat = at::empty_like(features), dw = at::empty_like(weights);
  if (!want_basis && tfgpc_mcconv_feature_grads_supported(k, c, fp(features), fp(dfeat))) {
    check(tfgpc_mcconv_backward_features(stream(), k, c, cout, groups, k_src, cout_src,
                                         ranges.size(0), features.size(0), basis.size(0), fp(basis),
                                         fp(features), ip(neigh), ip(ranges), fp(weights), fp(g),
                                         reuse, fpm(dfeat), fpm(dw), ws.data_ptr(),
                                         (size_t)ws.numel()));
    return py::make_tuple(py::none(), dfeat, dw);
  }
  Tensor dbasis = at::empty_like(basis);
  check(tfgpc_mcconv_backward_blocks(stream(), k, c, cout, groups, k_src, cout_src,
                                     ranges.size(0), features.size(0), basis.size(0), fp(basis),
                                     fp(features), ip(neigh), ip(ranges), fp(weights), fp(g), reuse,
                                     fpm(dbasis), fpm(dfeat), fpm(dw), ws.data_ptr(),
                                     (size_t)ws.numel()));
  return py::make_tuple(dbasis, dfeat, dw);
}

void check_group_plan(int k, int c, int cout, int64_t ns, const Tensor& pair,
                      const Tensor& features, const Tensor& weights, const Tensor& order,
                      const Tensor& plan) {
  require(pair.dim() == 3 && pair.size(1) == 2 && pair.size(2) == k && pair.is_contiguous() &&
              pair.scalar_type() == at::kBFloat16,
          "MCConv expects the basis as bf16 pairs of the layer's width");
  check_projection(k, c, pair.size(0), pair.size(0), weights.numel(), (int64_t)k * c * cout,
                   features);
  require(order.numel() == ns &&
              (size_t)plan.numel() >= tfgpc_mcconv_group_plan_bytes(ns, pair.size(0)),
          "MCConv expects the group plan of these samples and pairs");
}

Tensor project_forward_grouped(int k, int c, int cout, int64_t ns, const Tensor& ws,
                               const Tensor& pair, const Tensor& features_, const Tensor& weights_,
                               const Tensor& order_, const Tensor& plan) {
  Tensor features = f32(features_), weights = f32(weights_), order = i32(order_);
  check_group_plan(k, c, cout, ns, pair, features, weights, order, plan);
  Tensor out = empty({ns, cout}, at::kFloat, features);
  check(tfgpc_mcconv_forward_grouped(stream(), k, c, cout, ns, features.size(0), pair.size(0),
                                     pair.data_ptr(), fp(features), fp(weights), ip(order),
                                     plan.data_ptr(), fpm(out), ws.data_ptr(), (size_t)ws.numel()));
  return out;
}

py::tuple project_backward_grouped(int k, int c, int cout, int64_t ns, const Tensor& ws,
                                   const Tensor& pair, const Tensor& features_,
                                   const Tensor& ranges_, const Tensor& weights_,
                                   const Tensor& out_grads_, bool reuse, const Tensor& order_,
                                   const Tensor& plan) {
  Tensor features = f32(features_), ranges = i32(ranges_), weights = f32(weights_),
         g = f32(out_grads_), order = i32(order_);
  const int64_t m = pair.size(0);
  check_group_plan(k, c, cout, ns, pair, features, weights, order, plan);
  require(g.numel() == ns * cout && ranges.size(0) == ns,
          "MCConv expects one gradient per output feature of every sample");
  Tensor dbasis = empty({m, pair.size(2)}, at::kFloat, features);
  Tensor dfeat = at::empty_like(features), dw = at::empty_like(weights);
  check(tfgpc_mcconv_backward_grouped(stream(), k, c, cout, ns, features.size(0), m,
                                      pair.data_ptr(), fp(features), ip(ranges), fp(weights),
                                      fp(g), reuse, ip(order), plan.data_ptr(), fpm(dbasis),
                                      fpm(dfeat), fpm(dw), ws.data_ptr(), (size_t)ws.numel()));
  return py::make_tuple(dbasis, dfeat, dw);
}

// Status word of a product, or of the workspace that begins with it; blocks on the stream.
void check_status(const Tensor& ws) {
  int status = 0, rc;
  void* st = stream();
  {
    py::gil_scoped_release release;
    rc = tfgpc_mcconv_status(st, ws.data_ptr(), &status);
  }
  check(rc);
}

Tensor matmul_f32(const Tensor& a_, const Tensor& b_, bool a_t, bool b_t) {
  Tensor a = f32(a_), b = f32(b_);
  const int64_t m = a.size(a_t ? 1 : 0), k = a.size(a_t ? 0 : 1), n = b.size(b_t ? 0 : 1);
  require(b.size(b_t ? 1 : 0) == k, "matmul expects matching inner dimensions");
  Tensor c = empty({m, n}, at::kFloat, a);
  const size_t need = tfgpc_matmul_workspace_bytes(m, n, k);
  Tensor ws = bytes(need, a);
  check(tfgpc_matmul_f32(stream(), m, n, k, fp(a), a_t, fp(b), b_t, fpm(c), ws.data_ptr(), need));
  check_status(ws);
  return c;
}

// ---- the drop-in projection op ----------------------------------------------------------

struct ProjArgs {
  Tensor basis, features, neigh, ranges, ws;
  int k, c;
  ProjArgs(const Tensor& b, const Tensor& f, const Tensor& nb, const Tensor& r, bool scratch)
      : basis(f32(b)), features(f32(f)), neigh(i32(nb)), ranges(i32(r)) {
    for (const Tensor* t : {&basis, &features, &neigh, &ranges}) on_gpu(*t);
    require(neigh.dim() == 2 && neigh.size(1) == 2,
            "BasisProjOp expects a neighbor tensor with 2 dimensions and 2 indices per neighbor.");
    require(basis.size(0) == neigh.size(0),
            "BasisProjOp expects the same number of basis as the number of neighbors.");
    k = (int)basis.size(1);
    c = (int)features.size(1);
    const size_t need = scratch ? tfgpc_basis_proj_workspace_bytes(k, c, features.size(0)) : 0;
    if (need) ws = bytes(need, features);
  }
  void* ws_ptr() const { return ws.defined() ? ws.data_ptr() : nullptr; }
  size_t ws_bytes() const { return ws.defined() ? (size_t)ws.numel() : 0; }
};

Tensor basis_proj(const Tensor& basis, const Tensor& features, const Tensor& neigh,
                  const Tensor& ranges, bool scratch) {
  ProjArgs a(basis, features, neigh, ranges, scratch);
  const int64_t ns = a.ranges.size(0);
  Tensor out = empty({ns, a.c, a.k}, at::kFloat, a.basis);
  check(tfgpc_basis_proj_ws(stream(), a.k, a.c, ns, a.features.size(0), a.basis.size(0),
                            fp(a.basis), fp(a.features), ip(a.neigh), ip(a.ranges), fpm(out),
                            a.ws_ptr(), a.ws_bytes()));
  return out;
}

py::tuple basis_proj_grads(const Tensor& basis, const Tensor& features, const Tensor& neigh,
                           const Tensor& ranges, const Tensor& in_grads, bool scratch) {
  ProjArgs a(basis, features, neigh, ranges, scratch);
  Tensor g = f32(in_grads);
  const int64_t ns = a.ranges.size(0);
  require(g.dim() == 3 && g.size(0) == ns && g.size(1) == a.c && g.size(2) == a.k,
          "BasisProjGradsOp expects gradients of shape [Ns, C, K]");
  Tensor dbasis = at::empty_like(a.basis), dfeat = at::empty_like(a.features);
  check(tfgpc_basis_proj_grads_ws(stream(), a.k, a.c, ns, a.features.size(0), a.basis.size(0),
                                  fp(a.basis), fp(a.features), ip(a.neigh), ip(a.ranges), fp(g),
                                  fpm(dbasis), fpm(dfeat), a.ws_ptr(), a.ws_bytes()));
  return py::make_tuple(dbasis, dfeat);
}

// ---- pooling, bias, activation ------------------------------------------------------------

Tensor neighborhood_pool(const Tensor& features_, const Tensor& neigh_, const Tensor& ranges_,
                         int mode) {
  Tensor features = f32(features_), neigh = i32(neigh_), ranges = i32(ranges_);
  const int64_t ns = ranges.size(0), c = features.size(1);
  Tensor out = empty({ns, c}, at::kFloat, features);
  check(tfgpc_neighborhood_pool(stream(), mode, (int)c, ns, features.size(0), neigh.size(0),
                                fp(features), ip(neigh), ip(ranges), fpm(out)));
  return out;
}

Tensor global_pool(const Tensor& features_, const Tensor& ids_, int64_t batch, int mode) {
  Tensor features = f32(features_), ids = i32(ids_);
  const int64_t n = features.size(0), c = features.size(1);
  Tensor out = empty({batch, c}, at::kFloat, features);
  const size_t need = tfgpc_global_pool_workspace_bytes(batch);
  Tensor ws = bytes(need, features);
  check(tfgpc_global_pool(stream(), mode, (int)c, n, batch, fp(features), ip(ids), fpm(out),
                          ws.data_ptr(), need));
  return out;
}

// x [N, C_in] @ weights [C_in, C_out] + bias; C_out that is not a multiple of 8 comes
// back as the front columns of a wider array.  status: an int32 that check_status reads
// before the result is used.
Tensor linear(const Tensor& x_, const Tensor& weights_, const Tensor& bias_,
              const Tensor& status) {
  Tensor x = f32(x_), weights = f32(weights_), bias = f32(bias_);
  const int64_t n = x.size(0), cin = x.size(1), cout = weights.size(1);
  require(weights.size(0) == cin, "matmul expects matching inner dimensions");
  require(bias.numel() == cout, "Conv1x1 expects one bias per output feature");
  require(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1,
          "Conv1x1 expects an int32 status word on the GPU");
  Tensor out = empty({n, (cout + 7) / 8 * 8}, at::kFloat, x);
  const size_t need = tfgpc_linear_workspace_bytes(n, cin, cout);
  Tensor ws = bytes(need, x);
  check(tfgpc_linear_f32(stream(), n, cin, cout, fp(x), fp(weights), fp(bias), fpm(out),
                         ipm(status), ws.data_ptr(), need));
  return out.size(1) == cout ? out : out.narrow(1, 0, cout);
}

void scale_bias_activation_(const Tensor& x, double scale, const OptTensor& bias_, bool act,
                            double alpha) {
  require(x.is_contiguous() && x.scalar_type() == at::kFloat,
          "scale_bias_activation_ expects a contiguous float32 tensor");
  Tensor keep;
  const float* bias = maybe(bias_, &keep);
  check(tfgpc_scale_bias_activation(stream(), x.size(0), (int)x.size(1), fpm(x), (float)scale, bias,
                                    act, (float)alpha));
}

}  // namespace

void bind_layers(py::module_& m) {
  m.def("pack_points_density", &pack_points_density);
  m.def("kernel_basis", &kernel_basis);
  m.def("kernel_basis_grads", &kernel_basis_grads);
  m.def("kernel_mlp_basis", &kernel_mlp_basis);
  m.def("kernel_mlp_grads", &kernel_mlp_grads);
  m.def("add_by_neighbor", &add_by_neighbor);
  m.def("kp_basis", &kp_basis);
  m.def("pointconv_pdf", &pointconv_pdf);
  m.def("group_plan", &group_plan);
  m.def("project_forward", &project_forward);
  m.def("project_backward", &project_backward);
  m.def("project_forward_grouped", &project_forward_grouped);
  m.def("project_backward_grouped", &project_backward_grouped);
  m.def("check_status", &check_status);
  m.def("matmul_f32", &matmul_f32);
  m.def("basis_proj", &basis_proj);
  m.def("basis_proj_grads", &basis_proj_grads);
  m.def("neighborhood_pool", &neighborhood_pool);
  m.def("global_pool", &global_pool);
  m.def("linear", &linear);
  m.def("blocks_supported", &tfgpc_mcconv_blocks_supported);
  m.def("scale_bias_activation_", &scale_bias_activation_);
}

}  // namespace tfgpc_host
