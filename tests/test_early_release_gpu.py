"""Chains behind a kernel of the library that lets its successor be set up at once and then
works for a while: their inputs are half their values until it has finished."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import mcconv, pc

pytestmark = pytest.mark.gpu
DEV = "cuda"
# eight turns of scale_bias_activation_'s grid on 148 SMs: the most for which it releases its
# successor early; the tensors stand at the end, which is written last
BUFFER = 4_800_000


def late(*tensors):
  """The same tensors, still being written by one kernel: nothing is enqueued behind it."""
  buf = torch.zeros(BUFFER, device=DEV)
  views, end = [], BUFFER
  for t in tensors:
    begin = (end - t.numel()) // 16 * 16
    buf[begin:begin + t.numel()] = t.reshape(-1) * 0.5
    views.append(buf[begin:begin + t.numel()].view(t.shape))
    end = begin
  torch.cuda.synchronize()
  mcconv.scale_bias_activation_(buf.view(-1, 4), 2.0)
  return views


def flat(o):
  return [x for y in o for x in flat(y)] if isinstance(o, (list, tuple)) else [o]


def check(run, *tensors):
  torch.cuda.synchronize()
  want = flat(run(*tensors))
  torch.cuda.synchronize()
  for _ in range(4):
    for x, y in zip(flat(run(*late(*tensors))), want):
      # sums by atomics: a few float32 roundings of at most 1e5 terms, 1e5^0.5 * 6e-8
      assert x.shape == y.shape and (x.double() - y.double()).norm() <= 2e-5 * y.double().norm()


def world(n, seed=7):
  g = torch.Generator(device=DEV).manual_seed(seed)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  pts = torch.rand((n, 3), generator=g, device=DEV)
  return pts, torch.zeros(n, dtype=torch.int32, device=DEV), r


# one cluster builds the smaller grid, separate kernels the larger one
@pytest.mark.parametrize("n,radius", [(900, 0.15), (6000, 0.1), (150000, 0.03)])
def test_grid_search_and_density(n, radius):
  pts, ids, _ = world(n)

  def run(p):
    cloud = pc.PointCloud(p, ids, 1)
    nb = pc.grid_neighborhood_with_pdf(cloud, radius, cloud)
    return nb._samples_neigh_ranges, nb._neighbors, nb.pdf_by_neighbor_id(), nb._packed

  check(run, pts)


@pytest.mark.parametrize("mode", ["poisson", "average"])
@pytest.mark.parametrize("n", [6000, 150000])
def test_hierarchies(n, mode):
  pts, ids, _ = world(n)
  check(lambda p: [c._points for c in
                   pc.PointHierarchy(pc.PointCloud(p, ids, 1), [0.04, 0.08], mode)._point_clouds[1:]],
        pts)


def test_layers_and_pooling():
  n, cin, k, cout = 3000, 32, 16, 64
  pts, ids, r = world(n)
  cloud = pc.PointCloud(pts, ids, 1)
  nb = pc.grid_neighborhood(cloud, 0.12, cloud)
  pdf, pairs, ranges = nb.get_pdf(bandwidth=0.2), nb._original_neigh_ids, nb._samples_neigh_ranges
  m = pairs.shape[0]
  basis, feat = r(m, k), r(n, cin)
  check(lambda f: mcconv.neighborhood_pool(f, nb, "max"), feat)
  check(lambda f: mcconv.neighborhood_pool(f, nb, "avg"), feat)
  check(lambda f: mcconv.global_pool(f, cloud, "avg"), feat)
  check(lambda b, f: ops.basis_proj(b, f, pairs, ranges), basis, feat)
  check(lambda b, f, u: ops.basis_proj_grads(b, f, pairs, ranges, u), basis, feat, r(n, cin, k))
  check(lambda p, w, b: mcconv.kernel_basis(p, p, pairs, pdf, w, b, 0.12, 1), pts, r(3, k), r(k))
  check(lambda p, w, b, u: mcconv.kernel_basis_grads(p, p, pairs, pdf, w, b, 0.12, u, 1),
        pts, r(3, k), r(k), r(m, k))
  for widths in ((8, 16), (16, 16)):      # in registers, and the general kernel
    ws = [r(1, a, b) for a, b in zip((3,) + widths, widths)]
    bs = [r(1, 1, b) for b in widths]
    check(lambda p, *par: mcconv.kernel_mlp_basis(p, p, pairs, pdf, par[:2], par[2:], 0.12, 1),
          pts, *ws, *bs)
    check(lambda p, u, *par: mcconv.kernel_mlp_grads(p, p, pairs, pdf, par[:2], par[2:], 0.12, u, 1),
          pts, r(m, widths[-1]), *ws, *bs)
  check(lambda g: nb.pdf_point_grads(g), torch.rand(m, device=DEV))
  status = mcconv.product_status(DEV)
  check(lambda x, w, b: mcconv.conv1x1(x, w, b, status), r(n, 48), r(48, 40), r(1, 40))
  op = mcconv.ProjectionGemm(k, cin, cout, n, DEV, n_in=n)
  check(lambda b, f, w: op.forward(b, f, pairs, ranges, w).clone(), basis, feat, r(cin * k, cout))
