"""Kernels that are set up while their predecessor runs (launch_chained) behind kernels of
torch, which let nothing come early, and replayed from a captured graph.  (Behind a kernel
that does let its successor come early: test_early_release_gpu.py.)"""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import mcconv, pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def setup(n, cin, k, cout, seed=3):
  g = torch.Generator(device=DEV).manual_seed(seed)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  pts = torch.rand((n, 3), generator=g, device=DEV)
  cloud = pc.PointCloud(pts, torch.zeros(n, dtype=torch.int32, device=DEV), 1)
  neigh = pc.grid_neighborhood(cloud, 0.15, cloud)
  neigh.compute_pdf(bandwidth=0.2)
  pdf = neigh.pdf_by_neighbor_id()
  args = dict(ids=neigh._original_neigh_ids, ranges=neigh._samples_neigh_ranges, pdf=pdf, pts=pts)
  op = mcconv.ProjectionGemm(k, cin, cout, n, DEV, n_in=n)
  return args, op, r(n, cin), 0.3 * r(3, k), 0.1 * r(k), r(cin * k, cout), r(n, cout)


def step(a, op, feat, w1, b1, wf, up):
  packed = mcconv.pack_points_density(a["pts"], a["pdf"])
  basis = mcconv.kernel_basis(packed, a["pts"], a["ids"], None, w1, b1, 0.15, pdf_by_neighbor=2)
  out = op.forward(basis, feat, a["ids"], a["ranges"], wf)
  dbasis, dfeat, dw = op.backward(basis, feat, a["ids"], a["ranges"], wf, up)
  dw1, db1 = mcconv.kernel_basis_grads(packed, a["pts"], a["ids"], None, w1, b1, 0.15, dbasis,
                                       pdf_by_neighbor=2)
  return [out, dbasis, dfeat, dw, dw1, db1]


def same(xs, ys):
  # sums by atomics differ in their order from run to run: a few float32 roundings of at most
  # 1e5 terms, 1e5^0.5 * 6e-8
  for x, y in zip(xs, ys):
    assert (x - y).norm() <= 2e-5 * y.norm()


# a SIMT layer, an MMA layer, one of several waves
@pytest.mark.parametrize("n,cin,k,cout", [(700, 8, 16, 16), (3000, 48, 32, 64),
                                          (20000, 64, 16, 128)])
def test_behind_a_slow_producer_and_from_a_graph(n, cin, k, cout):
  a, op, feat, w1, b1, wf, up = setup(n, cin, k, cout)
  want = step(a, op, feat, w1, b1, wf, up)
  torch.cuda.synchronize()
  # the inputs are still being written when the chain is enqueued
  big = torch.ones((4096, 4096), device=DEV)
  late = [torch.full_like(t, float("nan")) for t in (feat, wf, up)]
  for _ in range(3):
    for t, v in zip(late, (feat, wf, up)):
      t.fill_(float("nan"))
      for _ in range(3):
        big = big @ big
        big /= big.norm()
      t.copy_(v + 0.0 * big[0, 0])
    same(step(a, op, late[0], w1, b1, late[1], late[2]), want)
  # captured, replayed on other values
  s = torch.cuda.Stream()
  s.wait_stream(torch.cuda.current_stream())
  x = feat.clone()
  with torch.cuda.stream(s):
    step(a, op, x, w1, b1, wf, up)
  torch.cuda.current_stream().wait_stream(s)
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.graph(graph):
    got = step(a, op, x, w1, b1, wf, up)
  for scale in (2.0, -0.5):
    x.copy_(feat * scale)
    graph.replay()
    same(got, step(a, op, feat * scale, w1, b1, wf, up))
