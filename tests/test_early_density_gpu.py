"""Densities enqueued before the host reads the number of pairs: the same as those of
compute_pdf, for the forms a layer's neighborhood takes."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import mcconv, pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def cloud(n, b, d, g):
  ids = torch.sort(torch.randint(0, b, (n,), generator=g, device=DEV)).values.int()
  return pc.PointCloud(torch.rand((n, d), generator=g, device=DEV), ids, b)


# the last: a grid too fine for a cell table, whose densities come later
@pytest.mark.parametrize("n,b,d,radius", [(1, 1, 3, 0.1), (700, 3, 3, 0.2), (20011, 2, 3, 0.08),
                                          (90001, 4, 3, 0.05), (900, 2, 2, 0.1),
                                          (900, 2, 4, 0.3), (2000, 1, 3, 0.0005)])
@pytest.mark.parametrize("mode", [0, 1])
def test_same_as_compute_pdf(n, b, d, radius, mode):
  g = torch.Generator(device=DEV).manual_seed(n)
  a = cloud(n, b, d, g)
  out = pc.PointCloud(a._points[::2].contiguous(), a._batch_ids[::2].contiguous(), b)
  for samples in (a, out, None):
    early = pc.grid_neighborhood_with_pdf(a, radius, samples, bandwidth=0.3, mode=mode)
    late = pc.grid_neighborhood(a, radius, samples)
    late.compute_pdf(bandwidth=0.3, mode=mode)
    assert torch.equal(early.get_pdf(bandwidth=0.3, mode=mode), late.get_pdf())
    assert torch.equal(early.point_pdf(), late.point_pdf())
    assert torch.equal(early._neighbors, late._neighbors)
    if early._packed is not None:
      assert d == 3 and torch.equal(early._packed,
                                    mcconv.pack_points_density(a._points, early._sample_pdf))
    # asked for again with another bandwidth
    early.compute_pdf(bandwidth=0.1, mode=mode)
    late.compute_pdf(bandwidth=0.1, mode=mode)
    assert early._packed is None and torch.equal(early.get_pdf(), late.get_pdf())


def test_layers_take_overridden_neighborhoods():
  g = torch.Generator(device=DEV).manual_seed(1)
  a = cloud(500, 2, 3, g)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  args = (r(1, 3, 16), r(1, 1, 16), r(1, 64, 32), 4)
  feat = r(500, 4)
  seen = []

  class Layer(mcconv.MCConv):
    def build_neighborhood(self, *b):
      seen.append(b)
      return super().build_neighborhood(*b)

  out = Layer(*args).forward(feat, a, a, 0.2)
  assert len(seen) == 1 and torch.equal(out, mcconv.MCConv(*args).forward(feat, a, a, 0.2))


def test_density_transform_by_neighbor():
  g = torch.Generator(device=DEV).manual_seed(2)
  a = cloud(3000, 2, 3, g)
  neigh = pc.grid_neighborhood_with_pdf(a, 0.1, a)
  table, ids = neigh.pdf_by_neighbor_id(), neigh._original_neigh_ids
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  par = (r(1, 16), r(1, 16), r(16, 1), r(1, 1))
  ranges = neigh._samples_neigh_ranges
  assert torch.equal(mcconv.pointconv_pdf(table, ranges, *par, ids),
                     mcconv.pointconv_pdf(neigh.get_pdf(), ranges, *par))


def test_pointconv_takes_overridden_neighborhoods_and_densities():
  g = torch.Generator(device=DEV).manual_seed(5)
  a = cloud(500, 2, 3, g)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  args = (r(3, 16), r(16), r(16 * 4, 32), (r(1, 16), r(16, 1)), (r(1, 16), r(1, 1)), 4)
  feat = r(500, 4)
  seen = []

  class Layer(mcconv.PointConv):
    def _neighborhood(self, *b):
      seen.append(b)
      return super()._neighborhood(*b)

  want = mcconv.PointConv(*args).forward(feat, a, a, 0.2)
  assert torch.equal(Layer(*args).forward(feat, a, a, 0.2), want) and len(seen) == 1

  class Other(pc.Neighborhood):
    def get_pdf(self, **kw):
      seen.append(kw)
      return super().get_pdf(**kw)

  neigh = Other(pc.Grid(a, 0.2), 0.2, a)
  out = mcconv.PointConv(*args).forward(feat, a, a, 0.2, neighborhood=neigh)
  assert torch.equal(out, want) and len(seen) == 2


def test_a_neighborhood_given_by_the_caller_brings_no_points():
  """Its pairs and densities count; the kernel inputs are the points of the clouds given."""
  g = torch.Generator(device=DEV).manual_seed(6)
  a = cloud(400, 2, 3, g)
  moved = pc.PointCloud(a._points * 1.25 + 0.5, a._batch_ids, 2)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  args, feat = (r(1, 3, 16), r(1, 1, 16), r(1, 64, 32), 4), r(400, 4)
  outs = []
  for build in (pc.grid_neighborhood_with_pdf, pc.grid_neighborhood):
    layer = mcconv.MCConv(*args)
    outs.append(layer.forward(feat, moved, moved, 0.2, neighborhood=build(a, 0.2, a)))
  assert torch.equal(*outs)
