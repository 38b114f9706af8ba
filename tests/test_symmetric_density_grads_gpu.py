"""Point gradients of densities over symmetric lists, gathered, against those by atomics over the
same lists; and which neighborhoods take them."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


# lists of one pair, up to a warp's width and beyond
@pytest.mark.parametrize("n,b,d,radius", [(1, 1, 3, 0.1), (40, 2, 2, 0.5), (3001, 3, 3, 0.12),
                                          (2000, 1, 3, 0.5), (700, 2, 4, 0.4), (300, 1, 5, 0.6)])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("own", [True, False])
def test_same_as_by_atomics(n, b, d, radius, mode, own):
  g = torch.Generator(device=DEV).manual_seed(n)
  points = torch.rand((n, d), generator=g, device=DEV)
  if n > 1:
    points[1] = points[0]
  ids = torch.sort(torch.randint(0, b, (n,), generator=g, device=DEV)).values.int()
  cloud = pc.PointCloud(points, ids, b)
  nb = pc.Neighborhood(pc.Grid(cloud, radius), radius, cloud if own else None)
  grads = torch.randn(n, generator=g, device=DEV)
  bw = torch.linspace(2.0, 4.0, d, device=DEV)
  at = points if own else nb._grid._sorted_points
  lists = nb._original_neigh_ids if own else nb._neighbors
  args = (at, lists, nb._samples_neigh_ranges, bw, nb._inv_radii, grads, mode)
  ref, got = ops.compute_pdf_pt_grads(*args), ops.compute_pdf_pt_grads_symmetric(*args)
  # sums of as many float32 terms, in another order: relative to the terms, not to what is left
  scale = ref.abs().max() + 1e-30
  assert ((got - ref).abs() <= 2e-6 * scale).all()
  assert torch.equal(got, ops.compute_pdf_pt_grads_symmetric(*args))


def test_limited_lists_are_not_symmetric(monkeypatch):
  g = torch.Generator(device=DEV).manual_seed(9)
  cloud = pc.PointCloud(torch.rand((500, 3), generator=g, device=DEV),
                        torch.zeros(500, dtype=torch.int32, device=DEV), 1)
  seen, library = [], ops.compute_pdf_pt_grads_symmetric
  monkeypatch.setattr(ops, "compute_pdf_pt_grads_symmetric",
                      lambda *a: seen.append(1) or library(*a))
  grid = pc.Grid(cloud, 0.3)
  for samples, limit, taken in ((None, 0, 1), (cloud, 0, 2), (None, 5, 2)):
    nb = pc.Neighborhood(grid, 0.3, samples, limit)
    nb.pdf_point_grads(torch.rand(nb.num_pairs, generator=g, device=DEV))
    assert len(seen) == taken
  monkeypatch.setattr(ops, "compute_pdf_pt_grads", lambda *a: torch.zeros((500, 3), device=DEV))
  nb = pc.Neighborhood(grid, 0.3)
  assert not nb.pdf_point_grads(torch.rand(nb.num_pairs, device=DEV)).any() and len(seen) == 2


@pytest.mark.parametrize("own", [True, False])
@pytest.mark.parametrize("where", ["fill", "class"])
def test_lists_of_ones_own_need_not_be_symmetric(where, own, monkeypatch):
  """Lists of a replaced fill, or of a class derived from Neighborhood, are taken as they are:
  here every pair but the ones of a point with itself leads to the first point."""
  g = torch.Generator(device=DEV).manual_seed(11)
  cloud = pc.PointCloud(torch.rand((300, 3), generator=g, device=DEV),
                        torch.zeros(300, dtype=torch.int32, device=DEV), 1)

  def one_way(pairs):
    pairs = pairs.clone()
    pairs[:, 0] = torch.where(pairs[:, 0] == pairs[:, 1], pairs[:, 0], 0)
    return pairs

  library = ops.find_neighbors_fill
  if where == "fill":
    def fill(*args):
      lists = library(*args)
      return tuple(map(one_way, lists)) if isinstance(lists, tuple) else one_way(lists)
    monkeypatch.setattr(ops, "find_neighbors_fill", fill)
    nb = pc.Neighborhood(pc.Grid(cloud, 0.3), 0.3, cloud if own else None)
  else:
    class Mine(pc.Neighborhood):
      _neighbors = property(lambda self: one_way(pc.Neighborhood._neighbors.fget(self)))
      _original_neigh_ids = property(
          lambda self: one_way(pc.Neighborhood._original_neigh_ids.fget(self)))
    nb = Mine(pc.Grid(cloud, 0.3), 0.3, cloud if own else None)
  grads, grid = torch.randn(nb.num_pairs, generator=g, device=DEV), nb._grid
  lists = nb._original_neigh_ids if own else nb._neighbors
  per_point = torch.zeros(300, device=DEV).index_add_(0, lists[:, 0].long(), grads)
  ref = ops.compute_pdf_pt_grads(cloud._points if own else grid._sorted_points, lists,
                                 nb._samples_neigh_ranges, torch.full((3,), 5.0, device=DEV),
                                 nb._inv_radii, per_point, 0)
  if not own:
    ref = torch.empty_like(ref).index_copy_(0, grid._sorted_indices.long(), ref)
  # (float32 sums of up to 300 terms by atomics, in any order)
  scale = ref.abs().max()
  assert ((nb.pdf_point_grads(grads) - ref).abs() <= 300 * 6e-8 * scale).all()
