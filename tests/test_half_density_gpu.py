"""Densities by half the distance tests (tfgpc_cells_density_ws with a workspace) against those
by all of them and a sum in 64 bits: cells of one to several pieces of a warp, crowded ones, points
outside the batch, a point that is no number, every order of the results."""
import ctypes

import pytest
import torch
from test_cell_table_gpu import CellGridArrays

from tensorflow_graphics_point_clouds_b200 import _lib, pc
from tensorflow_graphics_point_clouds_b200._lib import c_i64, c_sz, ptr

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,b,d,radius", [(1, 1, 3, 0.1), (33, 2, 2, 0.3), (5003, 3, 3, 0.12),
                                          (70001, 4, 3, 0.06), (9000, 2, 4, 0.3),
                                          (900, 1, 5, 0.4), (4000, 2, 3, 0.9), (2000, 1, 6, 0.5)])
@pytest.mark.parametrize("mode", [0, 1])
def test_same_as_all_tests(n, b, d, radius, mode):
  gen = torch.Generator(device=DEV).manual_seed(n)
  points = torch.rand((n, d), generator=gen, device=DEV)
  ids = torch.sort(torch.randint(0, b, (n,), generator=gen, device=DEV)).values.int()
  if n > 100:
    ids[-3:] = b + 5                  # in no cell
    points[7, 0] = float("nan")
  lib, most = _lib.lib(), 32
  while not lib.tfgpc_cell_table_elems(d, c_i64(b), most):
    most //= 2
  g = CellGridArrays(d, most, n, b)
  need = lib.tfgpc_cell_grid_workspace_bytes(d, c_i64(n), c_i64(0), c_i64(b), most)
  ws = torch.empty(need, dtype=torch.uint8, device=DEV)
  stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  asked, total = (ctypes.c_int32 * d)(), c_i64(0)
  _lib.check(lib.tfgpc_cell_grid_neighborhood(
      stream, ctypes.byref(g), ptr(points), ptr(ids), (ctypes.c_float * d)(*[radius] * d), None,
      None, c_i64(0), None, None, 0, 0, None, ptr(ws), c_sz(need), asked, ctypes.byref(total)))
  inv_r = torch.full((d,), 1.0 / radius, device=DEV)
  bw = torch.linspace(3.0, 5.0, d, device=DEV)
  room = torch.empty(n, dtype=torch.int64, device=DEV)
  norm = (bw if mode == 0 else torch.full_like(bw, float(n)).sqrt()).double()
  for order in (1, 2):
    got = []
    for buffer, size in ((None, 0), (ptr(room), 8 * n)):
      out = torch.empty(n, device=DEV)
      _lib.check(lib.tfgpc_cells_density_ws(stream, ctypes.byref(g), ptr(inv_r), ptr(bw), mode,
                                            c_i64(n), None, None, order, buffer, c_sz(size),
                                            ptr(out)))
      got.append(out.double())
    # (each is a few roundings of its exponents and sums away)
    assert torch.allclose(got[0], got[1], rtol=1e-6, atol=0.0)
    which = torch.arange(n, device=DEV) if order == 1 else g.arrays["sorted_indices"].long()
    some = torch.randperm(n, generator=gen, device=DEV)[:200]
    at = which[some]
    diff = (points[at][:, None].double() - points[None].double()) * inv_r.double()
    near = ((diff * diff).sum(2) < 1.0) & (ids[at][:, None] == ids[None]) & (ids[at] < b)[:, None]
    terms = torch.exp(-0.5 * (diff * norm).square().sum(2)) * (norm * 0.3989422804014327).prod()
    exact = torch.where(near, terms, torch.zeros_like(terms)).sum(1)
    # (a pair within rounding of the radius may be decided either way: none in these clouds)
    assert torch.allclose(got[1][some], exact, rtol=1e-5, atol=0.0)


def test_workspace_rule():
  need = _lib.lib().tfgpc_cells_density_workspace_bytes
  assert need(3, c_i64(65535), c_i64(1 << 40)) == 0 and need(7, c_i64(1 << 20), c_i64(1 << 40)) == 0
  assert need(3, c_i64(65536), c_i64(65536 * 34)) == 0
  assert need(3, c_i64(65536), c_i64(65536 * 40)) == 65536 * 8
  assert need(4, c_i64(65536), c_i64(65536 * 16)) == 65536 * 8


def test_neighborhoods_of_many_neighbors_take_half():
  gen = torch.Generator(device=DEV).manual_seed(4)
  points = torch.rand((66000, 3), generator=gen, device=DEV)
  cloud = pc.PointCloud(points, torch.zeros(66000, dtype=torch.int32, device=DEV), 1)
  early = pc.grid_neighborhood_with_pdf(cloud, 0.08, cloud, bandwidth=0.2)     # nothing counted yet
  late = pc.grid_neighborhood(cloud, 0.08)
  late.compute_pdf(bandwidth=0.2)
  assert late._pairs_of_all_points() > 66000 * 100
  assert torch.allclose(early.point_pdf(), late.point_pdf(), rtol=1e-6, atol=0.0)


@pytest.mark.parametrize("b,half", [(700, False), (100, True)])
def test_clouds_of_few_points_take_all_tests(b, half):
  """Many neighbors are few candidates where a cloud has no more points (the workspace shows which
  way was taken)."""
  n = 80000
  gen = torch.Generator(device=DEV).manual_seed(b)
  ids = torch.sort(torch.randint(0, b, (n,), generator=gen, device=DEV)).values.int()
  neigh = pc.grid_neighborhood(pc.PointCloud(torch.rand((n, 3), generator=gen, device=DEV), ids, b), 0.57)
  assert neigh._pairs_of_all_points() > 40 * n
  torch.cuda.synchronize()
  torch.cuda.reset_peak_memory_stats()
  before = torch.cuda.memory_allocated()
  neigh.compute_pdf(bandwidth=0.2)
  assert (torch.cuda.max_memory_allocated() - before >= 12 * n) == half
