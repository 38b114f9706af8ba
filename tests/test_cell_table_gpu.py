"""Grids, searches, densities and sampling on the cell table, and layers of several
kernel MLPs, at the sizes where their kernels change form: whole numbers bit for bit
against the CPU oracle, float results within 1e-4 of the value or the result's rms."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import pylib_ref as pr
from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import _lib, mcconv, pc

pytestmark = pytest.mark.gpu
F32 = np.float32
DEV = "cuda"


def t(a):
  return torch.as_tensor(np.ascontiguousarray(a)).to(DEV)


def close(x, y, rel=1e-4):
  x = np.asarray(x, np.float64); y = np.asarray(y, np.float64)
  scale = np.maximum(np.abs(y), np.sqrt(np.mean(y * y)))
  assert (np.abs(x - y) <= rel * scale + 1e-30).all()


def same(a, b):
  assert np.array_equal(a.cpu().numpy(), b)


def clouds(seed, sizes, d, shuffled=True):
  rng = np.random.default_rng(seed)
  bid = np.repeat(np.arange(len(sizes)), sizes).astype(np.int32)
  if shuffled:
    rng.shuffle(bid)
  return rng.uniform(-1, 1, (len(bid), d)).astype(F32), bid, len(sizes)


# one cluster of 1, 2, .. 16 blocks, with the sorted copies in it (to 8192 points) and
# without (to 65536), and the separate kernels: above that, with more than 1024 box edges
# or a table of more than 2^21 cells
@pytest.mark.parametrize("sizes,d,cell", [
    ([1], 3, 0.5), ([31], 2, 0.01), ([1024], 3, 0.2), ([1000, 0, 25], 3, 0.1),
    ([2049, 6143], 3, 0.3), ([8193], 4, 0.4), ([20000, 1, 12000], 3, 0.07), ([65536], 3, 0.1),
    ([65537], 3, 0.1), ([7] * 341, 3, 0.9), ([7] * 342, 3, 0.9), ([300] * 40, 4, 0.6),
    ([900] * 10, 4, 0.6)])
@pytest.mark.parametrize("shuffled", [True, False])
def test_grid(sizes, d, cell, shuffled):
  pts, bid, b = clouds(11, sizes, d, shuffled)
  ref = pr.Grid(pts, bid, b, cell)
  g = pc.Grid(pc.PointCloud(t(pts), t(bid), b), cell)
  assert g._cells is not None
  same(g._num_cells, ref.num_cells)
  same(g._aabb_min, ref.aabb_min)
  same(g._aabb_max, ref.aabb_max)
  same(g._scaled_aabb_min, ref.scaled_aabb_min)
  same(g._cur_keys, ref.keys)
  same(g._sorted_indices, ref.sorted_indices)
  same(g._sorted_keys, ref.sorted_keys)
  same(g._sorted_points, ref.sorted_points)
  same(g._sorted_batch_ids, ref.sorted_batch_ids)
  same(g.get_DS(), ref.get_ds())


def test_grid_arrays_share_one_allocation():
  """Arrays of a grid outlive it, and are views of storage the allocator knows."""
  pts, bid, b = clouds(12, [500, 700], 3)
  g = pc.Grid(pc.PointCloud(t(pts), t(bid), b), 0.2)
  order, keys = g._sorted_indices, g._sorted_keys
  assert order.untyped_storage().data_ptr() == keys.untyped_storage().data_ptr()
  ref = pr.Grid(pts, bid, b, 0.2)
  order.record_stream(torch.cuda.Stream())
  del g
  torch.empty(1 << 20, device=DEV).fill_(1.0)
  same(order, ref.sorted_indices)
  same(keys, ref.sorted_keys)


# teams of blocks per cloud of equal, uneven and no points; more clouds than teams; every
# dimension; cells far wider than the radius, which hold more samples than a warp keeps
@pytest.mark.parametrize("sizes,d,cell,radius", [
    ([1], 3, 0.5, 0.5), ([3000], 2, 0.05, 0.05), ([5000, 17, 0, 900], 3, 0.12, 0.12),
    ([40] * 130, 3, 0.4, 0.4), ([9] * 600, 3, 0.5, 0.5), ([1500, 700], 4, 0.5, 0.5),
    ([900, 300], 5, 0.8, 0.8), ([500, 300], 6, 1.0, 1.0), ([4000, 100], 3, 0.9, 0.15),
    ([3000], 2, 0.7, 0.06)])
@pytest.mark.parametrize("mode", [0, 1])
def test_sampling(sizes, d, cell, radius, mode):
  pts, bid, b = clouds(13, sizes, d)
  nb_ref = pr.Neighborhood(pr.Grid(pts, bid, b, cell), radius)
  rp, rb, ri = pr.sample(nb_ref, mode)
  nb = pc.Neighborhood(pc.Grid(pc.PointCloud(t(pts), t(bid), b), cell), radius)
  cloud, idx = pc.sample(nb, 'poisson' if mode == 0 else 'average')
  same(cloud._batch_ids, rb)
  if mode == 0:
    same(idx, ri)
    same(cloud._points, rp)
  else:
    close(cloud._points.cpu().numpy(), rp)


# lists shorter and longer than a round of candidates, samples in and outside the boxes
@pytest.mark.parametrize("sizes,d,radius,limit", [
    ([2000, 1], 2, 0.3, 0), ([1500, 800], 3, 0.9, 0), ([1500, 800], 3, 0.2, 5),
    ([33, 2000], 4, 0.6, 0), ([800], 6, 1.2, 0)])
@pytest.mark.parametrize("mode", [0, 1])
def test_search_and_density(sizes, d, radius, limit, mode):
  pts, bid, b = clouds(14, sizes, d)
  smp, sbid, _ = clouds(15, [257] * b, d)
  smp = (1.5 * smp).astype(F32)
  g_ref = pr.Grid(pts, bid, b, radius)
  cloud = pc.PointCloud(t(pts), t(bid), b)
  for own in (True, False):
    s, sb = (pts, bid) if own else (smp, sbid)
    ref = pr.Neighborhood(g_ref, radius, s, sb, limit)
    nb = pc.grid_neighborhood(cloud, radius, cloud if own else pc.PointCloud(t(smp), t(sbid), b),
                              limit)
    same(nb._samples_neigh_ranges, ref.ranges)
    same(nb._neighbors, ref.neighbors)
    same(nb._original_neigh_ids, ref.original_neigh_ids)
    close(nb.get_pdf(bandwidth=0.3, mode=mode).cpu().numpy(), ref.get_pdf(0.3, mode))


# blocks of the weight product, channel passes side by side, few samples with long lists,
# one pair more or less than a block of the gradient kernel
@pytest.mark.parametrize("n_smp,cin,g,h,cout,radius,act", [
    (1, 16, 2, 8, 16, 3.0, 'elu'), (33, 48, 4, 8, 32, 0.9, 'leaky_relu'),
    (257, 64, 4, 16, 128, 0.4, 'elu'), (1200, 128, 1, 32, 40, 0.25, 'relu'),
    (1200, 3, 2, 8, 16, 0.3, 'leaky_relu')])
def test_layer_of_several_mlps(n_smp, cin, g, h, cout, radius, act):
  pts, bid, b = clouds(16, [900, 400], 3)
  smp, sbid, _ = clouds(17, [n_smp - n_smp // 2, n_smp // 2], 3)
  rng = np.random.default_rng(18)
  feat = rng.normal(size=(len(pts), cin)).astype(F32)
  ws = [rng.normal(size=(g, 3, h)).astype(F32)]
  bs = [(rng.normal(size=(g, 1, h)) * 0.1).astype(F32)]
  wf = (rng.normal(size=(g, cin * h, cout // g)) * 0.05).astype(F32)
  d_out = rng.normal(size=(n_smp, cout)).astype(F32)
  nb_ref = pr.Neighborhood(pr.Grid(pts, bid, b, radius), radius, smp, sbid)
  pdf = nb_ref.get_pdf(bandwidth=0.2, mode=0)
  ref_out = pr.mcconv_layer(pts, smp, feat, nb_ref, pdf, ws, bs, wf, radius, act)
  ref = pr.mcconv_layer_grads(pts, smp, feat, nb_ref, pdf, ws, bs, wf, radius, d_out, act)
  layer = mcconv.MCConv(t(ws[0]), t(bs[0]), t(wf), cin, non_linearity_type=act)
  out = layer.forward(t(feat), pc.PointCloud(t(pts), t(bid), b),
                      pc.PointCloud(t(smp), t(sbid), b), radius)
  dfeat, dw1, db1, dwf = layer.backward(t(d_out))
  layer._op.check_status()
  close(out.cpu().numpy(), ref_out)
  close(dfeat.cpu().numpy(), ref["d_features"])
  close(dwf.cpu().numpy(), ref["d_wf"])
  close(dw1.cpu().numpy(), ref["d_weights"][0])
  close(db1.cpu().numpy(), ref["d_biases"][0])


@pytest.mark.parametrize("m", [1, 255, 257, 75777])
@pytest.mark.parametrize("d,k", [(2, 8), (3, 16), (3, 64), (5, 32)])
def test_kernel_basis_grads(m, d, k):
  """Around one pair per thread, and the wave of blocks that loads ahead."""
  rng = np.random.default_rng(m + k)
  p_in = rng.uniform(0, 1, (50, d)).astype(F32)
  p_out = rng.uniform(0, 1, (20, d)).astype(F32)
  nb = np.stack([rng.integers(0, 50, m), rng.integers(0, 20, m)], 1).astype(np.int32)
  pdf = rng.uniform(0.5, 2, m).astype(F32)
  w, bias = rng.normal(size=(d, k)).astype(F32), rng.normal(size=k).astype(F32)
  grads = rng.normal(size=(m, k)).astype(F32)
  dw, db = mcconv.kernel_basis_grads(t(p_in), t(p_out), t(nb), t(pdf), t(w), t(bias), 0.5,
                                     t(grads))
  diff = (p_in[nb[:, 0]].astype(np.float64) - p_out[nb[:, 1]]) / 0.5
  pre = diff @ w + bias
  dpre = grads / pdf[:, None].astype(np.float64) * np.where(pre > 0, 1.0, 0.2)
  # (a pair whose pre-activation rounds to the other side of 0 changes one term of the
  # sum by 0.8 of it: of m * k terms of random sign about 1e-7 do)
  close(dw.cpu().numpy(), diff.T @ dpre, 2e-4)
  close(db.cpu().numpy(), dpre.sum(0), 2e-4)


# runs of points that end at, before and after a change of cloud, and an empty cloud
@pytest.mark.parametrize("n,c", [(1, 4), (16, 8), (17, 3), (4001, 12), (70000, 1)])
@pytest.mark.parametrize("mode", ['max', 'avg'])
def test_global_pool(n, c, mode):
  rng = np.random.default_rng(n + c)
  ids = np.sort(rng.integers(0, 9, n)).astype(np.int32)
  feat = rng.normal(size=(n, c)).astype(F32)
  cloud = pc.PointCloud(t(np.zeros((n, 3), F32)), t(ids), 10)
  out = mcconv.global_pool(t(feat), cloud, mode).cpu().numpy()
  ref = pr.global_pool(feat, ids, 10, mode)
  if mode == 'max':
    assert np.array_equal(out, ref)
  else:
    close(out, ref)


# the density's error against 64 bits: no larger than that of the walk over the list,
# which takes one expf per dimension
@pytest.mark.parametrize("d,n,radius,bandwidth,mode", [
    (3, 16384, 0.15, 0.2, 0), (4, 16384, 0.28, 0.2, 0), (3, 16384, 0.15, 0.1, 0),
    (2, 4096, 0.1, 0.2, 0), (3, 2048, 0.3, 0.2, 1)])
def test_density_error(d, n, radius, bandwidth, mode):
  pts, bid, b = clouds(61, [n] * 4, d, False)
  g = pc.Grid(pc.PointCloud(t(pts), t(bid), b), radius)
  nb = pc.Neighborhood(g, radius)
  inv_bw = pc._to_dims(bandwidth, d, nb._radii.device, inverse=True)
  nb.compute_pdf(bandwidth=bandwidth, mode=mode)
  by_list = ops.compute_pdf_with_pt_grads(g._sorted_points, nb._neighbors,
                                          nb._samples_neigh_ranges, inv_bw, nb._inv_radii, mode)
  bw = inv_bw.double() if mode == 0 else torch.full_like(inv_bw, np.sqrt(F32(b * n))).double()
  p = g._sorted_points.double()
  i, j = nb._neighbors[:, 0].long(), nb._neighbors[:, 1].long()
  u = (p[i] - p[j]) * nb._inv_radii.double() * bw
  terms = torch.exp(-0.5 * (u * u).sum(1)) * (bw / np.sqrt(2 * np.pi)).prod()
  exact = torch.zeros(b * n, dtype=torch.float64, device=DEV).index_add_(0, j, terms)
  error = lambda x: float((x.double() - exact).norm() / exact.norm())
  assert error(nb.point_pdf()) <= 1.01 * error(by_list)


# a wait of the sampling that runs out is reported if any block left its samples
# unwritten, whichever block was late and at whichever barrier; a block that is late
# because it works (shows progress) is waited for
@pytest.mark.parametrize("late_block,late_at,working", [
    (-1, 0, 0), (0, 0, 0), (0, 1, 0), (0, 2, 0), (0, 3, 0), (7, 0, 0), (7, 3, 0), (15, 2, 0),
    (0, 1, 1), (9, 0, 1), (3, 3, 1)])
def test_sampling_barrier_reports(late_block, late_at, working):
  ws = torch.empty(256, dtype=torch.uint8, device=DEV)
  reported, gave_up = _lib.c_int(-1), _lib.c_int(-1)
  _lib.check(_lib.lib().tfgpc_debug_sampling_barrier(
      None, _lib.ptr(ws), _lib.c_sz(256), _lib.c_int(20000), _lib.c_int(late_block),
      _lib.c_int(late_at), _lib.c_int(working), ctypes.byref(reported), ctypes.byref(gave_up)))
  assert (gave_up.value > 0) == (late_block >= 0 and not working)
  assert reported.value == (1 if gave_up.value else 0)


# a cell much wider than the radius, with many of its points taken, is sampled from the
# neighbor list: from the grid one block marks around all of them
@pytest.mark.parametrize("cell,radius,by_list", [(0.5, 0.03, True), (0.13, 0.04, True),
                                                 (0.12, 0.04, False), (0.04, 0.04, False)])
def test_sampling_of_wide_cells(cell, radius, by_list, monkeypatch):
  pts, bid, b = clouds(71, [20000], 3)
  calls = []
  real = ops.sampling
  monkeypatch.setattr(ops, "sampling", lambda *a, **k: calls.append(1) or real(*a, **k))
  nb = pc.Neighborhood(pc.Grid(pc.PointCloud(t(pts), t(bid), b), cell), radius)
  cloud, idx = pc.sample(nb)
  assert bool(calls) == by_list
  rp, rb, ri = pr.sample(pr.Neighborhood(pr.Grid(pts, bid, b, cell), radius), 0)
  same(idx, ri)
  same(cloud._points, rp)


class CellGridArrays(ctypes.Structure):
  """tfgpc_cell_grid with arrays of its own, filled with -7."""
  _fields_ = [("D", ctypes.c_int), ("max_cells", ctypes.c_int), ("n", ctypes.c_int64),
              ("batch_size", ctypes.c_int64)] + [(name, ctypes.c_void_p) for name in (
                  "aabb_min", "aabb_max", "num_cells", "scaled_aabb_min", "inv_cell_sizes", "keys",
                  "sorted_indices", "sorted_keys", "sorted_points", "sorted_batch_ids", "packed",
                  "cell_start", "ds")]

  def __init__(self, d, max_cells, n, b):
    table = _lib.lib().tfgpc_cell_table_elems(d, _lib.c_i64(b), max_cells)
    f, i, l = torch.float32, torch.int32, torch.int64
    self.arrays = dict(
        aabb_min=(b * d, f), aabb_max=(b * d, f), num_cells=(d, i), scaled_aabb_min=(b * d, f),
        inv_cell_sizes=(d, f), keys=(n, l), sorted_indices=(n, i), sorted_keys=(n, l),
        sorted_points=(n * d, f), sorted_batch_ids=(n, i), packed=(4 * n, f), cell_start=(table, i),
        ds=(2 * b * max_cells ** 2, i))
    self.arrays = {k: torch.full((s,), -7, dtype=ty, device=DEV)
                   for k, (s, ty) in self.arrays.items()}
    super().__init__(d, max_cells, n, b, *[v.data_ptr() for v in self.arrays.values()])


# a grid that asks for more cells than its arrays were sized for is not sorted, searched
# or sampled: in one cluster (with and without the sorted copies), and in separate kernels
@pytest.mark.parametrize("n", [3000, 20000, 70000])
@pytest.mark.parametrize("sample", [True, False])
def test_too_few_cells(n, sample):
  lib, d, b, max_cells = _lib.lib(), 3, 1, 8
  pts, bid, _ = clouds(81, [n], d)
  pts, bid = t(pts), t(bid)
  g = CellGridArrays(d, max_cells, n, b)
  sizes = (ctypes.c_float * d)(0.1, 0.5, 0.5)
  asked, total = (ctypes.c_int32 * d)(), _lib.c_i64(-1)
  inv = torch.full((d,), 10.0, device=DEV)
  out = [torch.full((s,), -7, dtype=ty, device=DEV)
         for s, ty in ((3 * n, torch.float32), (n, torch.int32), (n, torch.int32))]
  lib.tfgpc_cell_grid_workspace_bytes.restype = ctypes.c_size_t
  need = lib.tfgpc_cell_grid_workspace_bytes(d, _lib.c_i64(n), _lib.c_i64(n), _lib.c_i64(b), max_cells)
  need_s = lib.tfgpc_cells_sample_workspace_bytes(_lib.c_i64(n))
  ws, ws_s = (torch.empty(k, dtype=torch.uint8, device=DEV) for k in (need, need_s))
  stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  head = (stream, ctypes.byref(g), _lib.ptr(pts), _lib.ptr(bid), sizes, None)
  if sample:
    rc = lib.tfgpc_cell_grid_sample(*head, 0, _lib.ptr(inv), *[_lib.ptr(o) for o in out],
                                    _lib.ptr(ws), _lib.c_sz(need), _lib.ptr(ws_s),
                                    _lib.c_sz(need_s), asked, ctypes.byref(total))
  else:
    rc = lib.tfgpc_cell_grid_neighborhood(*head, _lib.ptr(inv), _lib.c_i64(n), None, None, 2, 0,
                                          _lib.ptr(out[1]), _lib.ptr(ws), _lib.c_sz(need), asked,
                                          ctypes.byref(total))
  assert rc == 3
  ext = (pts.max(0).values - pts.min(0).values).cpu().numpy()
  assert list(asked) == [int(c) for c in np.ceil(ext / np.array([0.1, 0.5, 0.5], F32))]
  for x in [g.arrays[k] for k in ("keys", "sorted_indices", "sorted_points", "packed")] + out[::2]:
    assert bool((x == -7).all())


def test_a_fine_grid_leaves_later_grids_as_they_are():
  """Whether a grid gets a table, and of what size, does not depend on the grids of the
  same batch size before it."""
  pts, bid, b = clouds(91, [300] * 16, 3)
  cloud = pc.PointCloud(t(pts), t(bid), b)
  def size_of(cell):
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    grid = pc.Grid(cloud, cell)
    grown = torch.cuda.memory_allocated() - before
    return grid._cells is not None, grown
  pc.Grid(cloud, 0.25)
  pc.Grid(cloud, 0.25)
  alone = size_of(0.25)
  assert alone[0]
  # 40 cells: a larger table; [100, 1, 1]: 16 x 128^3 cells have none; 0.0015: over 1024 cells
  for cell in (0.05, [0.02, 3.0, 3.0], 0.0015):
    fine = pc.Grid(cloud, cell)
    assert (fine._cells is not None) == (cell == 0.05)
    ref = pr.Grid(pts, bid, b, cell)
    same(fine._sorted_keys, ref.sorted_keys)
    same(fine._sorted_indices, ref.sorted_indices)
    assert size_of(0.25) == alone


def test_an_outlier_costs_the_table_for_a_while_only():
  pts, bid, b = clouds(92, [500] * 3, 3)
  far = pts.copy()
  far[7] = 1000.0
  cloud, outlier = (pc.PointCloud(t(p), t(bid), b) for p in (pts, far))
  assert pc.Grid(cloud, 0.21)._cells is not None
  nb = pc.grid_neighborhood(outlier, 0.21)
  assert nb._grid._cells is None
  ref = pr.Neighborhood(pr.Grid(far, bid, b, 0.21), 0.21)
  same(nb._samples_neigh_ranges, ref.ranges)
  same(nb._neighbors, ref.neighbors)
  assert any(pc.Grid(cloud, 0.21)._cells is not None for _ in range(20))
  assert pc.Grid(cloud, 0.21)._cells is not None


# cells of more points than a tile of the sort (512 slots, 1024 in the cluster), around the
# line where the block ranks them together, at tile edges, several side by side, with and
# without points that belong to no cell
@pytest.mark.parametrize("cells", [
    [1024], [1025], [8192], [1, 1025, 3], [511, 1500, 1500, 2], [1026] * 7, [40000], [3000, 60000],
    [70001], [1025, 1, 90000, 700], [100000, 100000]])
@pytest.mark.parametrize("strays", [0, 1500])
def test_crowded_cells(cells, strays):
  rng = np.random.default_rng(101)
  pts = np.concatenate([np.full((m, 3), k) for k, m in enumerate(cells)]).astype(F32)
  pts += rng.uniform(0.1, 0.9, pts.shape).astype(F32)
  bid = np.zeros(len(pts), np.int32)
  if strays:
    pts = np.concatenate([pts, rng.uniform(0, 1, (2 * strays, 3)).astype(F32)])
    bid = np.concatenate([bid, np.repeat(np.array([-1, 2], np.int32), strays)])
  order = rng.permutation(len(pts))
  pts, bid = pts[order], bid[order]
  g = pc.Grid(pc.PointCloud(t(pts), t(bid), 1), 1.0)
  assert g._cells is not None
  keys = g._cur_keys.cpu().numpy()
  assert len(np.unique(keys)) >= len(cells)
  perm = np.argsort(-keys, kind="stable")
  same(g._sorted_indices, perm.astype(np.int32))
  same(g._sorted_keys, keys[perm])
  same(g._sorted_points, pts[perm])
  same(g._sorted_batch_ids, bid[perm])


@pytest.mark.parametrize("n", [8192 * 4096, 8192 * 4096 + 1, 9000 * 4096 + 77])
def test_ranges_of_millions_of_samples(n):
  """Scans above and below the line where the sums of their tiles are scanned by themselves."""
  pts, bid, b = clouds(111, [100], 3)
  grid = pc.Grid(pc.PointCloud(t(pts), t(bid), b), 0.6)
  at = torch.cat([torch.arange(0, n, 1_000_003), torch.tensor([n - 1])]).to(DEV)
  samples = torch.zeros(n, 3, device=DEV)
  samples[at] = t(pts)[torch.arange(len(at), device=DEV) % 100]
  ids = torch.full((n,), -1, device=DEV, dtype=torch.int32)
  ids[at] = 0
  few = pc.Neighborhood(grid, 0.6, pc.PointCloud(samples[at].contiguous(), ids[at], b))
  counts = torch.zeros(n, device=DEV, dtype=torch.int64)
  counts[at] = few._samples_neigh_ranges.long().diff(prepend=torch.zeros(1, device=DEV).long())
  many = pc.Neighborhood(grid, 0.6, pc.PointCloud(samples, ids, b))
  assert torch.equal(many._samples_neigh_ranges.long(), counts.cumsum(0))
