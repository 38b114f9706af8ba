"""Grids built by one cluster at the edges of what a thread and a warp of it hold: one to four
points per thread, tables of one to several pieces of 128 cells per warp, tables that do not
begin at a multiple of 16 bytes.  All arrays bit for bit against the CPU oracle, and nothing
written beside the table."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import pylib_ref as pr
from tensorflow_graphics_point_clouds_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
NAMES = ("aabb_min", "aabb_max", "num_cells", "scaled_aabb_min", "inv_cell_sizes", "keys",
         "sorted_indices", "sorted_keys", "sorted_points", "sorted_batch_ids", "packed",
         "cell_start", "ds")


class CellGrid(ctypes.Structure):
  _fields_ = [("D", ctypes.c_int), ("max_cells", ctypes.c_int), ("n", ctypes.c_int64),
              ("batch_size", ctypes.c_int64)] + [(name, ctypes.c_void_p) for name in NAMES]


# sizes, dimensions, cell, cells per dimension at most, place of the table, form of the points
@pytest.mark.parametrize("sizes,d,cell,most,shift,form", [
    ([1], 3, 0.5, 8, 0, "apart"), ([33], 3, 0.3, 8, 1, "apart"),
    ([16384], 3, 0.1, 32, 0, "apart"), ([16385], 3, 0.1, 32, 3, "apart"),
    ([9000, 0, 23769], 3, 0.1, 24, 0, "apart"), ([32768, 1], 2, 0.01, 256, 2, "mixed"),
    ([12288] * 4, 3, 0.06, 36, 0, "apart"), ([7001] * 7, 3, 0.0669, 32, 0, "mixed"),
    ([49153], 3, 0.0313, 64, 0, "apart"), ([65535], 3, 0.0157, 128, 1, "apart"),
    ([65536], 2, 0.00144, 1440, 0, "mixed"), ([30000, 30000], 3, 0.4, 6, 0, "crowded"),
    ([40000], 3, 0.2, 12, 0, "strange"),
    # a warp of two clouds whose last 32 points are fewer than a box has corners' coordinates
    ([32768, 1], 3, 0.1, 32, 0, "apart"), ([20000, 3], 3, 0.1, 32, 0, "apart"),
    ([20511, 2], 2, 0.02, 128, 0, "apart"), ([16992, 7], 6, 0.4, 8, 0, "apart"),
    ([16600, 16201], 3, 0.1, 32, 0, "last")])
def test_grid_of_one_cluster(sizes, d, cell, most, shift, form):
  rng = np.random.default_rng(5)
  n, b = sum(sizes), len(sizes)
  bid = np.repeat(np.arange(b), sizes).astype(np.int32)
  pts = rng.uniform(-1, 1, (n, d)).astype(np.float32)
  if form in ("mixed", "last"):
    rng.shuffle(bid)
  if form == "last":               # the corner of its cloud
    pts[-1] = 1.0625
  if form == "crowded":            # a cell of thousands, in runs and single points
    pts[5000:29000] = 0.5 + 0.01 * pts[5000:29000]
    pts[30000::3] = -0.5
  if form == "strange":            # zeros of both signs, and ids outside the batch
    pts[::7] = 0.0
    pts[1::7] = -0.0
    bid[100:20000:31] = 1
    bid[101:20000:37] = -1
  lib = _lib.lib()
  table = lib.tfgpc_cell_table_elems(d, _lib.c_i64(b), most)
  f, i, l = torch.float32, torch.int32, torch.int64
  shapes = dict(aabb_min=(b * d, f), aabb_max=(b * d, f), num_cells=(d, i),
                scaled_aabb_min=(b * d, f), inv_cell_sizes=(d, f), keys=(n, l),
                sorted_indices=(n, i), sorted_keys=(n, l), sorted_points=(n * d, f),
                sorted_batch_ids=(n, i), packed=(4 * n, f), cell_start=(table + 16, i),
                ds=(2 * b * most ** 2, i))
  arrays = {k: torch.full((s,), -7, dtype=ty, device=DEV) for k, (s, ty) in shapes.items()}
  at = {k: v.data_ptr() for k, v in arrays.items()}
  at["cell_start"] += 4 * (8 + shift)
  g = CellGrid(d, most, n, b, *[at[k] for k in NAMES])
  lib.tfgpc_cell_grid_workspace_bytes.restype = ctypes.c_size_t
  need = lib.tfgpc_cell_grid_workspace_bytes(d, _lib.c_i64(n), _lib.c_i64(0), _lib.c_i64(b), most)
  ws = torch.empty(need, dtype=torch.uint8, device=DEV)
  points, ids = torch.as_tensor(pts).to(DEV), torch.as_tensor(bid).to(DEV)
  cells, total = (ctypes.c_int32 * d)(), _lib.c_i64(-1)
  rc = lib.tfgpc_cell_grid_neighborhood(
      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(g),
      _lib.ptr(points), _lib.ptr(ids), (ctypes.c_float * d)(*[cell] * d), None, None,
      _lib.c_i64(0), None, None, 0, 0, None, _lib.ptr(ws), _lib.c_sz(need), cells,
      ctypes.byref(total))
  assert rc == 0
  got = {k: v.cpu().numpy() for k, v in arrays.items()}
  inside = (bid >= 0) & (bid < b)
  lo = np.stack([pts[bid == c].min(0) if (bid == c).any() else np.full(d, np.inf, np.float32)
                 for c in range(b)]) - np.float32(1e-9)
  hi = np.stack([pts[bid == c].max(0) if (bid == c).any() else np.full(d, -np.inf, np.float32)
                 for c in range(b)]) + np.float32(1e-9)
  assert np.array_equal(got["aabb_min"].reshape(b, d), lo)
  assert np.array_equal(got["aabb_max"].reshape(b, d), hi)
  if inside.all():
    ref = pr.Grid(pts, bid, b, cell)
    assert np.array_equal(got["num_cells"], ref.num_cells)
    assert np.array_equal(got["keys"], ref.keys)
  nc = got["num_cells"]
  assert list(cells) == list(nc) and (nc <= most).all()
  keys, count = got["keys"], b * int(np.prod(nc.astype(np.int64)))
  # (the keys of ids outside the batch are sorted by side only)
  bucket = np.where(keys >= count, 0, np.where(keys < 0, count + 1, count - keys))
  order = np.argsort(bucket, kind="stable")
  assert np.array_equal(got["sorted_indices"], order)
  assert np.array_equal(got["sorted_keys"], keys[order])
  assert np.array_equal(got["sorted_points"].reshape(n, d), pts[order])
  assert np.array_equal(got["sorted_batch_ids"], bid[order])
  start = np.concatenate([[0], np.cumsum(np.bincount(bucket, minlength=count + 2))])
  have = got["cell_start"]
  assert np.array_equal(have[8 + shift:8 + shift + count + 3], start)
  assert (have[:8 + shift] == -7).all() and (have[8 + shift + table:] == -7).all()
  if d <= 3:
    packed = got["packed"].reshape(n, 4)
    assert np.array_equal(packed[:, :d], pts[order])
    assert np.array_equal(packed[:, 3].view(np.int32), order)
