"""Levels of a hierarchy that follow one another without a blocking read, against one call per
level: bit for bit, at the edges of what a level may hold.  And neighborhoods with densities on a
grid that is there already."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import _lib, mcconv, pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def cloud(n, b, d, seed, outside=0):
  g = torch.Generator(device=DEV).manual_seed(seed)
  ids = torch.sort(torch.randint(0, b, (n,), generator=g, device=DEV)).values.int()
  if outside:
    ids[-outside:] = b + 3
  return pc.PointCloud(torch.rand((n, d), generator=g, device=DEV), ids, b)


def one_by_one(start, radii, mode):
  cur, out = start, []
  for r in radii:
    neigh, cur, idx = pc.PointHierarchy._level(cur, r, mode)
    out.append((neigh, cur, idx))
  return out


# level 1 with 1 to 8192 points (sorted copies in the cluster) and more, with more than the 65 536
# that can follow, a radius that shrinks (a table too large to follow), per dimension, many clouds
@pytest.mark.parametrize("n,b,d,radii,outside", [
    (1, 1, 3, [0.1, 0.2], 0), (3000, 3, 3, [0.05, 0.1, 0.2], 5), (60000, 2, 3, [0.02, 0.04], 0),
    (60000, 1, 2, [0.004, 0.3, 0.4], 0), (100000, 4, 3, [0.05, 0.1, 0.2, 0.4], 0),
    (90000, 1, 2, [0.002, 0.004, 0.01], 0), (5000, 2, 3, [0.2, 0.01, 0.3], 0),
    (5000, 2, 3, [[0.1, 0.2, 0.05], [0.2, 0.1, 0.1]], 0), (4000, 400, 3, [0.3, 0.6], 0),
    (5000, 2, 4, [0.2, 0.4, 0.8], 0)])
@pytest.mark.parametrize("mode", ["poisson", "average"])
def test_same_as_one_level_at_a_time(n, b, d, radii, outside, mode):
  if mode == "average" and outside:
    outside = 0
  a = cloud(n, b, d, n + d, outside)
  ref = one_by_one(a, radii, mode)
  for _ in range(2):                    # (with bounds of cells not known yet, and known)
    hier = pc.PointHierarchy(a, radii, mode)
    assert len(hier._point_clouds) == len(radii) + 1
    before = a
    for l, (neigh, points, idx) in enumerate(ref):
      got, grid = hier._point_clouds[l + 1], hier._neighborhoods[l]._grid
      assert torch.equal(got._points, points._points)
      assert torch.equal(got._batch_ids, points._batch_ids)
      assert (idx is None) == (hier._sample_indices[l] is None)
      assert idx is None or torch.equal(hier._sample_indices[l], idx)
      assert grid._point_cloud is before and got._batch_size == b and got._dimension == d
      for name in ("_sorted_points", "_sorted_indices", "_cur_keys", "_num_cells"):
        assert torch.equal(getattr(grid, name), getattr(neigh._grid, name)), name
      assert torch.equal(hier._neighborhoods[l]._neighbors, neigh._neighbors)
      before = got


@pytest.mark.parametrize("held", [32768, 0])
@pytest.mark.parametrize("n", [40000, 32768, 70000])
def test_devices_whose_clusters_hold_less(n, held, monkeypatch):
  """A partition of a device may grant smaller clusters, or none: levels of more points than
  they hold are refused by the entry, and such hierarchies are built as ever."""
  host = _lib.host()

  class Levels:
    def __init__(self, *args):
      self.run, self.n = host.SampleLevels(*args), args[0].shape[0]

    def __getattr__(self, name):
      return getattr(self.run, name)

    def add(self, sizes, max_cells, inv_radii, room):
      if min(room, self.n) > held:
        raise _lib.TfgpcError(1, "too large a level for points not counted yet")
      return self.run.add(sizes, max_cells, inv_radii, room)

  class Host:
    SampleLevels = Levels

    def __getattr__(self, name):
      return getattr(host, name)

    def level_points(self, *args):
      return min(host.level_points(*args), held)

  a = cloud(n, 2, 3, 6)
  ref = one_by_one(a, [0.02, 0.04, 0.1], "poisson")
  monkeypatch.setattr(_lib, "host", Host)
  monkeypatch.setattr(pc, "_LEVEL_SIZES", {})
  hier = pc.PointHierarchy(a, [0.02, 0.04, 0.1])
  for got, (_, points, _) in zip(hier._point_clouds[1:], ref):
    assert torch.equal(got._points, points._points)


def host_with(add):
  """The host layer with add(run, ..) in the place of SampleLevels.add."""
  host = _lib.host()

  class Levels:
    def __init__(self, *args):
      self.run = host.SampleLevels(*args)

    def __getattr__(self, name):
      return getattr(self.run, name)

    def add(self, *args):
      return add(self.run, *args)

  class Host:
    SampleLevels = Levels

    def __getattr__(self, name):
      return getattr(host, name)

  return Host


def same_levels(hier, ref):
  assert len(hier._point_clouds) == len(ref) + 1
  for got, neigh, (n, points, _) in zip(hier._point_clouds[1:], hier._neighborhoods, ref):
    assert torch.equal(got._points, points._points)
    for name in ("_sorted_indices", "_sorted_points", "_cur_keys"):
      assert torch.equal(getattr(neigh._grid, name), getattr(n._grid, name))
    assert torch.equal(neigh._neighbors, n._neighbors)


@pytest.mark.parametrize("n,b,d,radii", [(65000, 4, 3, [0.05, 0.1, 0.2, 0.4]),
                                         (100000, 8, 3, [0.03, 0.06, 0.12, 0.24]),
                                         (60000, 1, 2, [0.004, 0.3, 0.4])])
@pytest.mark.parametrize("mode", ["poisson", "average"])
def test_memory_that_a_hierarchy_keeps(n, b, d, radii, mode, monkeypatch):
  """Arrays of levels whose size was not known when they were made are as large as their content,
  and no larger than twice that once such levels have been seen."""
  a = cloud(n, b, d, 12)
  pc.PointHierarchy(a, radii, mode)
  monkeypatch.setattr(pc, "_LEVEL_SIZES", {})

  def kept(build):
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    held = build()
    return torch.cuda.memory_allocated() - before, held

  one_by_one(a, radii, mode)
  own, ref = kept(lambda: one_by_one(a, radii, mode))
  for call in range(3):
    used, hier = kept(lambda: pc.PointHierarchy(a, radii, mode))
    assert used <= 1.3 * own + 3 * (1 << 20)
    same_levels(hier, ref)


@pytest.mark.parametrize("mode", ["poisson", "average"])
def test_levels_known_to_be_too_large_are_not_asked_for(mode, monkeypatch):
  a, radii, asked = cloud(100000, 1, 3, 13), [0.008, 0.01, 0.03], []
  ref = one_by_one(a, radii, mode)
  monkeypatch.setattr(_lib, "host", host_with(lambda run, *args: asked.append(1) or run.add(*args)))
  monkeypatch.setattr(pc, "_LEVEL_SIZES", {})
  same_levels(pc.PointHierarchy(a, radii, mode), ref)
  assert asked
  del asked[:]
  same_levels(pc.PointHierarchy(a, radii, mode), ref)
  assert not asked


def test_levels_larger_than_the_ones_before(monkeypatch):
  """Levels that do not fit what their kind has needed so far are built all the same, and the next
  one's fit; so are those that there is no memory for."""
  small, large = cloud(40000, 2, 3, 14), cloud(40000, 2, 3, 14)
  small._points *= 0.2
  radii = [0.02, 0.04, 0.08]
  ref = one_by_one(large, radii, "poisson")
  monkeypatch.setattr(pc, "_LEVEL_SIZES", {})
  pc.PointHierarchy(small, radii)
  (kind, (seen, _, _)), = pc._LEVEL_SIZES.items()
  for _ in range(2):
    same_levels(pc.PointHierarchy(large, radii), ref)
  now, first, rooms = pc._LEVEL_SIZES[kind]
  assert len(now) == len(seen) == 6 and all(x > y for x, y in zip(now[::2], seen[::2]))
  assert all(x >= y > 0 for x, y in zip(now[1:4:2], seen[1::2])) and len(rooms) == 2
  pc._LEVEL_SIZES[kind] = [[points * (i % 2 == 0) + 2 * (i % 2) for i, points in enumerate(now)],
                           first, [(2, room) for _, room in rooms]]                # too few cells
  for _ in range(2):
    same_levels(pc.PointHierarchy(large, radii), ref)
  assert pc._LEVEL_SIZES[kind] == [now, first, rooms]
  monkeypatch.setattr(_lib, "host", host_with(lambda run, *args: False))           # no memory
  same_levels(pc.PointHierarchy(large, radii), ref)


@pytest.mark.parametrize("unit", [0.25, 3.0, 1.0 / 128])
@pytest.mark.parametrize("mode", ["poisson", "average"])
def test_the_same_scene_in_another_unit(mode, unit, monkeypatch):
  """Levels of a scene that has been seen in another unit of length are made for what it needed
  there (and cell sizes that are no numbers are like no others)."""
  a, rooms = cloud(40000, 2, 3, 16), []
  radii = [0.02, 0.04, 0.08]
  small = cloud(40000, 2, 3, 16)
  small._points *= unit
  ref = one_by_one(small, [r * unit for r in radii], mode)

  def add(run, sizes, max_cells, inv_radii, room):
    rooms.append((max_cells, room))
    return run.add(sizes, max_cells, inv_radii, room)

  monkeypatch.setattr(_lib, "host", host_with(add))
  monkeypatch.setattr(pc, "_LEVEL_SIZES", {})
  for _ in range(2):
    del rooms[:]
    pc.PointHierarchy(a, radii, mode)
  first = list(rooms)
  del rooms[:]
  same_levels(pc.PointHierarchy(small, [r * unit for r in radii], mode), ref)
  assert rooms == first and len(pc._LEVEL_SIZES) == 2
  (kind, _), _ = pc._LEVEL_SIZES.items()
  for no_number in (0.0, float("nan"), float("inf"), -1.0):
    sizes = tuple(tuple(c * no_number for c in size) for size in kind[-1])
    assert pc._same_in_another_unit(kind[:-1] + (sizes,)) is None


def test_grids_that_are_too_fine_are_tried_as_often(monkeypatch):
  """A grid whose table would be too large is tried once in 17 hierarchies, by whichever way the
  level is built."""
  a, tried = cloud(3000, 64, 3, 15), []
  host = _lib.host()

  def levels(*args):
    tried.append(args[4])
    return host.SampleLevels(*args)

  class Host:
    SampleLevels = staticmethod(levels)

    def __getattr__(self, name):
      return getattr(host, name)

  monkeypatch.setattr(_lib, "host", Host)
  for name in ("_TOO_FINE", "_MAX_CELLS", "_LEVEL_SIZES"):
    monkeypatch.setattr(pc, name, {}, raising=False)
  for call in range(18):
    del tried[:]
    hier = pc.PointHierarchy(a, [0.002, 0.2])
    assert len(hier._point_clouds) == 3 and hier._neighborhoods[0]._grid._cells is None
    # (the second level is one of its own: no SampleLevels for it)
    assert bool(tried) == (call in (0, 17)), call


def test_points_of_a_level():
  points = _lib.lib().tfgpc_cell_grid_level_points
  assert points(3, _lib.c_i64(1), 128) in (32768, 65536)
  assert points(3, _lib.c_i64(1), 129) == 0 and points(2, _lib.c_i64(1), 1 << 30) == 0
  assert points(3, _lib.c_i64(342), 2) == 0 and points(3, _lib.c_i64(341), 2) > 0
  assert points(7, _lib.c_i64(1), 2) == points(3, _lib.c_i64(0), 2) == points(3, _lib.c_i64(1), 0) == 0


def test_a_replaced_level_is_called(monkeypatch):
  seen, library = [], pc.PointHierarchy._level
  monkeypatch.setattr(pc.PointHierarchy, "_level",
                      staticmethod(lambda *a: seen.append(1) or library(*a)))
  pc.PointHierarchy(cloud(500, 2, 3, 1), [0.1, 0.2])
  assert len(seen) == 2


def test_a_replaced_cloud_is_called(monkeypatch):
  class Cloud(pc.PointCloud):
    pass

  a = cloud(500, 2, 3, 2)
  monkeypatch.setattr(pc, "PointCloud", Cloud)
  hier = pc.PointHierarchy(a, [0.1, 0.2])
  assert [type(c) for c in hier._point_clouds[1:]] == [Cloud, Cloud]


@pytest.mark.parametrize("radii", [[0.1, 0.0], [0.1, -0.2]])
def test_levels_are_refused_as_before(radii):
  a = cloud(500, 2, 3, 3)
  with pytest.raises(_lib.TfgpcError):
    one_by_one(a, radii, "poisson")
  with pytest.raises(_lib.TfgpcError):
    pc.PointHierarchy(a, radii)


@pytest.mark.parametrize("where", ["_to_dims", "_attach"])
def test_levels_under_way_are_waited_for(where, monkeypatch):
  """Where anything fails between the first level and the report, no kernel is left that would
  write to what the thread's next call reads."""
  a = cloud(5000, 2, 3, 4)
  pc.PointHierarchy(a, [0.1, 0.2])
  holder, calls = (pc, 1) if where == "_to_dims" else (pc.Neighborhood, 0)
  library, seen = getattr(holder, where), []

  def failing(*args, **kwargs):
    seen.append(1)
    if len(seen) > calls:
      raise KeyboardInterrupt
    return library(*args, **kwargs)

  stream = torch.cuda.Stream()
  with torch.cuda.stream(stream):
    torch.cuda._sleep(100_000_000)              # (tens of ms: the levels wait behind it)
    monkeypatch.setattr(holder, where, failing)
    with pytest.raises(KeyboardInterrupt):
      pc.PointHierarchy(a, [0.1, 0.2])
    assert stream.query()
  monkeypatch.undo()
  assert len(pc.PointHierarchy(a, [0.1, 0.2])._point_clouds) == 3


@pytest.mark.parametrize("n,ns,d", [(1, 1, 3), (5000, 700, 3), (5000, 20000, 2), (90000, 70000, 3)])
def test_neighborhood_on_a_grid(n, ns, d):
  a, out = cloud(n, 2, d, n), cloud(ns, 2, d, n + 1)
  grid = pc.Grid(a, 0.1)
  got = pc.grid_neighborhood_on(grid, 0.1, out, bandwidth=0.3)
  ref = pc.grid_neighborhood_with_pdf(a, 0.1, out, bandwidth=0.3)
  assert torch.equal(got._samples_neigh_ranges, ref._samples_neigh_ranges)
  assert torch.equal(got._original_neigh_ids, ref._original_neigh_ids)
  assert torch.equal(got.pdf_by_neighbor_id(), ref.pdf_by_neighbor_id())
  assert d != 3 or torch.equal(got._packed, ref._packed)


def test_a_layer_on_a_grid():
  a, out = cloud(3000, 2, 3, 5), cloud(900, 2, 3, 6)
  g = torch.Generator(device=DEV).manual_seed(7)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  layer = mcconv.MCConv(r(1, 3, 16), r(1, 1, 16), r(1, 128, 32), 8)
  x = r(3000, 8)
  ref = layer.forward(x, a, out, 0.1)
  given = mcconv.layer_on_grid(layer, pc.Grid(a, 0.1))
  assert torch.equal(layer.forward(x, a, out, 0.1, neighborhood=given), ref)
  layer.build_neighborhood = lambda *args: None
  assert mcconv.layer_on_grid(layer, pc.Grid(a, 0.1)) is None


@pytest.mark.parametrize("what", ["narrow cells", "wide cells", "cells per dimension",
                                  "another cloud", "replaced"])
def test_a_layer_is_given_a_grid_of_something_else(what, monkeypatch):
  """A grid with other cells than the layer's radius, or of another cloud than its input, or where
  the call that it stands for is somebody else's: the layer finds its neighbors as usual."""
  a, b, out = cloud(2000, 2, 3, 5), cloud(2000, 2, 3, 8), cloud(600, 2, 3, 6)
  g = torch.Generator(device=DEV).manual_seed(7)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  layer = mcconv.MCConv(r(1, 3, 16), r(1, 1, 16), r(1, 128, 32), 8)
  x = r(2000, 8)
  ref = layer.forward(x, a, out, 0.2)
  cells = {"narrow cells": 0.05, "wide cells": 0.4, "cells per dimension": [0.2, 0.2, 0.1]}
  grid, seen = pc.Grid(b if what == "another cloud" else a, cells.get(what, 0.2)), []
  library = pc.grid_neighborhood_with_pdf
  if what == "replaced":
    monkeypatch.setattr(pc, "grid_neighborhood_with_pdf",
                        lambda *args, **kw: seen.append(1) or library(*args, **kw))
  given = mcconv.layer_on_grid(layer, grid)
  assert torch.equal(layer.forward(x, a, out, 0.2, neighborhood=given), ref)
  assert len(seen) == (what == "replaced")


def test_layers_of_a_classifier_work_on_its_grids(monkeypatch):
  a = cloud(3000, 2, 3, 9)
  hier = pc.PointHierarchy(a, [0.1, 0.2])
  for i, radius in enumerate([0.1, 0.2]):
    assert pc.is_grid_of(hier._neighborhoods[i]._grid, hier._point_clouds[i], radius)
    assert not pc.is_grid_of(hier._neighborhoods[i]._grid, hier._point_clouds[i], 0.15)
