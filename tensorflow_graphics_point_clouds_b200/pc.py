"""Callers of the custom ops: torch mirrors of the reference's pylib classes.

  PointCloud / AABB   pylib/pc/PointCloud.py:23-134, 235-247
  Grid                pylib/pc/Grid.py:20-83
  Neighborhood        pylib/pc/Neighborhood.py:203-329
  sample              pylib/pc/sampling.py:23-28, 123-150
  PointHierarchy      pylib/pc/PointHierarchy.py:25-98

Only what feeds the ops is kept (segmented [N, D] input with batch ids); the
arithmetic around the ops is float32 torch code that follows the TensorFlow
expressions of the reference one to one, and the ops themselves run through
`custom_ops` (the C ABI).
"""
import itertools
import math
import operator

import torch

from . import custom_ops as ops

SAMPLE_MODES = {'average': 1, 'cell average': 1, 'cell_average': 1,
                'poisson': 0, 'poisson disk': 0, 'poisson_disk': 0}


# Small per-dimension constants (radii, bandwidths) given as Python numbers are
# uploaded once per value and device: creating a device tensor from host data
# blocks the host until the stream has drained, once per call otherwise.  The
# cached tensors are never written to.
_DIMS_CACHE = {}


def _to_dims(value, dims, device, inverse=False):
  """value per dimension as a device tensor, or (inverse) its float32 reciprocal."""
  if type(value) is float:
    t = _DIMS_CACHE.get((value, dims, device, inverse))
    if t is not None:
      return t
  if not torch.is_tensor(value):
    flat = [float(v) for v in (value if hasattr(value, '__len__') else [value])]
    key = (tuple(flat), dims, device, inverse)
    t = _DIMS_CACHE.get(key)
    if t is None:
      if len(_DIMS_CACHE) > 256:
        _DIMS_CACHE.clear()
      t = torch.tensor(flat * dims if len(flat) == 1 else flat, dtype=torch.float32)
      t = (torch.reciprocal(t) if inverse else t).to(device)
      _DIMS_CACHE[key] = t
    if type(value) is float:
      _DIMS_CACHE[value, dims, device, inverse] = t
    return t
  if inverse:
    return torch.reciprocal(_to_dims(value, dims, device))
  t = torch.as_tensor(value, dtype=torch.float32, device=device).reshape(-1)
  if t.shape[0] == 1:
    t = t.repeat(dims)
  return t


def _host_dims(value, dims):
  """value per dimension as a list of floats (a device tensor costs a blocking read)."""
  if type(value) is float:
    return [value] * dims
  flat = (value.detach().reshape(-1).cpu().tolist() if torch.is_tensor(value) else
          [float(v) for v in (value if hasattr(value, '__len__') else [value])])
  return flat * dims if len(flat) == 1 else flat


def _is_array(t, dtype):
  return type(t) is torch.Tensor and t.dtype is dtype and t.is_contiguous()


_LIBRARY_FILL, _LIBRARY_COUNT = ops.find_neighbors_fill, ops.find_neighbors_count
_LIBRARY_PT_GRADS = ops.compute_pdf_pt_grads


class PointCloud:
  """Segmented point cloud: points [N, D] float32 and batch ids [N] int32."""

  def __init__(self, points, batch_ids, batch_size=None, num_cells_reduce=None):
    # num_cells_reduce: for a cloud that is one shard of a batch spread over
    # several ranks.  Grid.py:44-48 takes the cell counts as the maximum over the
    # WHOLE batch; the callable gets this shard's counts ([D] int32 on the device)
    # and returns the maximum over all shards (dist.allreduce_max_), so that every
    # rank builds the keys the unsharded batch would have.
    self._num_cells_reduce = num_cells_reduce
    # (arrays that are what the ops take already, as the output of one is, are looked at once;
    # as_tensor moves the points to a default device, where one is set)
    points = torch.as_tensor(points)
    if not _is_array(points, torch.float32):
      points = points.to(torch.float32).contiguous()
    if not (_is_array(batch_ids, torch.int32) and batch_ids.device == points.device):
      batch_ids = torch.as_tensor(batch_ids, device=points.device).to(torch.int32).contiguous()
    self._points, self._batch_ids = points, batch_ids
    if batch_size is None:
      batch_size = int(ops.read_device(self._batch_ids.max().reshape(1))[0]) + 1
    self._batch_size = int(batch_size)
    self._dimension = self._points.shape[1]
    self._aabb = None

  def get_AABB(self):
    """PointCloud.py:38-43: per-cloud min - 1e-9 and max + 1e-9 in float32."""
    if self._aabb is None:
      mn, mx = ops.compute_aabb(self._points, self._batch_ids, self._batch_size)
      self._aabb = (mn - 1e-9, mx + 1e-9)
    return self._aabb


# Cells per dimension that arrays are sized for, a power of two.  Of a cell table: per
# (dimension, batch size, cell sizes, bits of the number of points) what such a grid asked
# for; for sizes not met before what the last grid of about as many points asked for (the
# same level of a scene in another unit of length), else _first_bound.  Of the key-based
# call's tube array and sort keys: per (dimension, batch size), raised when one did not fit.
# (One bound for both kept every later grid of a batch size on the tables, or off them, that
# its finest one had needed.)
_MAX_CELLS = {}
_FIRST_BOUND = 16
_FIRST_KEY_BOUND = 64
_ONE_CALL_CELLS_LIMIT = 1024
# Grids whose table would be too large: [calls that do not try one again, the bound asked
# for].  Finding that out costs a call its bounding boxes and a blocking read.
_TOO_FINE = {}
_TOO_FINE_CALLS = 16


def _remember(table, key, value):
  if len(table) > 256:
    table.clear()
  table[key] = value


def _asked_bound(err, max_cells):
  """The bound to repeat a call with that reported too few cells; other errors pass."""
  asked = max(getattr(err, 'num_cells', [0]))
  if err.code != 3 or asked <= max_cells:
    raise err
  return 1 << (asked - 1).bit_length()


def _raise_bound(pc, err, max_cells):
  """_asked_bound of the key-based call, or None if a grid this fine would make its
  fixed-size arrays too large."""
  bigger = _asked_bound(err, max_cells)
  if bigger > _ONE_CALL_CELLS_LIMIT or pc._batch_size * float(bigger) ** pc._dimension >= 4e18:
    return None
  _remember(_MAX_CELLS, (pc._dimension, pc._batch_size), bigger)
  return bigger


def _bound_key(pc, sizes):
  return pc._dimension, pc._batch_size, pc._points.shape[0].bit_length(), tuple(sizes)


def _first_bound(pc):
  """Bound where nothing is known: a cell per two points, as far as a table goes."""
  d, b, bound = pc._dimension, pc._batch_size, _FIRST_BOUND
  while 2 * b * bound ** d < pc._points.shape[0] and ops.cell_table_elems(d, b, 2 * bound):
    bound *= 2
  return bound


def _reduced_cells(pc, sizes):
  """Boxes and cell counts of one shard of a distributed batch, the counts reduced
  over the ranks on the device; None for a cloud that is not a shard.  (The reduced
  counts are the same on every rank, so every rank takes the same turns after it.)"""
  if pc._num_cells_reduce is None:
    return None
  cells = ops.grid_cells(pc._points, pc._batch_ids, pc._batch_size, sizes, sizes)
  cells["num_cells"] = pc._num_cells_reduce(cells["num_cells"]).to(torch.int32)
  return cells


def _cell_grid(pc, sizes, build, **args):
  """build (ops.build_cell_grid or ops.build_cell_grid_and_sample) on a cloud with the
  bound of cells it needs; None if the cell table would be too large."""
  d, b = pc._dimension, pc._batch_size
  key = _bound_key(pc, sizes)
  fine = _TOO_FINE.get(key)
  if fine is not None and fine[0] > 0:
    fine[0] -= 1
    return None
  found = known = _MAX_CELLS.get(key)
  like = None if known else key[:3]
  max_cells = known or _MAX_CELLS.get(like) or _first_bound(pc)
  while max_cells <= _ONE_CALL_CELLS_LIMIT and ops.cell_table_elems(d, b, max_cells):
    try:
      built = build(pc._points, pc._batch_ids, b, sizes, max_cells, **args)
    except ops._lib.TfgpcError as err:
      max_cells = known = _asked_bound(err, max_cells)
      if max_cells <= _ONE_CALL_CELLS_LIMIT:       # (where the key-based call starts)
        _remember(_MAX_CELLS, (d, b), max(max_cells, _MAX_CELLS.get((d, b), 0)))
      continue
    if known is None:
      known = max(_FIRST_BOUND, 1 << (max(built[0].num_cells_host.tolist()) - 1).bit_length())
    if found != known:
      _remember(_MAX_CELLS, key, known)
      if like is not None:
        _remember(_MAX_CELLS, like, known)
    if fine is not None:
      _TOO_FINE.pop(key, None)
    return built
  _remember(_TOO_FINE, key, [_TOO_FINE_CALLS, max_cells])
  return None


class Grid:
  """Grid.py:32-83: keys, descending sort, sorted copies, tube ranges.  Built through
  a cell table (ops.CellGrid) unless the grid is too fine for one."""

  def __init__(self, point_cloud, cell_sizes):
    cells, pc = None, point_cloud
    if pc._points.shape[0] > 0:
      sizes = _host_dims(cell_sizes, pc._dimension)
      cells = _reduced_cells(pc, sizes)
      built = _cell_grid(pc, sizes, ops.build_cell_grid, cells=cells)
      if built is not None:
        self._cell_sizes = _to_dims(cell_sizes, pc._dimension, pc._points.device)
        self._adopt(pc, built[0], sizes)
        return
    self._build_by_keys(pc, cell_sizes, cells)

  def _build_by_keys(self, pc, cell_sizes, cells):
    """Boxes, keys and radix sort one by one.  cells: see _reduced_cells."""
    dev = pc._points.device
    self._cell_sizes = _to_dims(cell_sizes, pc._dimension, dev)
    self._cells = None
    self._point_cloud = pc
    self._batch_size = pc._batch_size
    self._aabb_min, self._aabb_max = pc.get_AABB()
    sizes = self._aabb_max - self._aabb_min
    if cells is not None:
      self._num_cells = cells["num_cells"]
    else:
      batch_num_cells = torch.ceil(sizes / self._cell_sizes).to(torch.int32)
      self._num_cells = torch.clamp(batch_num_cells.max(dim=0).values, min=1).to(torch.int32)
      if pc._num_cells_reduce is not None:
        self._num_cells = pc._num_cells_reduce(self._num_cells).to(torch.int32)
    self._num_cells_host = ops.read_device(self._num_cells)
    # custom_ops_wrapper.py:37-43
    self._scaled_aabb_min = self._aabb_min / self._cell_sizes
    self._inv_cell_sizes = torch.reciprocal(self._cell_sizes)
    self._cur_keys = ops.compute_keys(pc._points, pc._batch_ids, self._scaled_aabb_min,
                                      self._num_cells, self._inv_cell_sizes)
    total = self._batch_size
    for c in self._num_cells_host.tolist():
      total *= int(c)
    key_bits = max(1, int(math.ceil(math.log2(total + 1))))
    (self._sorted_indices, self._sorted_keys, self._sorted_points,
     self._sorted_batch_ids) = ops.sort_keys_desc(self._cur_keys, pc._points, pc._batch_ids,
                                                  key_bits=min(64, key_bits))
    self._fast_DS = None

  def _adopt(self, pc, built, sizes):
    """Takes over a grid of ops.build_cell_grid with cells of these sizes."""
    self._cells = built
    self._sizes = sizes
    self._point_cloud = pc
    self._batch_size = pc._batch_size
    self._fast_DS = None

  _FIELDS = {'_cur_keys': 'keys'}

  def __getattr__(self, name):
    # arrays of a grid built through a cell table become tensors when first asked for
    cells = self.__dict__.get('_cells')
    if cells is None or not name.startswith('_') or name.startswith('__'):
      raise AttributeError(name)
    value = getattr(cells, self._FIELDS.get(name, name[1:]))
    self.__dict__[name] = value
    return value

  def get_DS(self):
    if self._fast_DS is None and self._cells is not None:
      self._fast_DS = self._cells.ds
    if self._fast_DS is None:
      self._fast_DS = ops.build_grid_ds(self._sorted_keys, self._num_cells,
                                        self._num_cells_host, self._batch_size)
    return self._fast_DS


class Neighborhood:
  """Neighborhood.py:218-329.  The count pass runs in the constructor (ranges and
  the number of pairs are known from then on); the neighbor list is written when
  it is first asked for, in one pass together with the list in original ids."""

  def __init__(self, grid, radius, point_cloud_sample=None, max_neighbors=0):
    self._attach(grid, radius, point_cloud_sample, max_neighbors)
    self._counted = self._run_count()

  def _attach(self, grid, radius, point_cloud_sample, max_neighbors, counted=None):
    cloud = grid._point_cloud
    dev, d = cloud._points.device, cloud._dimension
    self._radius = radius
    self._radii = _to_dims(radius, d, dev)
    self._inv_radii = _to_dims(radius, d, dev, inverse=True)
    self._equal_samples = point_cloud_sample is None
    self._sampled = point_cloud_sample
    # 2: the sorted points, 1: the grid's own cloud in its unsorted order, 0: other samples
    self._sample_mode = (2 if point_cloud_sample is None else
                         1 if point_cloud_sample is cloud else 0)
    self._grid = grid
    self.max_neighbors = max_neighbors
    self._counted = counted
    self._nbrs = self._orig_ids = self._pdf = self._point_pdf = self._sample_pdf = None
    self._packed = None       # (points, 1 / density) as one row per point, where known
    self._pdf_ready = False
    self._transposed = None
    return self

  def _run_count(self):
    grid = self._grid
    if grid._cells is not None:
      smp = self._sampled if self._sample_mode == 0 else None
      return ops._lib.host().count_neighbors(
          grid._cells, self._inv_radii, self._sample_mode, None if smp is None else smp._points,
          None if smp is None else smp._batch_ids, self.max_neighbors)
    smp = self._point_cloud_sampled
    return ops.find_neighbors_count(
        smp._points, smp._batch_ids, grid._sorted_points, grid._sorted_keys, grid.get_DS(),
        grid._num_cells, grid._scaled_aabb_min, grid._inv_cell_sizes, self._inv_radii,
        self.max_neighbors, sample_order=self._sample_order)

  @property
  def _count(self):
    # (a neighborhood of a PointHierarchy, whose sampling reads no lists, counts here)
    if self._counted is None:
      self._counted = self._run_count()
    return self._counted

  @property
  def _samples_neigh_ranges(self):
    return self._count.ranges

  @property
  def _point_cloud_sampled(self):
    if self._sampled is None:
      g = self._grid
      self._sampled = PointCloud(g._sorted_points, g._sorted_batch_ids, g._batch_size)
    return self._sampled

  @property
  def _sample_order(self):
    # a sequence that visits the samples cell by cell, where one is known: for the
    # grid's own cloud the key sort's permutation (the samples of a self
    # neighborhood are the sorted points: already in it)
    return self._grid._sorted_indices if self._sample_mode == 1 else None

  @property
  def num_pairs(self):
    return self._count.total

  def _fill(self):
    """Writes the neighbor list [M, 2] (index into the sorted points, sample
    index) and, in the same pass, the list with the neighbors' indices in the
    unsorted point order (Neighborhood.py:246-250)."""
    if self._nbrs is not None:
      return
    if self._equal_samples:
      # a self neighborhood mostly feeds the density estimate and the sampling,
      # which read sorted ids only: the original-id list is built if asked for
      self._nbrs = ops.find_neighbors_fill(self._count)
    elif self._count.cells is not None and ops.find_neighbors_fill is _LIBRARY_FILL:
      # (the library's own needs no permutation as a tensor)
      self._nbrs, self._orig_ids = ops._cells_fill(self._count, True, None, None)
    else:
      self._nbrs, self._orig_ids = ops.find_neighbors_fill(self._count,
                                                            self._grid._sorted_indices)

  @property
  def _neighbors(self):
    self._fill()
    return self._nbrs

  @property
  def _original_neigh_ids(self):
    self._fill()
    if self._orig_ids is None:
      self._orig_ids, _ = ops.original_neighbor_ids(self._nbrs, self._grid._sorted_indices)
    return self._orig_ids

  def _pairs_of_all_points(self):
    """About how many neighbors the grid's points have in all, 0 if nothing is counted yet."""
    count = self._counted
    if count is None or count.ranges.shape[0] == 0:
      return 0.0
    return float(count.total) * self._grid._point_cloud._points.shape[0] / count.ranges.shape[0]

  def _samples_are_grid_points(self):
    return self._equal_samples or (self._sample_mode == 1 and self.max_neighbors == 0)

  def compute_pdf(self, bandwidth=0.2, mode=0):
    """Neighborhood.py:257-311 (mode: 0 constant bandwidth, 1 by point count).
    The density is needed at every neighbor point.  pylib gets it from a second,
    self neighborhood of the grid (Neighborhood.py:284); when the samples are the
    grid's own cloud that second search is skipped: the density at sample s is
    the density of the point it coincides with."""
    g = self._grid
    d = g._point_cloud._dimension
    inv_bw, inv_r = _to_dims(bandwidth, d, self._radii.device, inverse=True), self._inv_radii
    self._pdf = self._point_pdf = self._sample_pdf = self._packed = None
    if g._cells is not None and not (self._equal_samples and self.max_neighbors > 0):
      # straight from the grid, without the list of a self neighborhood; by original
      # index, which the layers read the densities by, unless the samples are sorted
      pairs = self._pairs_of_all_points()
      if self._equal_samples:
        self._point_pdf = ops._lib.host().density(g._cells, inv_r, inv_bw, mode, 2, pairs)
      else:
        self._sample_pdf = ops._lib.host().density(g._cells, inv_r, inv_bw, mode, 1, pairs)
    elif self._equal_samples:
      self._point_pdf = ops.compute_pdf_with_pt_grads(
          g._sorted_points, self._neighbors, self._samples_neigh_ranges, inv_bw, inv_r, mode)
    elif self._samples_are_grid_points():
      # sample s is point s of the unsorted cloud
      self._sample_pdf = ops.compute_pdf_at_samples(
          self._point_cloud_sampled._points, g._sorted_points, self._neighbors,
          self._samples_neigh_ranges, inv_bw, inv_r, mode)
      self._point_pdf = None
    else:
      nb = Neighborhood(g, self._radius)
      self._point_pdf = ops.compute_pdf_with_pt_grads(
          g._sorted_points, nb._neighbors, nb._samples_neigh_ranges, inv_bw, inv_r, mode)
    self._pdf_ready = True

  def pdf_by_neighbor_id(self, **kwargs):
    """The densities as a table indexed by the FIRST column of _original_neigh_ids
    (one value per point of the grid's cloud), where the neighborhood has them in
    that form, else None: kernels that take the table read it in place of the
    per-pair array of get_pdf."""
    if not self._pdf_ready:
      self.compute_pdf(**kwargs)
    return self._sample_pdf

  def point_pdf(self, **kwargs):
    """Density of every point of the grid, in the SORTED order of the grid."""
    if not self._pdf_ready:
      self.compute_pdf(**kwargs)
    if self._point_pdf is None:
      self._point_pdf = self._sample_pdf[self._grid._sorted_indices.to(torch.int64)]
    return self._point_pdf

  def transpose(self):
    """Neighborhood.py:318-329: the neighborhood with the roles of samples and
    points exchanged (the samples' cloud on a grid of its own, searched around the
    points of this one); a self neighborhood is its own transpose."""
    if self._transposed is None:
      if self._equal_samples:
        self._transposed = self
      else:
        grid = Grid(self._point_cloud_sampled, self._radius)
        self._transposed = Neighborhood(grid, self._radius, self._grid._point_cloud)
    return self._transposed

  def get_pdf(self, **kwargs):
    """[M] density of every pair's neighbor point (Neighborhood.py:287)."""
    if not self._pdf_ready:
      self.compute_pdf(**kwargs)
    if self._pdf is None:
      if self._sample_pdf is not None:
        self._pdf = self._sample_pdf[self._original_neigh_ids[:, 0].to(torch.int64)]
      else:
        self._pdf = self._point_pdf[self._neighbors[:, 0].to(torch.int64)]
    return self._pdf

  def pdf_point_grads(self, pdf_grads, bandwidth=0.2, mode=0):
    """Gradient of a loss with respect to the grid's points [N, D] (in their
    original order) through the per-pair densities of get_pdf, given the loss's
    gradient pdf_grads [M] with respect to those densities.  The chain of the
    reference's autodiff: pdf[m] = point_pdf[neighbors[m, 0]] (Neighborhood.py:287),
    point_pdf = ComputePdfWithPtGrads(sorted points, self neighborhood), whose
    registered gradient is ComputePdfPtGrads (custom_ops_wrapper.py:159-169), and
    sorted points = gather(points, sorted indices) (Grid.py:60-62)."""
    g = self._grid
    d = g._point_cloud._dimension
    inv_bw = _to_dims(bandwidth, d, self._radii.device, inverse=True)
    n = g._point_cloud._points.shape[0]
    pdf_grads = torch.as_tensor(pdf_grads, dtype=torch.float32)
    # the library's lists of a self neighborhood without limit are symmetric
    pt_grads = ops.compute_pdf_pt_grads
    if (pt_grads is _LIBRARY_PT_GRADS and not (self._equal_samples and self.max_neighbors > 0) and
        ops.find_neighbors_fill is _LIBRARY_FILL and ops.find_neighbors_count is _LIBRARY_COUNT and
        type(self) is Neighborhood is _LIBRARY_NEIGHBORHOOD):
      pt_grads = ops.compute_pdf_pt_grads_symmetric
    if not self._equal_samples and self._samples_are_grid_points():
      # the grid's own cloud as samples: these lists are the self neighborhood's, in the
      # points' own order
      ids = self._original_neigh_ids
      per_point = ops._lib.host().add_by_neighbor(ids, pdf_grads, n)
      return pt_grads(g._point_cloud._points, ids, self._samples_neigh_ranges, inv_bw,
                      self._inv_radii, per_point, mode)
    per_point = ops._lib.host().add_by_neighbor(self._neighbors, pdf_grads, n)
    nb = self if self._equal_samples else Neighborhood(g, self._radius)
    grads_sorted = pt_grads(g._sorted_points, nb._neighbors, nb._samples_neigh_ranges, inv_bw,
                            self._inv_radii, per_point, mode)
    out = torch.empty_like(grads_sorted)
    out[g._sorted_indices.to(torch.int64)] = grads_sorted
    return out


_LIBRARY_NEIGHBORHOOD = Neighborhood
LIBRARY_GET_PDF = Neighborhood.get_pdf     # (the class's own may be replaced: mcconv.PointConv)


def grid_neighborhood(point_cloud, radius, point_cloud_sample=None, max_neighbors=0):
  """Grid(point_cloud, radius) and Neighborhood(grid, radius, point_cloud_sample,
  max_neighbors) built by ONE library call with ONE blocking read where pylib's two
  constructors read back twice (Grid.py:44-48 cell counts, Neighborhood.py:242-245 pair
  count).  Same objects, same contents: on the cell table (ops.build_cell_grid), or by
  keys (tfgpc_grid_neighborhood_count) for grids too fine for one.  For a cloud that is
  one shard of a distributed batch (num_cells_reduce set) the cell counts are reduced
  over the ranks on the device, before the main call: still one blocking read."""
  return grid_neighborhood_with_pdf(point_cloud, radius, point_cloud_sample, max_neighbors, None)


def grid_neighborhood_with_pdf(point_cloud, radius, point_cloud_sample=None, max_neighbors=0,
                               bandwidth=0.2, mode=0):
  """grid_neighborhood followed by compute_pdf(bandwidth, mode) (None: without it).  The
  densities need the grid only, so they are worked out while the host reads the number
  of pairs and goes on."""
  if point_cloud._points.shape[0] == 0:
    return Neighborhood(Grid(point_cloud, radius), radius, point_cloud_sample, max_neighbors)
  sizes = _host_dims(radius, point_cloud._dimension)
  return _grid_neighborhood(point_cloud, radius, sizes, point_cloud_sample, max_neighbors,
                            _reduced_cells(point_cloud, sizes), bandwidth, mode)


def _grid_neighborhood(pc, radius, sizes, point_cloud_sample, max_neighbors, cells,
                       bandwidth=None, pdf_mode=0):
  """grid_neighborhood of a cloud with points whose counts have been reduced: whether
  a rank's grid fits a table depends on its own share of the batch, and a second
  reduction on some ranks only would meet another one of theirs."""
  dev = pc._points.device
  d = pc._dimension
  # (the sorted points' densities come in the sorted order: compute_pdf's)
  with_pdf = bandwidth is not None and point_cloud_sample is not None
  mode = 2 if point_cloud_sample is None else 1 if point_cloud_sample is pc else 0
  smp = point_cloud_sample if mode == 0 else None
  samples = dict(samples=None if smp is None else smp._points,
                 samples_batch_ids=None if smp is None else smp._batch_ids,
                 samples_are_points=mode, max_neighs=max_neighbors)
  inv_radii = _to_dims(radius, d, dev, inverse=True)
  if with_pdf:
    built = _cell_grid(pc, sizes, ops.build_cell_grid_with_pdf, cells=cells, inv_radii=inv_radii,
                       inv_bandwidth=_to_dims(bandwidth, d, dev, inverse=True), pdf_mode=pdf_mode,
                       **samples)
  else:
    built = _cell_grid(pc, sizes, ops.build_cell_grid, cells=cells, inv_radii=inv_radii, **samples)
  grid = object.__new__(Grid)
  grid._cell_sizes = _to_dims(radius, d, dev)
  if built is not None:
    grid._adopt(pc, built[0], sizes)
    count = built[1]
  else:
    max_cells = _MAX_CELLS.get((d, pc._batch_size), _FIRST_KEY_BOUND)
    asked = _TOO_FINE.get(_bound_key(pc, sizes), [0, 0])[1]
    if asked > _ONE_CALL_CELLS_LIMIT:
      max_cells = None
    while True:
      if max_cells is None:
        # the separate constructors size the tube array and the sort keys exactly
        grid._build_by_keys(pc, radius, cells)
        return Neighborhood(grid, radius, point_cloud_sample, max_neighbors)
      try:
        g = ops.grid_neighborhood_count(pc._points, pc._batch_ids, pc._batch_size, sizes, sizes,
                                        max_cells, cells=cells, **samples)
        break
      except ops._lib.TfgpcError as err:
        max_cells = _raise_bound(pc, err, max_cells)
    grid._cells, count = None, g.pop("count")
    grid._point_cloud, grid._batch_size = pc, pc._batch_size
    grid._cur_keys, grid._fast_DS = g.pop("keys"), g.pop("ds")
    for name, value in g.items():
      setattr(grid, '_' + name, value)
  neigh = object.__new__(Neighborhood)._attach(grid, radius, point_cloud_sample, max_neighbors,
                                               count)
  if with_pdf and built is not None:
    neigh._sample_pdf, neigh._packed, neigh._pdf_ready = built[2], built[3], True
  return neigh


_LIBRARY_WITH_PDF, _LIBRARY_BUILD_WITH_PDF = grid_neighborhood_with_pdf, ops.build_cell_grid_with_pdf


def is_grid_of(grid, point_cloud, radius):
  """Whether grid_neighborhood_on(grid, radius, ..) is what grid_neighborhood_with_pdf gives
  for this cloud: a grid over it with cells of this radius (wider ones would list the same
  neighbors from more candidates, narrower ones would miss some), and nobody has replaced what
  would be called else."""
  return (type(grid) is Grid and grid._point_cloud is point_cloud and
          grid._cell_sizes is _to_dims(radius, point_cloud._dimension, point_cloud._points.device) and
          grid_neighborhood_with_pdf is _LIBRARY_WITH_PDF and
          ops.build_cell_grid_with_pdf is _LIBRARY_BUILD_WITH_PDF)


def grid_neighborhood_on(grid, radius, point_cloud_sample, bandwidth=0.2, mode=0):
  """grid_neighborhood_with_pdf on a grid of cells of `radius` that is there already, the
  samples another cloud's."""
  if grid._cells is None or point_cloud_sample is grid._point_cloud:
    neigh = Neighborhood(grid, radius, point_cloud_sample)
    neigh.compute_pdf(bandwidth=bandwidth, mode=mode)
    return neigh
  neigh = object.__new__(Neighborhood)._attach(grid, radius, point_cloud_sample, 0)
  inv_bw = _to_dims(bandwidth, grid._point_cloud._dimension, neigh._radii.device, inverse=True)
  neigh._counted, neigh._sample_pdf, neigh._packed = ops._lib.host().count_neighbors_with_pdf(
      grid._cells, neigh._inv_radii, 0, point_cloud_sample._points, point_cloud_sample._batch_ids,
      0, inv_bw, mode)
  neigh._pdf_ready = True
  return neigh


# Cells up to this many radii wide are sampled from the grid, wider ones from a neighbor
# list: a cell's taken points are marked around by one block, (taken) x (candidates) tests,
# and a wide cell holds many of both (and is a turn of the block per taken point).  From the grid /
# by lists, us, at 1, 3, 4, 6 and 8 radii: 100 000 points 96/260, 376/1141, 1251/2158, 6240/5650,
# 17115/10160 (40 neighbors a point), 106/279, 230/386, 723/630, 1803/1507, 6490/3040 (6);
# 20 000 points 54/202, 234/260, 680/367, 1244/748, 2633/1375 (6).
_SAMPLED_CELLS = 3.0


def _cells_near_radius(neighborhood):
  g = neighborhood._grid
  radii = _host_dims(neighborhood._radius, g._point_cloud._dimension)
  return all(c <= _SAMPLED_CELLS * abs(r) for c, r in zip(g._sizes, radii))


def sample(neighborhood, sample_mode='poisson'):
  """sampling.py:123-150 -> (PointCloud of the samples, original indices or None)."""
  mode = SAMPLE_MODES[sample_mode.lower()]
  g = neighborhood._grid
  symmetric = neighborhood._equal_samples and neighborhood.max_neighbors == 0
  if g._cells is not None and (mode == 1 or symmetric and _cells_near_radius(neighborhood)):
    # (cell averages need no neighbors, symmetric ones are found from the grid)
    pts, bids, idx = ops._lib.host().sample(g._cells, mode, neighborhood._inv_radii)
    return PointCloud(pts, bids, g._batch_size), idx
  pts, bids, idx = ops.sampling(g._sorted_points, g._sorted_batch_ids, g._sorted_keys,
                                g._num_cells, neighborhood._neighbors,
                                neighborhood._samples_neigh_ranges, mode, symmetric=symmetric)
  if mode == 0:
    idx = g._sorted_indices[idx.to(torch.int64)]
  else:
    idx = None
  return PointCloud(pts, bids, g._batch_size), idx


# Levels of one call (tfgpc_cell_grid_sample_level).
_LEVELS_MOST = 16
# Per kind of hierarchy (device, dimension, batch size, bits of the number of points, mode, cell
# sizes): [the most points and the most cells in a dimension (0: not known) that its levels behind
# the first have had, one after the other; the first one's bound of cells; (bound of cells, points)
# that the next such levels are made for].  Without, for as many points as a cluster holds.
_LEVEL_SIZES = {}
_LIBRARY_BUILD_AND_SAMPLE = ops.build_cell_grid_and_sample


def _level_rooms(host, batch_size, all_sizes, max_cells, seen):
  """[(bound of cells, points)] that the levels behind the first are made for, as far as they can
  follow it.  max_cells: the first one's bound; seen: see _LEVEL_SIZES."""
  rooms, first, d = [], all_sizes[0], len(all_sizes[0])
  seen = list(seen) + [0, 0] * len(all_sizes)
  for level, points, cells in zip(all_sizes[1:], seen[::2], seen[1::2]):
    # the box of a level lies in the one before: its cells are known to be no more than these
    bound = max_cells * max(a / c for a, c in zip(first, level)) + 1.0
    if bound > _ONE_CALL_CELLS_LIMIT:
      break
    bound = 1 << ((min(math.ceil(bound), cells) if cells else math.ceil(bound)) - 1).bit_length()
    room = host.level_points(d, batch_size, bound)      # (what a cluster holds: by the device)
    if room == 0 or points > room:
      break
    # (some more than there have been: they vary)
    rooms.append((bound, min(room, 1 << (points + points // 4).bit_length()) if points else room))
  return rooms


def _same_in_another_unit(kind):
  """What is known of hierarchies that differ from these in the unit of length alone, or None.
  (Grids made for as many points as a cluster holds are moved when they are built: the first
  hierarchy in a unit, of 45 000 points in three levels, took 240 us so and takes 214, of 800 000
  in four 620 and 587.)"""
  sizes = kind[-1]
  for other, known in reversed(list(_LEVEL_SIZES.items())):
    if other[:-1] == kind[:-1] and len(other[-1]) == len(sizes):
      unit = sizes[0][0] / other[-1][0][0]
      if unit > 0.0 and all(abs(x * unit - y) <= 1e-6 * y      # (not so where one is no number)
                            for a, c in zip(other[-1], sizes) for x, y in zip(a, c)):
        return known
  return None


class PointHierarchy:
  """PointHierarchy.py:40-98: per level Grid -> self Neighborhood -> sample.  Grid and
  sampling of a level are one library call; the levels after one follow it without a
  blocking read of their own, as long as one cluster can build their grids (65 536 points
  at most).  The neighborhoods count and write their lists when they are used (the sampling
  needs none)."""

  def __init__(self, point_cloud, cell_sizes, sample_mode='poisson'):
    self._point_clouds = [point_cloud]
    self._neighborhoods = []
    self._sample_indices = []
    cur, done, cell_sizes = point_cloud, 0, list(cell_sizes)
    while done < len(cell_sizes):
      levels = self._levels(cur, cell_sizes[done:], sample_mode)
      for neigh, cur, idx in levels or [self._level(cur, cell_sizes[done], sample_mode)]:
        self._neighborhoods.append(neigh)
        self._point_clouds.append(cur)
        self._sample_indices.append(idx)
        done += 1

  def _levels(self, pc, cell_sizes, sample_mode):
    """Several levels in one call, or None where that is not for these."""
    n, d, b = pc._points.shape[0], pc._dimension, pc._batch_size
    if (len(cell_sizes) < 2 or n == 0 or pc._num_cells_reduce is not None or
        getattr(self._level, '__func__', self._level) is not _LIBRARY_LEVEL or
        ops.build_cell_grid_and_sample is not _LIBRARY_BUILD_AND_SAMPLE or
        PointCloud is not _LIBRARY_CLOUD or PointCloud.__init__ is not _LIBRARY_CLOUD_INIT or
        torch.as_tensor(pc._points) is not pc._points):       # (a default device moves them)
      return None
    all_sizes = [_host_dims(cs, d) for cs in cell_sizes[:_LEVELS_MOST]]
    dev, host = pc._points.device, ops._lib.host()
    mode = SAMPLE_MODES[sample_mode.lower()]
    kind = dev, d, b, n.bit_length(), mode, tuple(map(tuple, all_sizes))
    known = _LEVEL_SIZES.get(kind)
    like = None if known else _same_in_another_unit(kind)
    if not (known or like) and (host.level_points(d, b, 1) == 0 or
                                not all(0.0 < c < math.inf for size in all_sizes for c in size)):
      return None
    seen, first, rooms = known or like or ((), 0, ())

    def build(points, batch_ids, batch_size, sizes, max_cells):
      run = host.SampleLevels(points, batch_ids, batch_size, sizes, max_cells, mode,
                              _to_dims(cell_sizes[0], d, dev, inverse=True))
      try:
        return further_levels(run, points, sizes, max_cells)
      except BaseException:
        run.wait()          # (its kernels write where the next call of this thread reads)
        raise

    def further_levels(run, points, sizes, max_cells):
      made = rooms if max_cells == first else _level_rooms(host, b, all_sizes, max_cells, seen)
      taken = 1
      for bound, room in made:
        if not run.add(all_sizes[taken], bound, _to_dims(cell_sizes[taken], d, dev, inverse=True),
                       room):
          break
        taken += 1
      # what does not take the numbers of samples is made while they are worked out
      cloud, levels = pc, []
      for l in range(taken):
        grid = object.__new__(Grid)
        grid._cell_sizes = _to_dims(cell_sizes[l], d, dev)
        grid._adopt(cloud, run.grid(l), all_sizes[l])
        neigh = object.__new__(Neighborhood)._attach(grid, cell_sizes[l], None, 0)
        cloud = object.__new__(PointCloud)
        # (what its constructor sets, its own points once they are known)
        cloud._points, cloud._batch_size, cloud._dimension = points, b, d
        cloud._num_cells_reduce = cloud._aabb = None
        levels.append((neigh, cloud))
      built, asked = run.finish()
      return levels[0][0]._grid._cells, levels, built, asked, max_cells, made[:taken - 1]

    built = _cell_grid(pc, all_sizes[0], build)
    if built is None:       # (_level looks at the same grid again: one try between them)
      fine = _TOO_FINE.get(_bound_key(pc, all_sizes[0]))
      if fine is not None:
        fine[0] += 1
      return None
    _, levels, built, asked, max_cells, made = built
    done, now = [], []
    for (neigh, cloud), (points, batch_ids, idx, cells) in zip(levels, built):
      if done:              # (what a grid of this cloud asks for, as _cell_grid keeps it)
        bound = max(_FIRST_BOUND, 1 << (cells - 1).bit_length())
        key = _bound_key(neigh._grid._point_cloud, neigh._grid._sizes)
        for known in (key, key[:3]):
          if _MAX_CELLS.get(known) != bound:
            _remember(_MAX_CELLS, known, bound)
        now += held, cells
      cloud._points, cloud._batch_ids = points, batch_ids
      held = points.shape[0]
      done.append((neigh, cloud, idx))
    missed = len(done) <= len(made)
    if like and max_cells != first:
      seen = ()             # (a scene of another density)
    if missed:
      # the next level got more points or cells than there was room for, those behind it may too
      now += held, asked if held <= made[len(done) - 1][1] else 0
      seen = seen[:len(now) - 1]
    else:
      now += held, 0
    if missed or max_cells != first or len(now) > len(seen) or any(map(operator.gt, now, seen)):
      seen = [max(x) for x in itertools.zip_longest(seen, now, fillvalue=0)]
      _remember(_LEVEL_SIZES, kind, [seen, max_cells,
                                     _level_rooms(host, b, all_sizes, max_cells, seen)])
    elif like:
      _remember(_LEVEL_SIZES, kind, like)
    return done

  @staticmethod
  def _level(pc, radius, sample_mode):
    mode = SAMPLE_MODES[sample_mode.lower()]
    if pc._points.shape[0] == 0:
      neigh = grid_neighborhood(pc, radius)
      return (neigh,) + sample(neigh, sample_mode)
    dev, d = pc._points.device, pc._dimension
    sizes = _host_dims(radius, d)
    cells = _reduced_cells(pc, sizes)
    built = _cell_grid(pc, sizes, ops.build_cell_grid_and_sample, mode=mode,
                       inv_radii=_to_dims(radius, d, dev, inverse=True), cells=cells)
    if built is None:
      neigh = _grid_neighborhood(pc, radius, sizes, None, 0, cells)
      return (neigh,) + sample(neigh, sample_mode)
    grid = object.__new__(Grid)
    grid._cell_sizes = _to_dims(radius, d, dev)
    grid._adopt(pc, built[0], sizes)
    neigh = object.__new__(Neighborhood)._attach(grid, radius, None, 0)
    return neigh, PointCloud(built[1], built[2], pc._batch_size), built[3]


_LIBRARY_LEVEL = PointHierarchy._level
_LIBRARY_CLOUD, _LIBRARY_CLOUD_INIT = PointCloud, PointCloud.__init__
