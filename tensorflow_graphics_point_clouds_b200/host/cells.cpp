// Grids with a cell table, neighborhoods, densities and sampling.
#include <algorithm>

#include "host.h"

namespace tfgpc_host {
namespace {

// Arrays of a grid by name, in the order of the struct.
struct Field { const char* name; at::ScalarType type; };
constexpr Field kFields[] = {
    {"aabb_min", at::kFloat}, {"aabb_max", at::kFloat}, {"num_cells", at::kInt},
    {"scaled_aabb_min", at::kFloat}, {"inv_cell_sizes", at::kFloat}, {"keys", at::kLong},
    {"sorted_indices", at::kInt}, {"sorted_keys", at::kLong}, {"sorted_points", at::kFloat},
    {"sorted_batch_ids", at::kInt}, {"packed", at::kFloat}, {"cell_start", at::kInt},
    {"ds", at::kInt}};
constexpr int kNumFields = 13;

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

// A built grid.  All its arrays lie in one allocation; tensors of them are made when
// asked for (most are never looked at).
class CellGrid {
 public:
  tfgpc_cell_grid g{};
  Tensor arena, points, batch_ids;
  std::vector<Tensor> given;            // the arrays a shard's grid got from its caller
  std::vector<int32_t> num_cells_host;

  CellGrid(const Tensor& pts, const Tensor& bids, int64_t batch_size, int max_cells,
           const py::object& cells) {
    points = f32(pts);
    batch_ids = i32(bids);
    on_gpu(points);
    on_gpu(batch_ids);
    require(batch_ids.size(0) == points.size(0),
            "ComputeKeysOp expects the same number of points as batch ids");
    allocate(points.size(0), points.size(1), batch_size, max_cells, points);
    if (!cells.is_none()) {
      void** slot = (void**)&g.aabb_min;
      for (int i : {0, 1, 3, 4}) {
        given.push_back(f32(cells[py::str(kFields[i].name)].cast<Tensor>()));
        slot[i] = given.back().data_ptr();
      }
      given.push_back(i32(cells[py::str("num_cells")].cast<Tensor>()));
    }
  }

  // A grid of at most n points that come later (set_points).
  CellGrid(int64_t n, int64_t d, int64_t batch_size, int max_cells, const Tensor& like) {
    allocate(n, d, batch_size, max_cells, like);
  }

  void set_points(const Tensor& pts, const Tensor& bids) {
    points = pts;
    batch_ids = bids;
    g.n = pts.size(0);
  }

  // Bytes of every array of a grid, in the order of the struct, and of all of them.
  struct Bytes { size_t of[kNumFields], total; };
  static Bytes sizes(int64_t n, int64_t d, int64_t b, int max_cells) {
    const int64_t table = (int64_t)tfgpc_cell_table_elems((int)d, b, max_cells);
    const int64_t elems[kNumFields] = {b * d, b * d, d, b * d, d, n, n, n, n * d, n,
                                       d <= 3 ? 4 * n : 0, table,
                                       2 * b * (int64_t)max_cells * max_cells};
    Bytes s{};
    for (int i = 0; i < kNumFields; ++i) {
      s.of[i] = (size_t)elems[i] * (kFields[i].type == at::kLong ? 8 : 4);
      s.total += align256(s.of[i]);
    }
    return s;
  }

  void allocate(int64_t n, int64_t d, int64_t b, int max_cells, const Tensor& like) {
    g.D = (int)d;
    g.max_cells = max_cells;
    g.n = n;
    g.batch_size = b;
    const Bytes s = sizes(n, d, b, max_cells);
    arena = bytes(s.total, like);
    char* p = (char*)arena.data_ptr();
    void** slot = (void**)&g.aabb_min;
    for (int i = 0; i < kNumFields; ++i) {
      slot[i] = s.of[i] > 0 ? p : nullptr;
      p += align256(s.of[i]);
    }
  }

  // Moves a built grid's arrays to an allocation for no more than its points and (of `max_cells`
  // in a dimension at most) its cells.
  void fit(int max_cells) {
    CellGrid own(g.n, g.D, g.batch_size, max_cells, arena);
    check(tfgpc_cell_grid_copy(stream(), &g, &own.g));
    g = own.g;
    arena = own.arena;
  }

  const int32_t* cells_in() const { return given.empty() ? nullptr : ip(given.back()); }

  Tensor get(const std::string& name) const {
    const int64_t n = g.n, d = g.D, b = g.batch_size;
    if (name == "aabb_min") return view(0, {b, d});
    if (name == "aabb_max") return view(1, {b, d});
    if (name == "num_cells") return view(2, {d});
    if (name == "scaled_aabb_min") return view(3, {b, d});
    if (name == "inv_cell_sizes") return view(4, {d});
    if (name == "keys") return view(5, {n});
    if (name == "sorted_indices") return view(6, {n});
    if (name == "sorted_keys") return view(7, {n});
    if (name == "sorted_points") return view(8, {n, d});
    if (name == "sorted_batch_ids") return view(9, {n});
    if (name == "ds") return view(12, {b, num_cells_host.at(0), num_cells_host.at(1), 2});
    if (name == "num_cells_host") return at::tensor(at::ArrayRef<int32_t>(num_cells_host), at::kInt);
    throw py::attribute_error(name);
  }

 private:
  Tensor view(int field, std::vector<int64_t> shape) const {
    void* p = ((void**)&g.aabb_min)[field];
    for (const Tensor& t : given)
      if (t.data_ptr() == p) return t;
    // (a view of the arena's storage: record_stream on it reaches the allocator)
    int64_t elems = 1;
    for (int64_t x : shape) elems *= x;
    const at::ScalarType type = kFields[field].type;
    return arena.narrow(0, (char*)p - (char*)arena.data_ptr(), elems * (int64_t)c10::elementSize(type))
        .view(type).view(shape);
  }
};

using GridPtr = std::shared_ptr<CellGrid>;

// The samples of a neighborhood: mode 0 the two tensors, 1 the grid's points in their
// own order, 2 the sorted points.
struct Samples {
  int mode = 0;
  int64_t ns = 0;
  Tensor points, ids;
  const float* p() const { return mode == 0 ? fp(points) : nullptr; }
  const int32_t* b() const { return mode == 0 ? ip(ids) : nullptr; }
};

static Samples make_samples(const CellGrid& grid, int mode, const OptTensor& points,
                            const OptTensor& ids) {
  Samples s;
  s.mode = mode;
  s.ns = grid.g.n;
  if (mode != 0) return s;
  require(points.has_value() && ids.has_value(), "FindNeighborsOp got no samples");
  s.points = f32(*points);
  s.ids = i32(*ids);
  on_gpu(s.points);
  on_gpu(s.ids);
  s.ns = s.points.size(0);
  require(s.points.size(1) == grid.g.D,
          "FindNeighborsOp expects inputs with the dimension of the samples");
  require(s.ids.size(0) == s.ns,
          "FindNeighborsOp expects the same number of batch ids as samples.");
  return s;
}

// Ranges and number of pairs of a neighborhood, and what its fill pass needs again.
struct Count {
  GridPtr grid;
  Samples samples;
  Tensor ranges, inv_radii;
  int64_t total = 0;
  int max_neighs = 0;
};

using CountPtr = std::shared_ptr<Count>;

static std::vector<float> to_floats(const std::vector<double>& v) {
  return std::vector<float>(v.begin(), v.end());
}

// (grid, count or None, density at the points in their own order or None, table of
// tfgpc_pack_points_density or None); the last two with inv_bandwidth
static py::tuple build_grid(const Tensor& points, const Tensor& batch_ids, int64_t batch_size,
                            const std::vector<double>& cell_sizes, int max_cells,
                            const py::object& cells, const OptTensor& inv_radii, int mode,
                            const OptTensor& samples, const OptTensor& sample_ids,
                            int max_neighs, const OptTensor& inv_bandwidth, int pdf_mode) {
  GridPtr grid = std::make_shared<CellGrid>(points, batch_ids, batch_size, max_cells, cells);
  CountPtr count;
  if (mode >= 0) {
    count = std::make_shared<Count>();
    count->grid = grid;
    count->samples = make_samples(*grid, mode, samples, sample_ids);
    count->inv_radii = f32(*inv_radii);
    count->max_neighs = max_neighs;
    count->ranges = empty({count->samples.ns}, at::kInt, grid->points);
  }
  const int64_t ns = count ? count->samples.ns : 0;
  const size_t need = tfgpc_cell_grid_workspace_bytes(grid->g.D, grid->g.n, ns, batch_size, max_cells);
  Tensor ws = bytes(need, grid->points);
  const std::vector<float> sizes = to_floats(cell_sizes);
  require((int)sizes.size() == grid->g.D, "GridNeighborhood expects one cell size per dimension");
  OptTensor pdf, packed;
  Tensor inv_bw;
  if (inv_bandwidth) {
    require(inv_radii.has_value(), "GridNeighborhood: densities need radii");
    inv_bw = f32(*inv_bandwidth);
    pdf = empty({grid->g.n}, at::kFloat, grid->points);
    if (grid->g.D == 3) packed = empty({grid->g.n, 4}, at::kFloat, grid->points);
  }
  std::vector<int32_t> nc(grid->g.D);
  int64_t total = 0;
  void* st = stream();
  int rc;
  {
    py::gil_scoped_release release;
    const float* radii = count ? fp(count->inv_radii) : nullptr;
    const float* smp = count ? count->samples.p() : nullptr;
    const int32_t* smp_ids = count ? count->samples.b() : nullptr;
    const int smp_mode = count ? count->samples.mode : 0;
    int32_t* ranges = count ? ipm(count->ranges) : nullptr;
    rc = pdf ? tfgpc_cell_grid_neighborhood_pdf(
                   st, &grid->g, fp(grid->points), ip(grid->batch_ids), sizes.data(),
                   grid->cells_in(), radii, ns, smp, smp_ids, smp_mode, max_neighs, ranges,
                   fp(inv_bw), pdf_mode, fpm(*pdf), packed ? fpm(*packed) : nullptr,
                   ws.data_ptr(), need, nc.data(), &total)
             : tfgpc_cell_grid_neighborhood(
                   st, &grid->g, fp(grid->points), ip(grid->batch_ids), sizes.data(),
                   grid->cells_in(), radii, ns, smp, smp_ids, smp_mode, max_neighs, ranges,
                   ws.data_ptr(), need, nc.data(), &total);
  }
  if (rc) raise_error(rc, tfgpc_last_error(), &nc);
  grid->num_cells_host = nc;
  if (count) count->total = total;
  return py::make_tuple(grid, count, pdf, packed);
}

static CountPtr count_neighbors(const GridPtr& grid, const Tensor& inv_radii, int mode,
                                const OptTensor& samples, const OptTensor& sample_ids,
                                int max_neighs) {
  CountPtr c = std::make_shared<Count>();
  c->grid = grid;
  c->samples = make_samples(*grid, mode, samples, sample_ids);
  c->inv_radii = f32(inv_radii);
  c->max_neighs = max_neighs;
  const int64_t ns = c->samples.ns;
  c->ranges = empty({ns}, at::kInt, grid->points);
  const size_t need = tfgpc_find_neighbors_workspace_bytes(ns);
  Tensor ws = bytes(need, grid->points);
  void* st = stream();
  int rc;
  {
    py::gil_scoped_release release;
    rc = tfgpc_cells_count(st, &grid->g, fp(c->inv_radii), ns, c->samples.p(), c->samples.b(),
                           mode, max_neighs, ipm(c->ranges), ws.data_ptr(), need, &c->total);
  }
  check(rc);
  return c;
}

// (count, density at the points in their own order, table of tfgpc_pack_points_density or None)
static py::tuple count_neighbors_with_pdf(const GridPtr& grid, const Tensor& inv_radii, int mode,
                                          const OptTensor& samples, const OptTensor& sample_ids,
                                          int max_neighs, const Tensor& inv_bandwidth,
                                          int pdf_mode) {
  CountPtr c = std::make_shared<Count>();
  c->grid = grid;
  c->samples = make_samples(*grid, mode, samples, sample_ids);
  c->inv_radii = f32(inv_radii);
  c->max_neighs = max_neighs;
  const int64_t ns = c->samples.ns;
  c->ranges = empty({ns}, at::kInt, grid->points);
  Tensor inv_bw = f32(inv_bandwidth), pdf = empty({grid->g.n}, at::kFloat, grid->points);
  OptTensor packed;
  if (grid->g.D == 3) packed = empty({grid->g.n, 4}, at::kFloat, grid->points);
  const size_t need = tfgpc_cells_count_pdf_workspace_bytes(ns);
  Tensor ws = bytes(need, grid->points);
  void* st = stream();
  int rc;
  {
    py::gil_scoped_release release;
    rc = tfgpc_cells_count_pdf(st, &grid->g, fp(c->inv_radii), ns, c->samples.p(), c->samples.b(),
                               mode, max_neighs, ipm(c->ranges), fp(inv_bw), pdf_mode, fpm(pdf),
                               packed ? fpm(*packed) : nullptr, ws.data_ptr(), need, &c->total);
  }
  check(rc);
  return py::make_tuple(c, pdf, packed);
}

// (pairs with sorted indices, pairs with original indices or None)
static py::tuple fill_neighbors(const CountPtr& c, bool with_ids) {
  const int64_t m = c->total;
  // one allocation: the two lists are mostly used together
  Tensor both = empty({with_ids ? 2 : 1, m, 2}, at::kInt, c->ranges);
  int32_t* neigh = ipm(both);
  check(tfgpc_cells_fill(stream(), &c->grid->g, fp(c->inv_radii), c->samples.ns, c->samples.p(),
                         c->samples.b(), c->samples.mode, c->max_neighs, ip(c->ranges), m, neigh,
                         with_ids ? neigh + 2 * m : nullptr));
  return py::make_tuple(both.select(0, 0),
                        with_ids ? py::cast(both.select(0, 1)) : py::object(py::none()));
}

// Density at every point of the grid, in the unsorted (mode 1) or sorted (2) order.  pairs:
// neighbors of all points within these radii, as far as known.
static Tensor density(const GridPtr& grid, const Tensor& inv_radii, const Tensor& inv_bandwidth,
                      int pdf_mode, int mode, double pairs) {
  Tensor r = f32(inv_radii), bw = f32(inv_bandwidth);
  Tensor out = empty({grid->g.n}, at::kFloat, grid->points);
  // (the rule takes a point's neighbors for those of a uniform cloud; a cloud of fewer than its 256
  // candidates has no more than all its points: 700 clouds of 114 with 98 neighbors 69 us by all
  // tests, 75 by half of them)
  const size_t need = grid->g.n < 256 * grid->g.batch_size ? 0 :
      tfgpc_cells_density_workspace_bytes(grid->g.D, grid->g.n, (int64_t)pairs);
  Tensor ws;
  if (need) ws = bytes(need, grid->points);
  check(tfgpc_cells_density_ws(stream(), &grid->g, fp(r), fp(bw), pdf_mode, grid->g.n, nullptr,
                               nullptr, mode, need ? ws.data_ptr() : nullptr, need, fpm(out)));
  return out;
}

static py::tuple cut_samples(const Tensor& pts, const Tensor& ids, const OptTensor& idx,
                             int64_t s) {
  return py::make_tuple(pts.narrow(0, 0, s), ids.narrow(0, 0, s),
                        idx ? py::cast(idx->narrow(0, 0, s)) : py::object(py::none()));
}

// (points, batch ids, original indices or None) sampled on a built grid
static py::tuple sample(const GridPtr& grid, int mode, const Tensor& inv_radii) {
  const int64_t n = grid->g.n;
  Tensor r = f32(inv_radii);
  Tensor pts = empty({n, grid->g.D}, at::kFloat, grid->points);
  Tensor ids = empty({n}, at::kInt, grid->points);
  OptTensor idx;
  if (mode == 0) idx = empty({n}, at::kInt, grid->points);
  const size_t need = tfgpc_cells_sample_workspace_bytes(n);
  Tensor ws = bytes(need, grid->points);
  int64_t s = 0;
  void* st = stream();
  int rc;
  {
    py::gil_scoped_release release;
    rc = tfgpc_cells_sample(st, &grid->g, mode, fp(r), fpm(pts), ipm(ids),
                            idx ? ipm(*idx) : nullptr, ws.data_ptr(), need, &s);
  }
  check(rc);
  return cut_samples(pts, ids, idx, s);
}

// (grid, points, batch ids, original indices or None): grid and sampling in one call
static py::tuple build_and_sample(const Tensor& points, const Tensor& batch_ids,
                                  int64_t batch_size, const std::vector<double>& cell_sizes,
                                  int max_cells, const py::object& cells, int mode,
                                  const Tensor& inv_radii) {
  GridPtr grid = std::make_shared<CellGrid>(points, batch_ids, batch_size, max_cells, cells);
  const int64_t n = grid->g.n;
  Tensor r = f32(inv_radii);
  Tensor pts = empty({n, grid->g.D}, at::kFloat, grid->points);
  Tensor ids = empty({n}, at::kInt, grid->points);
  OptTensor idx;
  if (mode == 0) idx = empty({n}, at::kInt, grid->points);
  const size_t need = tfgpc_cell_grid_workspace_bytes(grid->g.D, n, 0, batch_size, max_cells);
  const size_t need_s = tfgpc_cells_sample_workspace_bytes(n);
  Tensor ws = bytes(align256(need) + need_s, grid->points);
  char* p = (char*)ws.data_ptr();
  const std::vector<float> sizes = to_floats(cell_sizes);
  require((int)sizes.size() == grid->g.D, "SamplingOp expects one cell size per dimension");
  std::vector<int32_t> nc(grid->g.D);
  int64_t s = 0;
  void* st = stream();
  int rc;
  {
    py::gil_scoped_release release;
    rc = tfgpc_cell_grid_sample(st, &grid->g, fp(grid->points), ip(grid->batch_ids), sizes.data(),
                                grid->cells_in(), mode, fp(r), fpm(pts), ipm(ids),
                                idx ? ipm(*idx) : nullptr, p, need, p + align256(need), need_s,
                                nc.data(), &s);
  }
  if (rc) raise_error(rc, tfgpc_last_error(), &nc);
  grid->num_cells_host = nc;
  py::tuple cut = cut_samples(pts, ids, idx, s);
  return py::make_tuple(grid, cut[0], cut[1], cut[2]);
}

// The levels of a hierarchy one after the other: a level is under way from its add on, so that the
// host makes the next one's arrays meanwhile; finish blocks.  The levels under way write to the
// report page of this thread, as every reporting call of it does: where finish is not reached,
// they are waited for.
class SampleLevels {
 public:
  SampleLevels(const SampleLevels&) = delete;
  SampleLevels& operator=(const SampleLevels&) = delete;
  ~SampleLevels() { wait(); }

  SampleLevels(const Tensor& points, const Tensor& batch_ids, int64_t batch_size,
               const std::vector<double>& cell_sizes, int max_cells, int mode,
               const Tensor& inv_radii)
      : mode_(mode), stream_(stream()) {
    Level level;
    level.grid = std::make_shared<CellGrid>(points, batch_ids, batch_size, max_cells, py::none());
    require(level.grid->g.n > 0, "SamplingOp expects points");
    like_ = level.grid->points;
    counts_ = bytes(TFGPC_MAX_CHAINED_LEVELS * 8, like_);
    enqueue(std::move(level), cell_sizes, inv_radii);
  }

  // A level of at most `room` points; false if there is no memory for so many.
  bool add(const std::vector<double>& cell_sizes, int max_cells, const Tensor& inv_radii,
           int64_t room) {
    require(levels_.size() < TFGPC_MAX_CHAINED_LEVELS, "SamplingOp: too many levels");
    const tfgpc_cell_grid& first = levels_[0].grid->g;
    try {
      Level level;
      level.grid = std::make_shared<CellGrid>(std::min(room, first.n), first.D, first.batch_size,
                                              max_cells, like_);
      enqueue(std::move(level), cell_sizes, inv_radii);
    } catch (const c10::OutOfMemoryError&) {
      return false;
    }
    return true;
  }

  GridPtr grid(int level) const { return levels_.at(level).grid; }

  // Until nothing of it is under way; what the levels have reported is dropped.
  void wait() {
    if (!under_way_) return;
    under_way_ = false;
    int32_t nc[TFGPC_MAX_DIMS];
    int64_t count = 0;
    int done = 0;
    tfgpc_cell_grid_sample_report(stream_, 1, levels_[0].grid->g.D, 1, nc, &count, &done);
  }

  // ([(points, batch ids, original indices or None, cells per dimension at most)] of the levels
  // that could be built, such cells that the next one has asked for)
  py::tuple finish() {
    const int n = (int)levels_.size(), d = levels_[0].grid->g.D;
    std::vector<int32_t> nc((size_t)n * d);
    std::vector<int64_t> counts(n);
    int done = 0, rc;
    under_way_ = false;
    {
      py::gil_scoped_release release;
      rc = tfgpc_cell_grid_sample_report(stream_, n, d, levels_[0].grid->g.max_cells, nc.data(),
                                         counts.data(), &done);
    }
    if (rc) {
      const std::vector<int32_t> first(nc.begin(), nc.begin() + d);
      raise_error(rc, tfgpc_last_error(), &first);
    }
    py::list out;
    for (int l = 0; l < done; ++l) {
      Level& level = levels_[l];
      CellGrid& grid = *level.grid;
      grid.num_cells_host.assign(nc.begin() + l * d, nc.begin() + (l + 1) * d);
      const int cells = *std::max_element(nc.begin() + l * d, nc.begin() + (l + 1) * d);
      const Tensor pts = level.pts.narrow(0, 0, counts[l]), ids = level.ids.narrow(0, 0, counts[l]);
      const size_t own = CellGrid::sizes(grid.g.n, d, grid.g.batch_size, cells).total;
      if (l > 0 && (size_t)grid.arena.numel() > 2 * own + kSpareBytes) {
        try {
          grid.fit(cells);
        } catch (const c10::OutOfMemoryError&) {      // (it stays where it is)
        }
      }
      if (l + 1 < done) levels_[l + 1].grid->set_points(pts, ids);
      out.append(py::make_tuple(pts, ids,
                                level.idx ? py::cast(level.idx->narrow(0, 0, counts[l]))
                                          : py::object(py::none()),
                                cells));
    }
    const auto next = nc.begin() + done * d;
    return py::make_tuple(out, done < n ? *std::max_element(next, next + d) : 0);
  }

 private:
  struct Level {
    GridPtr grid;
    Tensor radii, pts, ids;
    OptTensor idx;
  };

  // A grid whose arrays are larger than twice its size and this gets ones of its size.
  static constexpr size_t kSpareBytes = 1 << 20;

  void enqueue(Level&& level, const std::vector<double>& cell_sizes, const Tensor& inv_radii) {
    const CellGrid& grid = *level.grid;
    const int64_t n = grid.g.n;
    const int l = (int)levels_.size();
    require((int)cell_sizes.size() == grid.g.D, "SamplingOp expects one cell size per dimension");
    const std::vector<float> sizes = to_floats(cell_sizes);
    level.radii = f32(inv_radii);
    level.pts = empty({n, grid.g.D}, at::kFloat, like_);
    level.ids = empty({n}, at::kInt, like_);
    if (mode_ == 0) level.idx = empty({n}, at::kInt, like_);
    const size_t need = tfgpc_cell_grid_workspace_bytes(grid.g.D, n, 0, grid.g.batch_size, grid.g.max_cells);
    const size_t need_s = tfgpc_cells_sample_workspace_bytes(n);
    if (!ws_.defined() || (size_t)ws_.numel() < align256(need) + need_s)
      ws_ = bytes(align256(need) + need_s, like_);
    char* p = (char*)ws_.data_ptr();
    int64_t* counts = (int64_t*)counts_.data_ptr();
    const Level* before = l > 0 ? &levels_[l - 1] : nullptr;
    check(tfgpc_cell_grid_sample_level(
        stream_, l, &grid.g, before ? fp(before->pts) : fp(grid.points),
        before ? ip(before->ids) : ip(grid.batch_ids), before ? counts + l - 1 : nullptr,
        sizes.data(), mode_, fp(level.radii), fpm(level.pts), ipm(level.ids),
        level.idx ? ipm(*level.idx) : nullptr, counts + l, p, need, p + align256(need), need_s));
    levels_.push_back(std::move(level));
    under_way_ = true;
  }

  int mode_;
  bool under_way_ = false;
  void* stream_;
  Tensor like_, counts_, ws_;
  std::vector<Level> levels_;
};

void bind_cells(py::module_& m) {
  py::class_<CellGrid, GridPtr>(m, "CellGrid")
      .def("__getattr__", [](const CellGrid& g, const std::string& name) { return g.get(name); })
      .def_readonly("source_points", &CellGrid::points);
  py::class_<Count, CountPtr>(m, "Count")
      .def_readonly("ranges", &Count::ranges)
      .def_readonly("total", &Count::total)
      .def_readonly("cells", &Count::grid)
      .def_readonly("inv_radii", &Count::inv_radii)
      .def_property_readonly("mode", [](const Count& c) { return c.samples.mode; })
      .def_property_readonly("samples", [](const Count& c) {
        return c.samples.mode == 0 ? c.samples.points
               : c.samples.mode == 1 ? c.grid->points : c.grid->get("sorted_points");
      });
  m.def("cell_table_elems", &tfgpc_cell_table_elems);
  m.def("build_grid", &build_grid);
  m.def("count_neighbors", &count_neighbors);
  m.def("count_neighbors_with_pdf", &count_neighbors_with_pdf);
  m.def("fill_neighbors", &fill_neighbors);
  m.def("density", &density, py::arg("grid"), py::arg("inv_radii"), py::arg("inv_bandwidth"),
        py::arg("pdf_mode"), py::arg("mode"), py::arg("pairs") = 0.0);
  m.def("level_points", &tfgpc_cell_grid_level_points);
  m.def("sample", &sample);
  m.def("build_and_sample", &build_and_sample);
  py::class_<SampleLevels>(m, "SampleLevels")
      .def(py::init<const Tensor&, const Tensor&, int64_t, const std::vector<double>&, int, int,
                    const Tensor&>())
      .def("add", &SampleLevels::add)
      .def("grid", &SampleLevels::grid)
      .def("wait", &SampleLevels::wait)
      .def("finish", &SampleLevels::finish);
}

}  // namespace tfgpc_host
