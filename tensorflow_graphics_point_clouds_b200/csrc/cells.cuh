// The cell table of a grid: where every cell's points begin in the sorted order.
//
// Keys are sorted DESCENDING, so bucket R(key) = total - key (total = batch size x
// cells) counts up along the sorted points.  start[R] is the first sorted point of
// bucket R and start[R + 1] its end.  Bucket 0 takes keys >= total and bucket
// total + 1 negative keys (points with a batch id outside the batch): they keep a
// place in the sorted arrays but belong to no cell, and no search finds them.
// A table of one int per cell turns the two binary searches per tube of the
// key-based search into two loads, and the sort by key into a counting sort.
#pragma once

#include "common.cuh"

namespace tfgpc {

// Tables above this many cells are not built (64 MB of int32): such grids take the
// radix sort and the binary searches over keys.
constexpr int64_t kMaxTableCells = int64_t(1) << 24;

// Cells a table for `max_cells` per dimension holds, 0 if it would be too large.
inline int64_t table_cells(int D, int64_t batch_size, int max_cells) {
  double c = (double)batch_size;
  for (int d = 0; d < D; ++d) c *= (double)max_cells;
  return c <= (double)kMaxTableCells ? (int64_t)c : 0;
}

// Device pointers of a built grid, as the search kernels take them.
struct CellsView {
  const int32_t* start;        // [cells + 3]
  const int32_t* num_cells;    // [D]
  const float* inv_cell;       // [D]
  const float* scaled_min;     // [batch_size, D]
  const float4* packed;        // [n] (x, y, z or 0, original index as bits), D <= 3
  const float* points;         // [n, D] sorted
  const int32_t* batch_ids;    // [n] sorted
  const int32_t* indices;      // [n] original index of sorted point
  int64_t n;
  int batch_size;
};

inline CellsView view_of(const tfgpc_cell_grid& g) {
  return CellsView{g.cell_start, g.num_cells, g.inv_cell_sizes, g.scaled_aabb_min,
                   (const float4*)g.packed, g.sorted_points, g.sorted_batch_ids,
                   g.sorted_indices, g.n, (int)g.batch_size};
}

template <int D>
__device__ __forceinline__ int total_cells(const int* nc, int batch_size) {
  int t = batch_size;
#pragma unroll
  for (int d = 0; d < D; ++d) t *= nc[d];
  return t;
}

template <int D>
__host__ __device__ constexpr int num_tubes() {
  int n = 1;
  for (int d = 0; d < D - 1; ++d) n *= 3;
  return n;
}

// Sorted points [x, y) of the tube `code` around `cell`: the cells whose leading D-1
// coordinates differ from the cell's by the code's digits minus one (most
// significant first) and whose last coordinate differs by at most one.  Tubes in
// descending code and points ascending inside a tube is ascending sorted index.
template <int D>
__device__ __forceinline__ int2 tube_points(int code, const int* cell, int batch, const int* nc,
                                            int total, const int32_t* start) {
  int base = 0, scale = 1, rem = code;
  bool ok = true;
#pragma unroll
  for (int d = D - 2; d >= 0; --d) {
    const int c = cell[d] + rem % 3 - 1;
    rem /= 3;
    ok = ok && c >= 0 && c < nc[d];
    base += c * scale;
    scale *= nc[d];
  }
  if (!ok) return make_int2(0, 0);
  base = (batch * scale + base) * nc[D - 1];
  const int hi = base + min(cell[D - 1] + 1, nc[D - 1] - 1);
  const int lo = base + max(cell[D - 1] - 1, 0);
  return make_int2(ld_global(start + (total - hi)), ld_global(start + (total - lo) + 1));
}

}  // namespace tfgpc
