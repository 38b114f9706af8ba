// Building a grid through its cell table (cell_grid.cu).
#pragma once

#include "cells.cuh"
#include "scan.cuh"

namespace tfgpc {

struct DimValues { float v[TFGPC_MAX_DIMS]; };

// Words of the report a build and a count leave in the mapped page: [0, D) cells asked
// for, [TFGPC_MAX_DIMS] set if a count was cut, then (word kReportTotal) a 64-bit total.
constexpr int kReportTotal = TFGPC_MAX_DIMS + 2;
constexpr int kReportWords = kReportTotal + 2;

struct CellGridWs {
  unsigned* box_keys;      // [2, batch_size, D] + ticket
  size_t box_bytes;
  int32_t *arrival, *members;   // [n]
  int64_t* sums;           // tile sums of the scans
  int64_t* total;          // [1]
  int32_t* crowded;        // [1] set if a bucket holds more than a sort tile
  size_t bytes;
};

CellGridWs carve_cell_grid(void* ws, int64_t n, int64_t ns, int D, int64_t batch_size,
                           int max_cells);

// Words that a build clears along the way, for what follows it.
struct AlsoClear { uint32_t* p = nullptr; int64_t words = 0; };

// Enqueues the build; the cell counts go to words 0 .. kReportTotal of `page`.  n_dev: the number
// of points where an earlier kernel of the stream works it out (0, or more than g.n: no grid, as if
// it had too many cells); only where g.n is cell_grid_cluster_points at most: the points of the
// largest such grid that a cluster of this device builds, 0: none.
int64_t cell_grid_cluster_points(int D, int64_t batch_size, int max_cells);
int cell_grid_build(cudaStream_t st, const tfgpc_cell_grid& g, const float* points,
                    const int32_t* batch_ids, const float* cell_sizes,
                    const int32_t* num_cells_in, const CellGridWs& w, int32_t* page,
                    AlsoClear also = AlsoClear(), const int64_t* n_dev = nullptr);

// Argument check of every entry on a built grid (cell_search.cu).
int check_cell_grid(const char* op, const tfgpc_cell_grid* g);

}  // namespace tfgpc
