// A grid built through its cell table (cells.cuh): bounding boxes and cell counts,
// keys, the counting sort by cell, the sorted copies and the tube ranges, without a
// host read in between.
//
// The chain of Grid.py:32-83 took twenty launches here when it ran as boxes, radix
// sort (a dozen of them), gathers and tube kernel, 95 us on a 4096-point batch of which
// 25 us were the sort; nothing in it moves more than a few tens of bytes per point, so
// launches and their dependencies bound it, not HBM.  Now: boxes + parameters in one
// kernel (its last block), keys + cell histogram, table scan, scatter, rank + gather +
// tubes.  The sort is stable without comparing keys: a point's place is its cell's
// start plus the number of points of the cell with a smaller index, counted over the
// cell's members; that is quadratic in the cell size like the neighbor search
// that follows, and a 27th of its work.
#include "cell_grid.cuh"

namespace tfgpc {
namespace {

constexpr int kThreads = 256;
constexpr int kBoxPer = 4;     // points per lane of the bounding-box pass

// Order-preserving map from floats to unsigned integers (-0.0 counts as 0.0).
__device__ __forceinline__ unsigned ordered(float v) {
  const unsigned b = __float_as_uint(__fadd_rn(v, 0.0f));
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// The cell counts asked for go to the report; the kernels index with the counts cut
// to max_cells, which the table and the tube array were sized for.
__device__ __forceinline__ void clip_and_report(int D, int max_cells, const int* asked,
                                                int32_t* __restrict__ used, int32_t* page) {
  int over = 0;
  for (int d = 0; d < D; ++d) {
    const int c = max(asked[d], 1);
    over |= c > max_cells;
    page[d] = c;
    used[d] = min(c, max_cells);
  }
  page[TFGPC_MAX_DIMS] = over;
  __threadfence_system();
}

// Per-cloud boxes (PointCloud.py:38-43) folded per lane, then per warp where a warp
// lies inside one cloud, then by integer atomics on order-preserving keys: lo holds
// the smallest key, hi the smallest complement, so that one memset to 0xff starts
// both (and the ticket).  The block that finishes last turns them into the boxes
// widened by 1e-9, cells per dimension = max over the clouds of ceil(size / cell), at
// least 1 (Grid.py:44-48), the scaled minima and the inverse sizes
// (custom_ops_wrapper.py:37-43); every division is the IEEE one.
template <int D>
__global__ void __launch_bounds__(kThreads)
boxes_kernel(int64_t n, const float* __restrict__ pts, const int32_t* __restrict__ batch_ids,
             int batch_size, unsigned* lo_keys, unsigned* hi_keys, unsigned* ticket,
             DimValues cell_sizes, int max_cells, float* __restrict__ aabb_min,
             float* __restrict__ aabb_max, int32_t* __restrict__ num_cells,
             float* __restrict__ scaled_min, float* __restrict__ inv_cell, int32_t* page) {
  __shared__ int cells[D];
  __shared__ bool last;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int lane = lane_id();
  const int64_t begin = warp * 32 * kBoxPer + lane;
  float lo[D], hi[D];
#pragma unroll
  for (int d = 0; d < D; ++d) { lo[d] = INFINITY; hi[d] = -INFINITY; }
  int cur = -1;
  auto flush = [&]() {
    if (cur < 0 || cur >= batch_size) return;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      atomicMin(lo_keys + (int64_t)cur * D + d, ordered(lo[d]));
      atomicMin(hi_keys + (int64_t)cur * D + d, ~ordered(hi[d]));
    }
  };
#pragma unroll
  for (int i = 0; i < kBoxPer; ++i) {
    const int64_t p = begin + i * 32;
    if (p >= n) break;
    const int b = __ldg(batch_ids + p);
    if (b != cur) {
      flush();
      cur = b;
#pragma unroll
      for (int d = 0; d < D; ++d) { lo[d] = INFINITY; hi[d] = -INFINITY; }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float v = __ldg(pts + p * D + d);
      lo[d] = fminf(lo[d], v);
      hi[d] = fmaxf(hi[d], v);
    }
  }
  const int cur0 = __shfl_sync(0xffffffffu, cur, 0);
  if (__all_sync(0xffffffffu, cur == cur0)) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    }
    if (lane == 0) flush();
  } else {
    flush();
  }
  // ---- the last block works out the grid's parameters
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) + 2u == gridDim.x;   // (starts at -1)
  if (threadIdx.x < D) cells[threadIdx.x] = 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int i = threadIdx.x; i < batch_size * D; i += kThreads) {
    const int d = i % D;
    const float cs = cell_sizes.v[d];
    const unsigned kl = __ldcg(lo_keys + i), kh = __ldcg(hi_keys + i);
    // a cloud without points has an empty box: it asks for no cells
    const float mn = __fsub_rn(kl == 0xffffffffu ? INFINITY : unordered(kl), 1e-9f);
    const float mx = __fadd_rn(kh == 0xffffffffu ? -INFINITY : unordered(~kh), 1e-9f);
    aabb_min[i] = mn;
    aabb_max[i] = mx;
    scaled_min[i] = __fdiv_rn(mn, cs);
    const float c = ceilf(__fdiv_rn(__fsub_rn(mx, mn), cs));
    if (c > 0.0f && c < 2147483000.0f) atomicMax(&cells[d], (int)c);
  }
  __syncthreads();
  if (threadIdx.x < D) inv_cell[threadIdx.x] = __fdiv_rn(1.0f, cell_sizes.v[threadIdx.x]);
  if (threadIdx.x == 0) clip_and_report(D, max_cells, cells, num_cells, page);
}

// Cell counts given by the caller (reduced over the shards of a batch).
__global__ void given_cells_kernel(int D, const int32_t* __restrict__ given, int max_cells,
                                   int32_t* __restrict__ used, int32_t* page) {
  if (threadIdx.x != 0) return;
  int asked[TFGPC_MAX_DIMS];
  for (int d = 0; d < D; ++d) asked[d] = given[d];
  clip_and_report(D, max_cells, asked, used, page);
}

__device__ __forceinline__ int bucket_of(int64_t key, int total) {
  return key >= total ? 0 : key < 0 ? total + 1 : total - (int)key;
}

// Keys, and the number of points per bucket; `arrival` is a point's number among
// those of its bucket, in no particular order.
template <int D>
__global__ void __launch_bounds__(kThreads)
keys_histogram_kernel(int64_t n, const float* __restrict__ pts,
                      const int32_t* __restrict__ batch_ids, int batch_size,
                      const float* __restrict__ smin_all, const int32_t* __restrict__ num_cells,
                      const float* __restrict__ inv_cell, int64_t* __restrict__ keys_out,
                      int32_t* counts, int32_t* __restrict__ arrival) {
  const Grid<D> g = load_grid<D>(num_cells, inv_cell);
  const int total = total_cells<D>(g.nc, batch_size);
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  const int b = __ldg(batch_ids + i);
  const int bs = min(max(b, 0), batch_size - 1);   // (the key keeps the id that was passed in)
  float p[D], smin[D];
  int cell[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    p[d] = __ldg(pts + i * D + d);
    smin[d] = __ldg(smin_all + (int64_t)bs * D + d);
  }
  cell_of<D>(p, smin, g, cell);
  const int64_t key = key_of<D>(cell, g, b);
  keys_out[i] = key;
  arrival[i] = atomicAdd(counts + bucket_of(key, total), 1);
}

template <int D>
__global__ void __launch_bounds__(kThreads)
scatter_kernel(int64_t n, const int64_t* __restrict__ keys, const int32_t* __restrict__ num_cells,
               int batch_size, const int32_t* __restrict__ start,
               const int32_t* __restrict__ arrival, int32_t* __restrict__ members) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  int nc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) nc[d] = __ldg(num_cells + d);
  const int r = bucket_of(__ldg(keys + i), total_cells<D>(nc, batch_size));
  members[__ldg(start + r) + __ldg(arrival + i)] = (int32_t)i;
}

// One thread per slot of `members`: the rank of its point inside the bucket, and the
// point's row of every sorted array; then the tube ranges, read off the table.
template <int D>
__global__ void __launch_bounds__(kThreads)
place_kernel(int64_t n, const int32_t* __restrict__ members, const int64_t* __restrict__ keys,
             const int32_t* __restrict__ num_cells, int batch_size,
             const int32_t* __restrict__ start, const float* __restrict__ pts,
             const int32_t* __restrict__ batch_ids, int32_t* __restrict__ perm,
             int64_t* __restrict__ skeys, float* __restrict__ spts, int32_t* __restrict__ sbid,
             float4* __restrict__ packed, int2* __restrict__ ds) {
  int nc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) nc[d] = __ldg(num_cells + d);
  const int total = total_cells<D>(nc, batch_size);
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i < n) {
    const int idx = __ldg(members + i);
    const int64_t key = __ldg(keys + idx);
    const int r = bucket_of(key, total);
    const int a = __ldg(start + r), e = __ldg(start + r + 1);
    int rank = 0;
#pragma unroll 4
    for (int q = a; q < e; ++q) rank += __ldg(members + q) < idx;
    const int64_t o = a + rank;
    perm[o] = idx;
    skeys[o] = key;
    sbid[o] = __ldg(batch_ids + idx);
    float p[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      p[d] = __ldg(pts + (int64_t)idx * D + d);
      spts[o * D + d] = p[d];
    }
    if (D <= 3) packed[o] = make_float4(p[0], p[1], D == 3 ? p[D - 1] : 0.0f, __int_as_float(idx));
  }
  int span = 1;
#pragma unroll
  for (int d = 2; d < D; ++d) span *= nc[d];
  const int tubes = total / span;
  for (int64_t t = i; t < tubes; t += (int64_t)gridDim.x * kThreads) {
    const int a = __ldg(start + (total - ((int)t * span + span - 1)));
    const int e = __ldg(start + (total - (int)t * span) + 1);
    ds[t] = e > a ? make_int2(a, e) : make_int2(0, 0);
  }
}

}  // namespace

CellGridWs carve_cell_grid(void* ws, int64_t n, int64_t ns, int D, int64_t batch_size,
                           int max_cells) {
  CellGridWs w;
  char* p = (char*)ws;
  auto take = [&](size_t b) { char* r = p; p += align_up(b, 256); return r; };
  const int64_t cells = table_cells(D, batch_size, max_cells) + 3;
  w.box_bytes = ((size_t)batch_size * D * 2 + 1) * 4;
  w.box_keys = (unsigned*)take(w.box_bytes);
  w.arrival = (int32_t*)take((size_t)n * 4);
  w.members = (int32_t*)take((size_t)n * 4);
  const int64_t a = scan_block_sums_elems(cells), b = scan_block_sums_elems(ns);
  w.sums = (int64_t*)take((size_t)(a > b ? a : b) * 8);
  w.total = (int64_t*)take(8);
  w.bytes = (size_t)(p - (char*)ws);
  return w;
}

int cell_grid_build(cudaStream_t st, const tfgpc_cell_grid& g, const float* points,
                    const int32_t* batch_ids, const float* cell_sizes,
                    const int32_t* num_cells_in, const CellGridWs& w, int32_t* page) {
  const int64_t n = g.n;
  const int D = g.D, B = (int)g.batch_size;
  const int64_t cells = table_cells(D, B, g.max_cells);
  DimValues cs{};
  for (int d = 0; d < D; ++d) cs.v[d] = cell_sizes[d];
  if (num_cells_in) {
    ProfScope prof(st, "grid_params");
    given_cells_kernel<<<1, 32, 0, st>>>(D, num_cells_in, g.max_cells, g.num_cells, page);
  } else {
    ProfScope prof(st, "grid_params");
    TFGPC_CUDA(cudaMemsetAsync(w.box_keys, 0xff, w.box_bytes, st));
    unsigned* lo = w.box_keys;
    unsigned* hi = lo + (size_t)B * D;
    TFGPC_DIM_SWITCH(D, boxes_kernel<kD><<<blocks_for(n, kThreads * kBoxPer), kThreads, 0, st>>>(
        n, points, batch_ids, B, lo, hi, hi + (size_t)B * D, cs, g.max_cells, g.aabb_min,
        g.aabb_max, g.num_cells, g.scaled_aabb_min, g.inv_cell_sizes, page));
  }
  TFGPC_LAUNCH_CHECK();
  const unsigned blocks = blocks_for(n, kThreads);
  {
    ProfScope prof(st, "compute_keys");
    TFGPC_CUDA(cudaMemsetAsync(g.cell_start, 0, (size_t)(cells + 3) * 4, st));
    TFGPC_DIM_SWITCH(D, keys_histogram_kernel<kD><<<blocks, kThreads, 0, st>>>(
        n, points, batch_ids, B, g.scaled_aabb_min, g.num_cells, g.inv_cell_sizes, g.keys,
        g.cell_start, w.arrival));
  }
  TFGPC_LAUNCH_CHECK();
  int rc = exclusive_scan_cells(st, g.cell_start, g.num_cells, D, B, cells + 3, w.sums);
  if (rc) return rc;
  ProfScope prof(st, "sort_cells");
  TFGPC_DIM_SWITCH(D, scatter_kernel<kD><<<blocks, kThreads, 0, st>>>(
      n, g.keys, g.num_cells, B, g.cell_start, w.arrival, w.members));
  TFGPC_LAUNCH_CHECK();
  TFGPC_DIM_SWITCH(D, place_kernel<kD><<<blocks, kThreads, 0, st>>>(
      n, w.members, g.keys, g.num_cells, B, g.cell_start, points, batch_ids, g.sorted_indices,
      g.sorted_keys, g.sorted_points, g.sorted_batch_ids, (float4*)g.packed, (int2*)g.ds));
  TFGPC_LAUNCH_CHECK();
  return TFGPC_OK;
}

}  // namespace tfgpc
