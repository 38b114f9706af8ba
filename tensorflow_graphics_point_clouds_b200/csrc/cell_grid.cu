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
// that follows, and a 27th of its work.  No search need follow, though, so that above
// kCrowdedBucket members they are read once per tile of slots and not once per slot:
// n points in one cell, before -> after: 65 000 1325 -> 98 us, 200 000 5430 -> 357, 500 000
// 39400 -> 1110, a million in 8 cells 16500 -> 810 (by sorted keys: 180 to 190 us for all).
//
// Up to kClusterPoints points the whole chain is ONE kernel of one thread-block cluster
// (grid_cluster_kernel): its phases meet at the cluster's hardware barrier, boxes and
// table sums are exchanged through distributed shared memory, and there is nothing to
// initialise before it.
#include <cooperative_groups.h>

#include "cell_grid.cuh"
#include "prepare.cuh"

namespace tfgpc {
namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kBoxPer = 4;     // points per lane of the bounding-box pass
// Members of a bucket above which the ranks of a tile of its slots are worked out by the
// block together (rank_in_tile).  At least a tile, so that one meets two such buckets at most.
constexpr int kCrowdedBucket = 1024;

// Order-preserving map from floats to unsigned integers (-0.0 counts as 0.0).
__device__ __forceinline__ unsigned ordered(float v) {
  const unsigned b = __float_as_uint(__fadd_rn(v, 0.0f));
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// The cell counts asked for go to the report.  A grid that asks for more than max_cells,
// which the table and the tube array were sized for, gets no cells at all: the call fails
// with the counts, and the kernels behind this one return at once (total_cells is 0).  Cut
// to max_cells, its border cells took all points beyond them, and ranks, counts and
// samples were worked out there (quadratic in the cell) to be thrown away.
__device__ __forceinline__ void clip_and_report(int D, int max_cells, const int* asked,
                                                int32_t* __restrict__ used, int32_t* page) {
  int over = 0;
  for (int d = 0; d < D; ++d) {
    const int c = max(asked[d], 1);
    over |= c > max_cells;
    page[d] = c;
    used[d] = c;
  }
  for (int d = 0; over && d < D; ++d) used[d] = 0;
  page[TFGPC_MAX_DIMS] = over;     // (read after the stream is synchronised: no fence)
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
boxes_kernel(int64_t n, const float* pts, const int32_t* batch_ids,
             int batch_size, unsigned* lo_keys, unsigned* hi_keys, unsigned* ticket,
             DimValues cell_sizes, int max_cells, float* __restrict__ aabb_min,
             float* __restrict__ aabb_max, int32_t* __restrict__ num_cells,
             float* __restrict__ scaled_min, float* __restrict__ inv_cell, int32_t* crowded,
             int32_t* page) {
  chain_enter();
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
    const int b = ld_global(batch_ids + p);
    if (b != cur) {
      flush();
      cur = b;
#pragma unroll
      for (int d = 0; d < D; ++d) { lo[d] = INFINITY; hi[d] = -INFINITY; }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float v = ld_global(pts + p * D + d);
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
  if (threadIdx.x == 0) {
    *crowded = 0;
    clip_and_report(D, max_cells, cells, num_cells, page);
  }
}

// Cell counts given by the caller (reduced over the shards of a batch).
__global__ void given_cells_kernel(int D, const int32_t* given, int max_cells,
                                   int32_t* __restrict__ used, int32_t* crowded,
                                   int32_t* page) {
  chain_enter();
  if (threadIdx.x != 0) return;
  *crowded = 0;
  int asked[TFGPC_MAX_DIMS];
  for (int d = 0; d < D; ++d) asked[d] = given[d];
  clip_and_report(D, max_cells, asked, used, page);
}

__device__ __forceinline__ int bucket_of(int64_t key, int total) {
  return key >= total ? 0 : key < 0 ? total + 1 : total - (int)key;
}

// A point's number among those of its bucket, in no particular order; a bucket of more
// than kCrowdedBucket points raises the flag.  Where more than a few lanes of a warp (`live`:
// those that are here) share a bucket it is one atomic per bucket: a million points in one
// cell would otherwise queue up at one address.
__device__ __forceinline__ int arrive(int32_t* counts, int bucket, unsigned live,
                                      int32_t* crowded) {
  const int lane = lane_id();
  const unsigned like_first =
      __ballot_sync(live, bucket == __shfl_sync(live, bucket, __ffs(live) - 1));
  if (__popc(like_first) <= 4) {
    const int at = atomicAdd(counts + bucket, 1);
    if (at >= kCrowdedBucket) __stcg(crowded, 1);
    return at;
  }
  const unsigned peers = __match_any_sync(live, bucket);
  const int leader = __ffs(peers) - 1;
  int first = 0;
  if (lane == leader) {
    first = atomicAdd(counts + bucket, __popc(peers));
    if (first + __popc(peers) > kCrowdedBucket) __stcg(crowded, 1);
  }
  return __shfl_sync(peers, first, leader) + __popc(peers & ((1u << lane) - 1u));
}

// Keys, and the number of points per bucket.
template <int D>
__global__ void __launch_bounds__(kThreads)
keys_histogram_kernel(int64_t n, const float* pts,
                      const int32_t* batch_ids, int batch_size,
                      const float* smin_all, const int32_t* num_cells,
                      const float* inv_cell, int64_t* __restrict__ keys_out,
                      int32_t* counts, int32_t* __restrict__ arrival, int32_t* crowded) {
  chain_enter();
  const Grid<D> g = load_grid<D>(num_cells, inv_cell);
  const int total = total_cells<D>(g.nc, batch_size);
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const unsigned live = __ballot_sync(0xffffffffu, i < n);
  if (i >= n || total == 0) return;
  const int b = ld_global(batch_ids + i);
  const int bs = min(max(b, 0), batch_size - 1);   // (the key keeps the id that was passed in)
  float p[D], smin[D];
  int cell[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    p[d] = ld_global(pts + i * D + d);
    smin[d] = ld_global(smin_all + (int64_t)bs * D + d);
  }
  cell_of<D>(p, smin, g, cell);
  const int64_t key = key_of<D>(cell, g, b);
  keys_out[i] = key;
  arrival[i] = arrive(counts, bucket_of(key, total), live, crowded);
}

template <int D>
__global__ void __launch_bounds__(kThreads)
scatter_kernel(int64_t n, const int64_t* keys, const int32_t* num_cells,
               int batch_size, const int32_t* start,
               const int32_t* arrival, int32_t* __restrict__ members) {
  chain_enter();
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= n) return;
  int nc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) nc[d] = ld_global(num_cells + d);
  const int total = total_cells<D>(nc, batch_size);
  if (total == 0) return;
  const int r = bucket_of(ld_global(keys + i), total);
  members[ld_global(start + r) + ld_global(arrival + i)] = (int32_t)i;
}

// Number of the members [a, e) of a bucket with an index below idx.
__device__ __forceinline__ int rank_in_bucket(const int32_t* members, int a, int e, int idx) {
  int rank = 0, q = a;
  for (; q < e && (q & 3); ++q) rank += members[q] < idx;
  for (; q + 4 <= e; q += 4) {
    const int4 m = *(const int4*)(members + q);
    rank += (m.x < idx) + (m.y < idx) + (m.z < idx) + (m.w < idx);
  }
  for (; q < e; ++q) rank += members[q] < idx;
  return rank;
}

template <int THREADS>
struct RankScratch {
  int idx[THREADS], sorted[THREADS], upto[THREADS], warp_sum[32];
  int below, first[2], last[2];
};

// rank_in_bucket for the slots of the crowded bucket [a, e) among those of the tile
// [tile0, tile0 + THREADS): the block sorts the tile's own members, reads the bucket once
// and counts, by binary search, before how many of the sorted ones each member comes.
// One read of the bucket per tile in place of one per warp.
template <int THREADS>
__device__ __forceinline__ int rank_in_crowded(RankScratch<THREADS>& s, const int32_t* members,
                                               int a, int e, int tile0, int idx) {
  const int tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
  const int lo = max(a, tile0) - tile0;
  const int count = min(e, tile0 + THREADS) - tile0 - lo;
  const bool mine = tid >= lo && tid < lo + count;
  if (mine) s.idx[tid - lo] = idx;
  s.upto[tid] = 0;
  if (tid == 0) s.below = 0;
  __syncthreads();
  int r = 0;
  if (mine) {
#pragma unroll 8
    for (int j = 0; j < count; ++j) r += s.idx[j] < idx;
    s.sorted[r] = idx;
  }
  __syncthreads();
  const int least = s.sorted[0], most = s.sorted[count - 1];
  int below = 0;
  for (int q = (a & ~3) + 4 * tid; q < e; q += 4 * THREADS) {
    const int4 m = *(const int4*)(members + q);
    const int x[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (q + k < a || q + k >= e) continue;
      if (x[k] < least) {
        ++below;
      } else if (x[k] < most) {      // it comes before the members from `from` on
        int from = 0, to = count - 1;
        while (from < to) {
          const int mid = (from + to) >> 1;
          if (s.sorted[mid] <= x[k]) from = mid + 1; else to = mid;
        }
        atomicAdd(&s.upto[from], 1);
      }
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0) atomicAdd(&s.below, below);
  __syncthreads();
  int x = s.upto[tid];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s.warp_sum[w] = x;
  __syncthreads();
  const int before = lane < w ? s.warp_sum[lane] : 0;
  s.upto[tid] = x + __reduce_add_sync(0xffffffffu, before);
  __syncthreads();
  const int rank = s.below + s.upto[mine ? r : 0];
  __syncthreads();
  return rank;
}

// Rank inside its bucket [a, e) of the member idx in slot tile0 + threadIdx.x (live: there
// is one); the whole block calls.  any: a bucket of the grid is crowded.
template <int THREADS>
__device__ __forceinline__ int rank_in_tile(RankScratch<THREADS>& s, const int32_t* members, int a,
                                            int e, int tile0, int idx, bool live, bool last,
                                            bool any) {
  static_assert(THREADS <= kCrowdedBucket, "more than two crowded buckets in a tile");
  if (!any) return live ? rank_in_bucket(members, a, e, idx) : 0;
  const bool crowded = live && e - a > kCrowdedBucket;
  int rank = live && !crowded ? rank_in_bucket(members, a, e, idx) : 0;
  if (!__syncthreads_or(crowded)) return rank;
  if (threadIdx.x == 0) { s.first[0] = a; s.first[1] = e; }
  if (last) { s.last[0] = a; s.last[1] = e; }
  __syncthreads();
  const int fa = s.first[0], fe = s.first[1], la = s.last[0], le = s.last[1];
  if (fe - fa > kCrowdedBucket) {
    const int r = rank_in_crowded<THREADS>(s, members, fa, fe, tile0, idx);
    if (crowded && a == fa) rank = r;
  }
  if (la != fa && le - la > kCrowdedBucket) {
    const int r = rank_in_crowded<THREADS>(s, members, la, le, tile0, idx);
    if (crowded && a == la) rank = r;
  }
  return rank;
}

// One thread per slot of `members`: the rank of its point inside the bucket, and the
// point's row of every sorted array; then the tube ranges, read off the table.
template <int D, int THREADS>
__global__ void __launch_bounds__(THREADS)
place_kernel(int64_t n, const int32_t* members, const int64_t* keys,
             const int32_t* num_cells, int batch_size,
             const int32_t* start, const float* pts,
             const int32_t* batch_ids, int32_t* __restrict__ perm,
             int64_t* __restrict__ skeys, float* __restrict__ spts, int32_t* __restrict__ sbid,
             float4* __restrict__ packed, int2* __restrict__ ds,
             const int32_t* crowded) {
  chain_enter();
  int nc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) nc[d] = ld_global(num_cells + d);
  const int total = total_cells<D>(nc, batch_size);
  if (total == 0) return;
  __shared__ RankScratch<THREADS> scratch;
  const int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x;
  const bool live = i < n;
  int idx = 0, a = 0, e = 0;
  int64_t key = 0;
  if (live) {
    idx = ld_global(members + i);
    key = ld_global(keys + idx);
    const int r = bucket_of(key, total);
    a = ld_global(start + r);
    e = ld_global(start + r + 1);
  }
  const int rank = rank_in_tile<THREADS>(
      scratch, members, a, e, (int)(i - threadIdx.x), idx, live,
      live && (threadIdx.x == THREADS - 1 || i == n - 1), ld_global(crowded) != 0);
  if (live) {
    const int64_t o = a + rank;
    perm[o] = idx;
    skeys[o] = key;
    sbid[o] = ld_global(batch_ids + idx);
    float p[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      p[d] = ld_global(pts + (int64_t)idx * D + d);
      spts[o * D + d] = p[d];
    }
    if (D <= 3) packed[o] = make_float4(p[0], p[1], D == 3 ? p[D - 1] : 0.0f, __int_as_float(idx));
  }
  int span = 1;
#pragma unroll
  for (int d = 2; d < D; ++d) span *= nc[d];
  const int tubes = total / span;
  for (int64_t t = i; t < tubes; t += (int64_t)gridDim.x * THREADS) {
    const int a = ld_global(start + (total - ((int)t * span + span - 1)));
    const int e = ld_global(start + (total - (int)t * span) + 1);
    ds[t] = e > a ? make_int2(a, e) : make_int2(0, 0);
  }
}

// ---- the chain in one cluster -------------------------------------------------------

constexpr int kClusterThreads = 1024;
constexpr int kClusterBoxes = 1024;        // batch size x D at most
// Where the cluster stops: its 16 SMs build a grid of 41 000 points in 20 us and the
// separate kernels in 25, and the host launches one kernel or two in place of eight
// (layer step on 4 x 1024 points 191 -> 173 us, 3-level cell averages of 5 x 9000 points
// 243 -> 197, three-level classifier 884 -> 834); the table is zeroed and scanned by
// them alone, so a large one goes to the whole GPU.  The sorted copies scatter 44 bytes
// a point: from 8192 points on they are a launch of their own (41 000 points: 13 us of
// the cluster's 33, 4.4 by themselves).
constexpr int kMaxRanks = 16;
constexpr int64_t kClusterPoints = 65536;
constexpr int64_t kClusterCells = int64_t(1) << 21;
constexpr int64_t kClusterPlacePoints = 8192;

struct ClusterBuild {
  int64_t n;
  const float* pts;
  const int32_t* batch_ids;
  int batch_size, max_cells;
  DimValues cell_sizes;
  tfgpc_cell_grid g;
  int32_t *arrival, *members, *crowded, *page;
  bool place;
  AlsoClear also;
};

template <int D>
__global__ void __launch_bounds__(kClusterThreads, 1)
grid_cluster_kernel(ClusterBuild a) {
  chain_enter();
  // [0] ordered keys of the lower corners, [1] complements of those of the upper ones
  __shared__ unsigned box[2][kClusterBoxes];
  __shared__ float smin_s[kClusterBoxes];
  __shared__ int asked[D], nc_s[D];
  __shared__ int warp_sum_s[32], block_sum_s;
  __shared__ RankScratch<kClusterThreads> scratch;
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
  const int n = (int)a.n, boxes = a.batch_size * D;
  const int stride = ranks * kClusterThreads, first = rank * kClusterThreads + tid;
  for (int64_t i = first; i < a.also.words; i += stride) a.also.p[i] = 0u;
  // ---- boxes of this block's points
  for (int i = tid; i < boxes; i += kClusterThreads) box[0][i] = box[1][i] = 0xffffffffu;
  if (tid < D) asked[tid] = 1;
  __syncthreads();
  for (int i0 = first - lane; i0 < n; i0 += stride) {
    const int i = i0 + lane;
    const bool live = i < n;
    const int b = live ? ld_global(a.batch_ids + i) : -1;
    float lo[D], hi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float v = live ? ld_global(a.pts + (int64_t)i * D + d) : 0.0f;
      // (a coordinate that is no number counts for no box)
      lo[d] = live ? fminf(INFINITY, v) : INFINITY;
      hi[d] = live ? fmaxf(-INFINITY, v) : -INFINITY;
    }
    const int b0 = __shfl_sync(0xffffffffu, b, 0);
    const bool uniform = __all_sync(0xffffffffu, b == b0 || !live);
    if (uniform) {
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
          hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
    }
    if (b >= 0 && b < a.batch_size && (!uniform || lane == 0)) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        atomicMin(&box[0][b * D + d], ordered(lo[d]));
        atomicMin(&box[1][b * D + d], ~ordered(hi[d]));
      }
    }
  }
  cluster.sync();
  // ---- parameters, by every block for itself (see boxes_kernel)
  for (int i = tid; i < boxes; i += kClusterThreads) {
    unsigned kl = 0xffffffffu, kh = 0xffffffffu;
#pragma unroll
    for (int r = 0; r < kMaxRanks; ++r) {      // (all loads in flight together)
      const unsigned* other = cluster.map_shared_rank(&box[0][0], min(r, ranks - 1));
      kl = min(kl, other[i]);
      kh = min(kh, other[kClusterBoxes + i]);
    }
    const int d = i % D;
    const float cs = a.cell_sizes.v[d];
    const float mn = __fsub_rn(kl == 0xffffffffu ? INFINITY : unordered(kl), 1e-9f);
    const float mx = __fadd_rn(kh == 0xffffffffu ? -INFINITY : unordered(~kh), 1e-9f);
    const float sm = __fdiv_rn(mn, cs);
    smin_s[i] = sm;
    if (rank == 0) {
      a.g.aabb_min[i] = mn;
      a.g.aabb_max[i] = mx;
      a.g.scaled_aabb_min[i] = sm;
    }
    const float c = ceilf(__fdiv_rn(__fsub_rn(mx, mn), cs));
    if (c > 0.0f && c < 2147483000.0f) atomicMax(&asked[d], (int)c);
  }
  __syncthreads();
  bool over = false;
#pragma unroll
  for (int d = 0; d < D; ++d) over = over || asked[d] > a.max_cells;
  if (over) {                // (the same in every block)
    if (rank == 0 && tid == 0) clip_and_report(D, a.max_cells, asked, a.g.num_cells, a.page);
    cluster.sync();          // no block leaves while others read its shared memory
    return;
  }
  if (tid < D) nc_s[tid] = asked[tid];
  __syncthreads();
  Grid<D> g;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    g.nc[d] = nc_s[d];
    g.inv[d] = __fdiv_rn(1.0f, a.cell_sizes.v[d]);
    if (rank == 0 && tid == 0) a.g.inv_cell_sizes[d] = g.inv[d];
  }
  const int total = total_cells<D>(g.nc, a.batch_size);
  int32_t* const table = a.g.cell_start;
  for (int i = first; i < total + 3; i += stride) __stcg(table + i, 0);
  if (first == 0) __stcg(a.crowded, 0);
  cluster.sync();
  // ---- keys and the number of points per bucket (see keys_histogram_kernel)
  for (int i0 = first - lane; i0 < n; i0 += stride) {
    const int i = i0 + lane;
    const unsigned live = __ballot_sync(0xffffffffu, i < n);
    if (i >= n) break;
    const int b = ld_global(a.batch_ids + i);
    const int bs = min(max(b, 0), a.batch_size - 1);
    float p[D];
    int cell[D];
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = ld_global(a.pts + (int64_t)i * D + d);
    cell_of<D>(p, smin_s + bs * D, g, cell);
    const int64_t key = key_of<D>(cell, g, b);
    __stcg((long long*)a.g.keys + i, (long long)key);
    __stcg(a.arrival + i, arrive(table, bucket_of(key, total), live, a.crowded));
  }
  cluster.sync();
  // ---- exclusive scan of the table: a stretch per block, its sum first
  const int per = (((total + 3) + ranks - 1) / ranks + 3) / 4 * 4;
  const int begin = min(rank * per, total + 3), end = min(begin + per, total + 3);
  int sum = 0;
  for (int i = begin + tid; i < end; i += kClusterThreads) sum += __ldcg(table + i);
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) warp_sum_s[w] = sum;
  __syncthreads();
  if (w == 0) {
    sum = __reduce_add_sync(0xffffffffu, warp_sum_s[lane]);
    if (lane == 0) block_sum_s = sum;
  }
  cluster.sync();
  int run = 0;
  if (lane < rank) run = *cluster.map_shared_rank(&block_sum_s, lane);
  run = __reduce_add_sync(0xffffffffu, run);
  for (int t0 = begin; t0 < end; t0 += 4 * kClusterThreads) {
    const int i = t0 + 4 * tid;
    int v[4], x = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = i + k < end ? __ldcg(table + i + k) : 0;
      x += v[k];
    }
    const int own = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) warp_sum_s[w] = x;
    __syncthreads();
    const int s = warp_sum_s[lane];
    int at = run + x - own + __reduce_add_sync(0xffffffffu, lane < w ? s : 0);
    run += __reduce_add_sync(0xffffffffu, s);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < end) __stcg(table + i + k, at);
      at += v[k];
    }
  }
  cluster.sync();
  // ---- members of the buckets, then every point's place (see place_kernel)
  for (int i = first; i < n; i += stride) {
    const int r = bucket_of(__ldcg((const long long*)a.g.keys + i), total);
    __stcg(a.members + __ldcg(table + r) + __ldcg(a.arrival + i), i);
  }
  cluster.sync();   // (also: no block leaves while others read its shared memory)
  if (rank == 0 && tid == 0) clip_and_report(D, a.max_cells, asked, a.g.num_cells, a.page);
  if (!a.place) return;
  const bool any = __ldcg(a.crowded) != 0;
  for (int tile0 = rank * kClusterThreads; tile0 < n; tile0 += stride) {
    const int i = tile0 + tid;
    const bool live = i < n;
    int idx = 0, from = 0, to = 0;
    int64_t key = 0;
    if (live) {
      idx = __ldcg(a.members + i);
      key = __ldcg((const long long*)a.g.keys + idx);
      const int r = bucket_of(key, total);
      from = __ldcg(table + r);
      to = __ldcg(table + r + 1);
    }
    const bool last = live && (tid == kClusterThreads - 1 || i == n - 1);
    const int o = from + rank_in_tile<kClusterThreads>(scratch, a.members, from, to, tile0, idx,
                                                       live, last, any);
    if (!live) break;
    a.g.sorted_indices[o] = idx;
    a.g.sorted_keys[o] = key;
    a.g.sorted_batch_ids[o] = ld_global(a.batch_ids + idx);
    float p[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      p[d] = ld_global(a.pts + (int64_t)idx * D + d);
      a.g.sorted_points[(int64_t)o * D + d] = p[d];
    }
    if (D <= 3)
      ((float4*)a.g.packed)[o] = make_float4(p[0], p[1], D == 3 ? p[D - 1] : 0.0f,
                                             __int_as_float(idx));
  }
  int span = 1;
#pragma unroll
  for (int d = 2; d < D; ++d) span *= g.nc[d];
  const int tubes = total / span;
  for (int t = first; t < tubes; t += stride) {
    const int x = __ldcg(table + (total - (t * span + span - 1)));
    const int y = __ldcg(table + (total - t * span) + 1);
    ((int2*)a.g.ds)[t] = y > x ? make_int2(x, y) : make_int2(0, 0);
  }
}

template <int D>
int launch_cluster(cudaStream_t st, const ClusterBuild& a) {
  static int ranks_of[64] = {0};     // per device (the same value whoever computes it)
  int dev = 0;
  TFGPC_CUDA(cudaGetDevice(&dev));
  int ranks = dev < 64 ? ranks_of[dev] : 0;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kClusterThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {kMaxRanks, 1, 1};
  cfg.gridDim = dim3(kMaxRanks);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (ranks == 0) {
    int fit = 0;
    if (cudaFuncSetAttribute(grid_cluster_kernel<D>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, grid_cluster_kernel<D>, &cfg) != cudaSuccess)
      fit = 0;
    cudaGetLastError();
    ranks = fit > 0 ? kMaxRanks : 8;
    if (dev < 64) ranks_of[dev] = ranks;
  }
  // a thread per point, and per 16 cells the table has room for
  const int64_t room = table_cells(D, a.batch_size, a.max_cells) / 16;
  const int64_t threads = a.n > room ? a.n : room;
  while (ranks > 1 && threads <= (int64_t)(ranks / 2) * kClusterThreads) ranks /= 2;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;    // (see launch_chained)
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3(ranks);
  at[0].val.clusterDim = {(unsigned)ranks, 1, 1};
  TFGPC_CUDA(cudaLaunchKernelEx(&cfg, grid_cluster_kernel<D>, a));
  return TFGPC_OK;
}

// A tile (a block) reads a crowded bucket once: large ones for clouds that can have cells
// of hundreds of thousands of points, small ones spread a small cloud over the SMs.
constexpr int64_t kLargeTilePoints = 131072;

template <int THREADS>
int launch_place(cudaStream_t st, const tfgpc_cell_grid& g, const float* points,
                  const int32_t* batch_ids, const CellGridWs& w) {
  TFGPC_DIM_SWITCH(g.D, TFGPC_CUDA(launch_chained(st, blocks_for(g.n, THREADS), THREADS, 0,
      place_kernel<kD, THREADS>, g.n, w.members, g.keys, g.num_cells, (int)g.batch_size,
      g.cell_start, points, batch_ids, g.sorted_indices, g.sorted_keys, g.sorted_points,
      g.sorted_batch_ids, (float4*)g.packed, (int2*)g.ds, w.crowded)));
  return TFGPC_OK;
}

int place(cudaStream_t st, const tfgpc_cell_grid& g, const float* points, const int32_t* batch_ids,
          const CellGridWs& w) {
  return g.n >= kLargeTilePoints ? launch_place<512>(st, g, points, batch_ids, w)
                                 : launch_place<256>(st, g, points, batch_ids, w);
}

}  // namespace

CellGridWs carve_cell_grid(void* ws, int64_t n, int64_t ns, int D, int64_t batch_size,
                           int max_cells) {
  CellGridWs w;
  char* p = (char*)align_up((size_t)ws, 256);
  auto take = [&](size_t b) { char* r = p; p += align_up(b, 256); return r; };
  const int64_t cells = table_cells(D, batch_size, max_cells) + 3;
  w.box_bytes = ((size_t)batch_size * D * 2 + 1) * 4;
  w.box_keys = (unsigned*)take(w.box_bytes);
  w.arrival = (int32_t*)take((size_t)n * 4);
  w.members = (int32_t*)take((size_t)n * 4);
  const int64_t a = scan_block_sums_elems(cells), b = scan_block_sums_elems(ns);
  w.sums = (int64_t*)take((size_t)(a > b ? a : b) * 8);
  w.total = (int64_t*)take(8);
  w.crowded = (int32_t*)take(4);
  w.bytes = (size_t)(p - (char*)align_up((size_t)ws, 256));
  return w;
}

int cell_grid_build(cudaStream_t st, const tfgpc_cell_grid& g, const float* points,
                    const int32_t* batch_ids, const float* cell_sizes,
                    const int32_t* num_cells_in, const CellGridWs& w, int32_t* page,
                    AlsoClear also) {
  const int64_t n = g.n;
  const int D = g.D, B = (int)g.batch_size;
  const int64_t cells = table_cells(D, B, g.max_cells);
  DimValues cs{};
  for (int d = 0; d < D; ++d) cs.v[d] = cell_sizes[d];
  const unsigned blocks = blocks_for(n, kThreads);
  if (!num_cells_in && n <= kClusterPoints && cells <= kClusterCells &&
      (int64_t)B * D <= kClusterBoxes) {
    ProfScope prof(st, "grid_cluster");
    const ClusterBuild a{n, points, batch_ids, B, g.max_cells, cs, g, w.arrival, w.members,
                         w.crowded, page, n <= kClusterPlacePoints, also};
    int rc = TFGPC_OK;
    TFGPC_DIM_SWITCH(D, rc = launch_cluster<kD>(st, a));
    if (rc) return rc;
    return a.place ? TFGPC_OK : place(st, g, points, batch_ids, w);
  }
  if (num_cells_in) {
    ProfScope prof(st, "grid_params");
    TFGPC_CUDA(launch_chained(st, 1, 32, 0, given_cells_kernel, D, num_cells_in, g.max_cells,
        g.num_cells, w.crowded, page));
  } else {
    ProfScope prof(st, "grid_params");
    TFGPC_CUDA(cudaMemsetAsync(w.box_keys, 0xff, w.box_bytes, st));
    unsigned* lo = w.box_keys;
    unsigned* hi = lo + (size_t)B * D;
    TFGPC_DIM_SWITCH(D, TFGPC_CUDA(launch_chained(st, blocks_for(n, kThreads * kBoxPer), kThreads,
        0, boxes_kernel<kD>, n, points, batch_ids, B, lo, hi, hi + (size_t)B * D, cs, g.max_cells,
        g.aabb_min, g.aabb_max, g.num_cells, g.scaled_aabb_min, g.inv_cell_sizes, w.crowded,
        page)));
  }
  {
    ProfScope prof(st, "compute_keys");
    Prepare jobs;
    jobs.zero(g.cell_start, (size_t)(cells + 3) * 4);
    jobs.zero(also.p, (size_t)also.words * 4);
    int rc = prepare(st, jobs);
    if (rc) return rc;
    TFGPC_DIM_SWITCH(D, TFGPC_CUDA(launch_chained(st, blocks, kThreads, 0,
        keys_histogram_kernel<kD>, n, points, batch_ids, B, g.scaled_aabb_min, g.num_cells,
        g.inv_cell_sizes, g.keys, g.cell_start, w.arrival, w.crowded)));
  }
  int rc = exclusive_scan_cells(st, g.cell_start, g.num_cells, D, B, cells + 3, w.sums);
  if (rc) return rc;
  ProfScope prof(st, "sort_cells");
  TFGPC_DIM_SWITCH(D, TFGPC_CUDA(launch_chained(st, blocks, kThreads, 0, scatter_kernel<kD>, n,
      g.keys, g.num_cells, B, g.cell_start, w.arrival, w.members)));
  return place(st, g, points, batch_ids, w);
}

}  // namespace tfgpc
