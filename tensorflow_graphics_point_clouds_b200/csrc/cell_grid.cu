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

// Loads under predicates: those of a thread's points are under way together, and what is not there
// costs an issue slot.
__device__ __forceinline__ int load_if(const int32_t* p, bool ok, int otherwise) {
  int v = otherwise;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.cg.s32 %0, [%1];}"
               : "+r"(v) : "l"(p), "r"((unsigned)ok) : "memory");
  return v;
}
__device__ __forceinline__ float load_if(const float* p, bool ok) {
  float v = 0.0f;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; @q ld.global.f32 %0, [%1];}"
               : "+f"(v) : "l"(p), "r"((unsigned)ok) : "memory");
  return v;
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
  __shared__ int cells[D], warp_cloud[kThreads / 32];
  __shared__ float warp_lo[kThreads / 32][D], warp_hi[kThreads / 32][D];
  __shared__ bool last;
  const int64_t warp = ((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
  const int lane = lane_id(), w = threadIdx.x >> 5;
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
  // (all points' loads under way together, not one after the other point's id)
  int cloud[kBoxPer];
  float v[kBoxPer][D];
#pragma unroll
  for (int i = 0; i < kBoxPer; ++i) {
    const int64_t p = begin + i * 32;
    cloud[i] = load_if(batch_ids + p, p < n, -1);
#pragma unroll
    for (int d = 0; d < D; ++d) v[i][d] = load_if(pts + p * D + d, p < n);
  }
#pragma unroll
  for (int i = 0; i < kBoxPer; ++i) {
    if (begin + i * 32 >= n) break;
    if (cloud[i] != cur) {
      flush();
      cur = cloud[i];
#pragma unroll
      for (int d = 0; d < D; ++d) { lo[d] = INFINITY; hi[d] = -INFINITY; }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      lo[d] = fminf(lo[d], v[i][d]);
      hi[d] = fmaxf(hi[d], v[i][d]);
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
    if (lane == 0) {
      warp_cloud[w] = cur;
#pragma unroll
      for (int d = 0; d < D; ++d) { warp_lo[w][d] = lo[d]; warp_hi[w][d] = hi[d]; }
    }
  } else {
    flush();
    if (lane == 0) warp_cloud[w] = -1;
  }
  // The block's warps mostly lie in one cloud too: one atomic of theirs where each had one (the
  // atomics of all blocks meet on a few hundred bytes and wait for each other: 800 000 points
  // of 8 clouds 30 -> 9 us, 530 000 of 16 17 -> 9, 131 000 of 16 9 -> 7; with a look at the box
  // before the atomics, which meets them there, 51).
  __syncthreads();
  if (w == 0) {
    cur = lane < kThreads / 32 ? warp_cloud[lane] : -1;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      lo[d] = cur >= 0 ? warp_lo[lane & (kThreads / 32 - 1)][d] : INFINITY;
      hi[d] = cur >= 0 ? warp_hi[lane & (kThreads / 32 - 1)][d] : -INFINITY;
    }
    const int most = __reduce_max_sync(0xffffffffu, cur);
    if (__all_sync(0xffffffffu, cur == most || cur < 0)) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int o = kThreads / 64; o > 0; o >>= 1) {
          lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
          hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
      }
      cur = lane == 0 ? most : -1;
    }
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

// Points up to which the cluster writes the sorted copies itself (see ClusterBuild).
constexpr int64_t kClusterPlacePoints = 8192;

// One thread per slot of `members`: the rank of its point inside the bucket, and the
// point's row of every sorted array; then the tube ranges, read off the table.
template <int D, int THREADS>
__global__ void __launch_bounds__(THREADS)
place_kernel(int64_t n, const int64_t* n_dev, const int32_t* members, const int64_t* keys,
             const int32_t* num_cells, int batch_size,
             const int32_t* start, const float* pts,
             const int32_t* batch_ids, int32_t* __restrict__ perm,
             int64_t* __restrict__ skeys, float* __restrict__ spts, int32_t* __restrict__ sbid,
             float4* __restrict__ packed, int2* __restrict__ ds,
             const int32_t* crowded) {
  chain_enter();
  if (n_dev) {
    const int64_t most = n;
    n = ld_global(n_dev);
    if (n <= kClusterPlacePoints || n > most) return;     // (placed by the cluster, or no grid)
  }
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
// It is bound by its barriers (900 to 1900 cycles each) and, between them, by single trips
// to L2 and by instructions that are not in the cache yet: 11 us for 4096 points.  Hence each
// trip is made once, for all points of a thread together: points are read for the boxes and
// kept until the cell is known, bucket and number until the place is; a warp takes neighboring
// points and folds their box in registers; the scan keeps what it summed up, without a barrier
// of the block per 4096 cells; sums go to the other blocks before a barrier instead of being
// fetched after it.  us before -> now, kernel: 42 000 points in 7300 cells 23 -> 19, 38 000 in
// 226 000 28 -> 18; 3-level cell averages of 5 x 9000 points 171 -> 158, three-level classifier
// 668 -> 639 (its runs differ by up to 15 %), layer step on 59 000 points 208 -> 203.  Left: the atomics of 16 SMs (7300 cycles
// for 59 000 points, about two per atomic of an SM).
constexpr int kMaxRanks = 16;
constexpr int kHeld = 4;                   // points of a thread at most
constexpr int64_t kClusterPoints = 65536;
constexpr int64_t kClusterCells = int64_t(1) << 21;

struct ClusterBuild {
  int64_t n;                   // points, or (n_dev) at most so many
  const int64_t* n_dev;        // their number where the host does not know it; 0, or more: no grid
  const float* pts;
  const int32_t* batch_ids;
  int batch_size, max_cells;
  DimValues cell_sizes;
  tfgpc_cell_grid g;
  int32_t *members, *crowded, *page;
  bool place;
  AlsoClear also;
};

// The atomic under a predicate, as load_if.
__device__ __forceinline__ int count_if(int32_t* p, bool ok) {
  int v = 0;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %2, 0; @q atom.global.add.s32 %0, [%1], 1;}"
               : "+r"(v) : "l"(p), "r"((unsigned)ok) : "memory");
  return v;
}
// table[at .. at + 4), zeros from `end` on; wide: the table begins at a multiple of 16 bytes.
__device__ __forceinline__ int4 load_four(const int32_t* table, int at, int end, bool wide) {
  int4 v = make_int4(0, 0, 0, 0);
  const bool all = wide && at + 4 <= end;
  asm volatile("{.reg .pred q; setp.ne.u32 q, %5, 0; @q ld.global.cg.v4.s32 {%0, %1, %2, %3}, [%4];}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "l"(table + at), "r"((unsigned)all) : "memory");
  v.x = load_if(table + at, !all && at < end, v.x);
  v.y = load_if(table + at + 1, !all && at + 1 < end, v.y);
  v.z = load_if(table + at + 2, !all && at + 2 < end, v.z);
  v.w = load_if(table + at + 3, !all && at + 3 < end, v.w);
  return v;
}
__device__ __forceinline__ void store_four(int32_t* table, int at, int end, bool wide, int4 v) {
  if (wide && at + 4 <= end) {
    __stcg((int4*)(table + at), v);
    return;
  }
  if (at < end) __stcg(table + at, v.x);
  if (at + 1 < end) __stcg(table + at + 1, v.y);
  if (at + 2 < end) __stcg(table + at + 2, v.z);
  if (at + 3 < end) __stcg(table + at + 3, v.w);
}

// A thread holds its points (kHeld at most) from the boxes to their places: coordinates until
// the cell is known, then bucket and number in it.
template <int D>
__global__ void __launch_bounds__(kClusterThreads, 1)
grid_cluster_kernel(ClusterBuild a) {
  chain_enter();
  // [0] ordered keys of the lower corners, [1] complements of those of the upper ones
  __shared__ unsigned box[2][kClusterBoxes];
  __shared__ float smin_s[kClusterBoxes], inv_s[D];
  __shared__ int asked[D];
  __shared__ int warp_sum_s[32], block_sum_s[kMaxRanks];     // (of every block)
  __shared__ RankScratch<kClusterThreads> scratch;
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
  const int64_t points = a.n_dev ? ld_global(a.n_dev) : a.n;
  const int n = points <= a.n ? (int)points : 0, boxes = a.batch_size * D;
  const int stride = ranks * kClusterThreads, first = rank * kClusterThreads + tid;
  // A warp's points follow one another, as they mostly lie in one cloud.
  const int steps = (n + stride - 1) / stride;
  const int mine = (w * ranks + rank) * 32 * steps + lane;
  const int here = (min(n - mine, 32 * steps) + 31) >> 5;    // this lane's points (or none: <= 0)
  float p[kHeld][D];
  int cloud[kHeld];
#pragma unroll
  for (int k = 0; k < kHeld; ++k) {
    const bool live = k < here;
    cloud[k] = load_if(a.batch_ids + (mine + 32 * k), live, -1);
#pragma unroll
    for (int d = 0; d < D; ++d) p[k][d] = load_if(a.pts + (int64_t)(mine + 32 * k) * D + d, live);
  }
  for (int64_t i = first; i < a.also.words; i += stride) a.also.p[i] = 0u;
  // ---- boxes of this block's points
  for (int i = tid; i < boxes; i += kClusterThreads) box[0][i] = box[1][i] = 0xffffffffu;
  if (tid < D) asked[tid] = 1;
  __syncthreads();
  // (the lanes' least keys; `uniform`: all of them of cloud b, the same in every lane)
  auto fold = [&](const float* lo, const float* hi, int b, bool live, bool uniform) {
    unsigned kl[D], kh[D];
#pragma unroll
    for (int d = 0; d < D; ++d) { kl[d] = ordered(lo[d]); kh[d] = ~ordered(hi[d]); }
    if (uniform) {
      unsigned least = 0xffffffffu;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const unsigned l = __reduce_min_sync(0xffffffffu, kl[d]);
        const unsigned h = __reduce_min_sync(0xffffffffu, kh[d]);
        if (lane == d) least = l;
        if (lane == D + d) least = h;
      }
      if (lane < 2 * D && b >= 0 && b < a.batch_size)
        atomicMin(&box[lane >= D][b * D + lane - (lane >= D ? D : 0)], least);
    } else if (live && b >= 0 && b < a.batch_size) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        atomicMin(&box[0][b * D + d], kl[d]);
        atomicMin(&box[1][b * D + d], kh[d]);
      }
    }
  };
  {
    const int b0 = __shfl_sync(0xffffffffu, cloud[0], 0);
    bool same = true;
#pragma unroll
    for (int k = 0; k < kHeld; ++k) same = same && (k >= here || cloud[k] == b0);
    if (__all_sync(0xffffffffu, same)) {
      float lo[D], hi[D];
#pragma unroll
      for (int d = 0; d < D; ++d) { lo[d] = INFINITY; hi[d] = -INFINITY; }
#pragma unroll
      for (int k = 0; k < kHeld; ++k)
#pragma unroll
        for (int d = 0; d < D; ++d) {
          // (a coordinate that is no number counts for no box)
          lo[d] = k < here ? fminf(lo[d], p[k][d]) : lo[d];
          hi[d] = k < here ? fmaxf(hi[d], p[k][d]) : hi[d];
        }
      fold(lo, hi, b0, false, true);
    } else {
#pragma unroll 1
      for (int k = 0; k < steps; ++k) {
        const bool live = k < here;
        int b = cloud[0];
        float lo[D], hi[D];
#pragma unroll
        for (int d = 0; d < D; ++d) lo[d] = p[0][d];
#pragma unroll
        for (int q = 1; q < kHeld; ++q) {
          b = k == q ? cloud[q] : b;
#pragma unroll
          for (int d = 0; d < D; ++d) lo[d] = k == q ? p[q][d] : lo[d];
        }
#pragma unroll
        for (int d = 0; d < D; ++d) {
          hi[d] = live ? fmaxf(-INFINITY, lo[d]) : -INFINITY;
          lo[d] = live ? fminf(INFINITY, lo[d]) : INFINITY;
        }
        // (a lane without a point writes a value too where all of them lie in one cloud)
        const int first_b = __shfl_sync(0xffffffffu, b, 0);
        const bool uniform = __all_sync(0xffffffffu, b == first_b || !live);
        fold(lo, hi, uniform ? first_b : b, live, uniform);
      }
    }
  }
  cluster.sync();
  // ---- parameters, by every block for itself (see boxes_kernel)
  // (each of the `ranks` blocks, a power of two, is read by a warp or several; that others read
  // this one's boxes meanwhile, some of them lowered already, changes no minimum)
  if (w % ranks != rank) {
    const unsigned* other = cluster.map_shared_rank(&box[0][0], w % ranks);
    for (int i = w / ranks * 32 + lane; i < boxes; i += max(32 / ranks, 1) * 32) {
      const unsigned kl = ld_global(other + i), kh = ld_global(other + kClusterBoxes + i);
      atomicMin(&box[0][i], kl);
      atomicMin(&box[1][i], kh);
    }
  }
  if (w == 31 && lane < D) {
    inv_s[lane] = __fdiv_rn(1.0f, a.cell_sizes.v[lane]);
    if (rank == 0) a.g.inv_cell_sizes[lane] = inv_s[lane];
  }
  __syncthreads();
  // (two threads per box, so that their divisions are one piece of code: instructions that are
  // not in the cache yet cost more here than the work)
  for (int x = tid; x < 2 * boxes; x += kClusterThreads) {
    const int i = x >> 1, d = i % D;
    const unsigned kl = box[0][i], kh = box[1][i];
    const float mn = __fsub_rn(kl == 0xffffffffu ? INFINITY : unordered(kl), 1e-9f);
    const float mx = __fadd_rn(kh == 0xffffffffu ? -INFINITY : unordered(~kh), 1e-9f);
    const float q = __fdiv_rn(x & 1 ? __fsub_rn(mx, mn) : mn, a.cell_sizes.v[d]);
    if (x & 1) {
      const float c = ceilf(q);
      if (c > 0.0f && c < 2147483000.0f) atomicMax(&asked[d], (int)c);
    } else {
      smin_s[i] = q;
      if (rank == 0) {
        a.g.aabb_min[i] = mn;
        a.g.aabb_max[i] = mx;
        a.g.scaled_aabb_min[i] = q;
      }
    }
  }
  __syncthreads();
  bool over = n == 0;          // (what it would be a grid of has failed, or does not fit)
  if (over && tid < D) asked[tid] = a.max_cells + 1;
  __syncthreads();
  Grid<D> g;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    g.nc[d] = asked[d];
    g.inv[d] = inv_s[d];
    over = over || g.nc[d] > a.max_cells;
  }
  if (over) {                // (the same in every block)
    if (rank == 0 && tid == 0) clip_and_report(D, a.max_cells, asked, a.g.num_cells, a.page);
    cluster.sync();          // no block leaves while others read its shared memory
    return;
  }
  const int total = total_cells<D>(g.nc, a.batch_size);
  int32_t* const table = a.g.cell_start;
  const bool wide = ((uintptr_t)table & 15) == 0;
  for (int i = 4 * first; i < total + 3; i += 4 * stride)
    store_four(table, i, total + 3, wide, make_int4(0, 0, 0, 0));
  if (first == 0) __stcg(a.crowded, 0);
  cluster.sync();
  // ---- keys and the number of points per bucket (see keys_histogram_kernel and arrive)
  int bucket[kHeld], number[kHeld];
  bool apart = true;
#pragma unroll
  for (int k = 0; k < kHeld; ++k) {
    bucket[k] = number[k] = 0;
    if (k >= steps) continue;
    const bool live = k < here;
    if (live) {
      int cell[D];
      cell_of<D>(p[k], smin_s + min(max(cloud[k], 0), a.batch_size - 1) * D, g, cell);
      const int64_t key = key_of<D>(cell, g, cloud[k]);
      __stcg((long long*)a.g.keys + mine + 32 * k, (long long)key);
      bucket[k] = bucket_of(key, total);
    }
    const int b0 = __shfl_sync(0xffffffffu, bucket[k], 0);
    apart = apart && __popc(__ballot_sync(0xffffffffu, live && bucket[k] == b0)) <= 4;
  }
  if (apart) {
    int most = 0;
#pragma unroll
    for (int k = 0; k < kHeld; ++k) number[k] = count_if(table + bucket[k], k < here);
#pragma unroll
    for (int k = 0; k < kHeld; ++k) most = max(most, number[k]);
    if (most >= kCrowdedBucket) __stcg(a.crowded, 1);
  } else {
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      const unsigned live = __ballot_sync(0xffffffffu, k < here);
      if (k < here) number[k] = arrive(table, bucket[k], live, a.crowded);
    }
  }
  cluster.sync();
  // ---- exclusive scan of the table: a stretch per block and of it one per warp, the sums first
  const int per = (((total + 3) + ranks - 1) / ranks + 3) / 4 * 4;
  const int per_warp = ((per + 31) / 32 + 127) / 128 * 128;
  const int block_end = min((rank + 1) * per, total + 3);
  const int begin = rank * per + w * per_warp, end = min(begin + per_warp, block_end);
  int4 v[kHeld];          // the warp's first pieces of 128
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kHeld; ++k) v[k] = load_four(table, begin + 128 * k + 4 * lane, end, wide);
#pragma unroll
  for (int k = 0; k < kHeld; ++k) sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
  for (int i = begin + 128 * kHeld + 4 * lane; i < end; i += 128) {
    const int4 x = load_four(table, i, end, wide);
    sum += (x.x + x.y) + (x.z + x.w);
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) warp_sum_s[w] = sum;
  __syncthreads();
  if (w == 0) {
    sum = __reduce_add_sync(0xffffffffu, warp_sum_s[lane]);
    if (lane < ranks) *cluster.map_shared_rank(&block_sum_s[rank], lane) = sum;
  }
  cluster.sync();
  int run = __reduce_add_sync(0xffffffffu, (lane < rank ? block_sum_s[lane & (kMaxRanks - 1)] : 0) +
                                               (lane < w ? warp_sum_s[lane] : 0));
  auto scan_piece = [&](int at, int4 x) {
    const int own = (x.x + x.y) + (x.z + x.w);
    int y = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    const int s = run + y - own;
    store_four(table, at, end, wide, make_int4(s, s + x.x, s + x.x + x.y, s + x.x + x.y + x.z));
    run += __shfl_sync(0xffffffffu, y, 31);
  };
#pragma unroll
  for (int k = 0; k < kHeld; ++k)
    if (begin + 128 * k < end) scan_piece(begin + 128 * k + 4 * lane, v[k]);
  for (int i = begin + 128 * kHeld; i < end; i += 128)
    scan_piece(i + 4 * lane, load_four(table, i + 4 * lane, end, wide));
  cluster.sync();
  // ---- members of the buckets, then every point's place (see place_kernel)
#pragma unroll
  for (int k = 0; k < kHeld; ++k) number[k] += load_if(table + bucket[k], k < here, 0);
#pragma unroll
  for (int k = 0; k < kHeld; ++k)
    if (k < here) __stcg(a.members + number[k], mine + 32 * k);
  cluster.sync();   // (also: no block leaves while others read its shared memory)
  if (rank == 0 && tid == 0) clip_and_report(D, a.max_cells, asked, a.g.num_cells, a.page);
  if (a.n_dev ? n > kClusterPlacePoints : !a.place) return;
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

// Blocks of the largest cluster the device takes.
template <int D>
int cluster_ranks(int* most) {
  static int ranks_of[64] = {0};     // per device (the same value whoever computes it)
  int dev = 0;
  TFGPC_CUDA(cudaGetDevice(&dev));
  int ranks = dev < 64 ? ranks_of[dev] : 0;
  if (ranks == 0) {
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kClusterThreads);
    cfg.gridDim = dim3(kMaxRanks);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim = {kMaxRanks, 1, 1};
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaFuncSetAttribute(grid_cluster_kernel<D>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, grid_cluster_kernel<D>, &cfg) != cudaSuccess)
      fit = 0;
    cudaGetLastError();
    ranks = fit > 0 ? kMaxRanks : 8;
    if (dev < 64) ranks_of[dev] = ranks;
  }
  *most = ranks;
  return TFGPC_OK;
}

template <int D>
int launch_cluster(cudaStream_t st, const ClusterBuild& a, int ranks) {
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(kClusterThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  cfg.attrs = at;
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
                  const int32_t* batch_ids, const CellGridWs& w, const int64_t* n_dev) {
  TFGPC_DIM_SWITCH(g.D, TFGPC_CUDA(launch_chained(st, blocks_for(g.n, THREADS), THREADS, 0,
      place_kernel<kD, THREADS>, g.n, n_dev, w.members, g.keys, g.num_cells, (int)g.batch_size,
      g.cell_start, points, batch_ids, g.sorted_indices, g.sorted_keys, g.sorted_points,
      g.sorted_batch_ids, (float4*)g.packed, (int2*)g.ds, w.crowded)));
  return TFGPC_OK;
}

int place(cudaStream_t st, const tfgpc_cell_grid& g, const float* points, const int32_t* batch_ids,
          const CellGridWs& w, const int64_t* n_dev = nullptr) {
  return g.n >= kLargeTilePoints ? launch_place<512>(st, g, points, batch_ids, w, n_dev)
                                 : launch_place<256>(st, g, points, batch_ids, w, n_dev);
}

// Blocks of the cluster that a grid of so many points can be built by, 0: it is too large for one.
int cluster_for(int D, int64_t n, int64_t batch_size, int max_cells, int* ranks) {
  *ranks = 0;
  const int64_t cells = table_cells(D, batch_size, max_cells);
  if (n > kClusterPoints || cells <= 0 || cells > kClusterCells || batch_size * D > kClusterBoxes)
    return TFGPC_OK;
  int rc = TFGPC_OK;
  TFGPC_DIM_SWITCH(D, rc = cluster_ranks<kD>(ranks));
  if (!rc && n > (int64_t)*ranks * kClusterThreads * kHeld) *ranks = 0;
  return rc;
}

// Arrays of words, one after the other, kCopyWords to a thread.
constexpr int kCopies = 13, kCopyWords = 8;
struct Copies {
  const uint32_t* from[kCopies];
  uint32_t* to[kCopies];
  int64_t words[kCopies];
  int first_block[kCopies + 1];
};
__global__ void __launch_bounds__(kThreads) copy_kernel(const __grid_constant__ Copies a) {
  int i = 0;
  while ((int)blockIdx.x >= a.first_block[i + 1]) ++i;
  const int64_t w0 = (int64_t)((int)blockIdx.x - a.first_block[i]) * (kThreads * kCopyWords);
#pragma unroll
  for (int u = 0; u < kCopyWords; ++u) {
    const int64_t w = w0 + u * kThreads + (int)threadIdx.x;
    if (w < a.words[i]) a.to[i][w] = a.from[i][w];
  }
}

}  // namespace

int64_t cell_grid_cluster_points(int D, int64_t batch_size, int max_cells) {
  int ranks = 0;
  if (cluster_for(D, 1, batch_size, max_cells, &ranks)) return 0;
  const int64_t held = (int64_t)ranks * kClusterThreads * kHeld;
  return held < kClusterPoints ? held : kClusterPoints;
}

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
                    AlsoClear also, const int64_t* n_dev) {
  const int64_t n = g.n;
  const int D = g.D, B = (int)g.batch_size;
  const int64_t cells = table_cells(D, B, g.max_cells);
  DimValues cs{};
  for (int d = 0; d < D; ++d) cs.v[d] = cell_sizes[d];
  const unsigned blocks = blocks_for(n, kThreads);
  int ranks = 0;
  if (!num_cells_in) {
    int rc = cluster_for(D, n, B, g.max_cells, &ranks);
    if (rc) return rc;
  }
  TFGPC_REQUIRE(!n_dev || ranks > 0, "a grid of points not counted yet is too large for a cluster");
  if (ranks > 0) {
    ProfScope prof(st, "grid_cluster");
    const ClusterBuild a{n, n_dev, points, batch_ids, B, g.max_cells, cs, g, w.members, w.crowded,
                         page, n <= kClusterPlacePoints, also};
    int rc = TFGPC_OK;
    TFGPC_DIM_SWITCH(D, rc = launch_cluster<kD>(st, a, ranks));
    if (rc) return rc;
    return a.place ? TFGPC_OK : place(st, g, points, batch_ids, w, n_dev);
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

// Arrays that were made for more points than came are held for as long as the grid: a level of a
// hierarchy whose number of points nobody knew kept up to 13 MB.  One launch of 4 to 8 us.
extern "C" int tfgpc_cell_grid_copy(void* stream, const tfgpc_cell_grid* from,
                                    const tfgpc_cell_grid* to) {
  using namespace tfgpc;
  int rc = check_cell_grid("CellGridCopy", from);
  if (!rc) rc = check_cell_grid("CellGridCopy", to);
  if (rc) return rc;
  TFGPC_REQUIRE(from->D == to->D && from->n == to->n && from->batch_size == to->batch_size &&
                to->max_cells <= from->max_cells,
                "CellGridCopy expects grids of as many points and clouds, into no larger a table");
  const int64_t n = to->n, D = to->D, b = to->batch_size;
  const int64_t words[kCopies] = {b * D, b * D, D, b * D, D, 2 * n, n, 2 * n, n * D, n,
                                  D <= 3 ? 4 * n : 0,
                                  (int64_t)tfgpc_cell_table_elems(to->D, b, to->max_cells),
                                  2 * b * (int64_t)to->max_cells * to->max_cells};
  const void* const* src = (const void* const*)&from->aabb_min;
  void* const* dst = (void* const*)&to->aabb_min;
  Copies a;
  int64_t blocks = 0;
  for (int i = 0; i < kCopies; ++i) {
    a.from[i] = (const uint32_t*)src[i];
    a.to[i] = (uint32_t*)dst[i];
    a.words[i] = words[i];
    a.first_block[i] = (int)blocks;
    blocks += (words[i] + kThreads * kCopyWords - 1) / (kThreads * kCopyWords);
  }
  a.first_block[kCopies] = (int)blocks;
  ProfScope prof((cudaStream_t)stream, "grid_copy");
  copy_kernel<<<(unsigned)blocks, kThreads, 0, (cudaStream_t)stream>>>(a);
  TFGPC_CUDA(cudaGetLastError());
  return TFGPC_OK;
}
