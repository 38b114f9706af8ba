// Poisson-disk and cell-average sampling straight from the cell table of a grid.
//
// Poisson disk (count_sampling_pd_kernels.cu.cc:42-108, 157-180): 2^D passes, pass p
// takes the cells whose coordinate d has parity bit d of p; inside a cell the points
// are visited in sorted order and a point is taken iff none of its neighbors is.  A
// taken point marks the points within the radius itself (the relation is symmetric),
// so no neighbor list is needed: on 8 clouds of 100 000 Gaussian-mixture points
// searching and writing the lists of four levels took 3.2 ms, the passes over them 0.6.
// The passes and the compaction of the taken points in ascending index are one
// cooperative launch; what bounds it is the marking of crowded cells.  Levels of up to 65 536
// points are first tried without passes, whose chain bounds them (settle_kernel).  Only cells of
// later passes are marked (13 of 26 neighbors on average).  Clouds do not meet, so each has a team
// of blocks, in proportion to its points, with barriers of its own.
//
// Cell average (sampling_avg_kernels.cu.cc:43-88): one thread per occupied cell,
// sequential fp32 sum of its points / count, cells in ascending first index (a warp per cell
// of many points: kLongCell).
#include "cell_grid.cuh"
#include "grid_barrier.cuh"

namespace tfgpc {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxBlocks = 1024;
constexpr int kMaxTeams = kMaxBlocks / 2;
// Cells of more points than this are left to the end of a block's pass, for all its
// warps together: one warp with a cell of a thousand points, and a few thousand to
// mark, keeps its whole team waiting.  us of this kernel at 48, 96, 160, 256 and 512: first of four
// levels of 8 x 100 000 Gaussian-mixture points 201, 203, 209, 210, 251; 70 000 points in 400
// clumps 73, 63, 61, 61, 61; 400 000 in 40 clumps 182, 229, 238, 254, 336; no cell that full: the same.
constexpr int kCrowded = 96;
constexpr int kMaxCrowded = 128;
constexpr int kHeadWords = 8;             // before the teams' counters
constexpr size_t kHeadBytes = (size_t)(kMaxTeams + kHeadWords) * 4;   // before the states
// Levels of up to this many points are first tried without passes (settle_kernel).
constexpr int64_t kFlowPoints = 65536;
constexpr int kFlowPer = 128;             // points of a block
constexpr int kFlowLists = 32;            // words of neighbors of a point
constexpr int kFlowCell = 256;            // points of a cell
// Candidates (points of earlier passes in the cells around a point, and before it in its own) that a
// level has on average, times the points of eight lanes, above which its passes are the faster
// ones.  Settling takes as long as its tests, the passes about as long with few candidates as with
// many.  us of a hierarchy of one level of four clouds, settled / by passes: 30 000 points in all (two
// per eight lanes) with 101, 188 and 268 candidates 93/95, 106/103 and 116/110, 60 000 (four) with 55,
// 106 and 202 107/106, 131/107 and 155/111; in two dimensions 15 000 with 149 and 296 71/69 and 80/75,
// 60 000 with 28 and 55 90/95 and 98/86; in four 30 000 with 184 129/175, 60 000 with 203 189/190.
// With more than kFlowMost candidates some lists run over: 15 000 points with 332 and 467 100/105
// and 199/123.  Not so in levels of kFlowFew points, whose blocks each decide: 2000 points with 249
// 80/103.
constexpr int kFlowMost = 256, kFlowFew = 2048;
__host__ __device__ constexpr int flow_work(int D) {
  return D == 2 ? 160 : D == 3 ? 320 : 768 << (D - 4);
}
// Candidates of a mark loop between two signs of progress: well under a millisecond, and
// none at all in cells of ordinary size.  A selection shows none (its loop has no register
// left for it: spills, 1 % of a hierarchy); one over all points of a call takes some 30 ns
// a point, which the period of the barriers allows for.
constexpr int kProgressMarks = 65536;
// A cell of more points than that has its average worked out by its warp together, 32 points'
// loads at a time, added up in the same order.  (By one thread, four loads at a time, the cells of several
// hundred points decided: 5 x 9001 points, cells of 0.04, 22 -> 13 us in this kernel.)
constexpr int kLongCell = 64;
inline unsigned long long barrier_period_ns(int64_t n) { return 500000000ull + 100ull * n; }

// Blocks of the two kernels for n points: a warp per 8 points (16: 158 against 140 us in the
// three-level classifier), 8 lanes per point.
__host__ __device__ __forceinline__ int64_t blocks_wanted(int64_t n) {
  return (n + 8 * kWarps - 1) / (8 * kWarps);
}
__host__ __device__ __forceinline__ int64_t settle_blocks(int64_t n) {
  return (n + kThreads / 8 - 1) / (kThreads / 8);
}
__device__ __forceinline__ int sample_blocks(int64_t n, int grid) {
  return (int)min((int64_t)grid, blocks_wanted(n));
}

struct SampleArgs {
  CellsView c;
  const int64_t* keys;         // sorted
  int mode;                    // 0 Poisson disk, 1 cell average
  const float* inv_radii;
  uint8_t* state;              // [n] 0 open, 1 blocked, 2 taken (zero on entry)
  unsigned* arrived;           // barrier counter of the grid, error word, progress, a word unused,
                               // whether settle_kernel has failed, from kHeadWords on the teams'
                               // counters; all zero on entry
  unsigned long long* settled; // [n / 32] taken points below, settled ones above, zero on entry; null:
                               // settle_kernel does not run
  int write_blocks;            // gridDim.x of cells_sample_kernel
  int32_t* block_total;        // [gridDim.x], zero on entry where `settled` is
  float* pts_out;
  int32_t* batch_out;
  int32_t* index_out;          // original indices (Poisson)
  int32_t* page;               // number of samples (64 bits), then the error word
  const int64_t* n_dev;        // number of points (c.n: at most), or null
  int64_t* samples_dev;        // number of samples, 0 if anything failed, or null
  unsigned long long period_ns;
};

// The points of one cell that a warp has taken and not marked the neighbors of yet:
// lane k holds the k-th.
template <int D>
struct Taken {
  float p[D];
  int j;
  int count;     // the same in every lane
};

template <int D>
__device__ __forceinline__ void load_coords(const CellsView& c, int j, float* p) {
  if (D <= 3) {
    const float4 v = __ldg(c.packed + j);
    p[0] = v.x; p[1] = v.y;
    if (D == 3) p[D - 1] = v.z;
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = __ldg(c.points + (int64_t)j * D + d);
  }
}

// The distance test of the search (cell_search.cu).
template <int D>
__device__ __forceinline__ bool within(const float* s, const float* p, const float* inv_r) {
  float u = __fmul_rn(__fsub_rn(s[0], p[0]), inv_r[0]);
  float d2 = __fmul_rn(u, u);
#pragma unroll
  for (int d = 1; d < D; ++d) {
    u = __fmul_rn(__fsub_rn(s[d], p[d]), inv_r[d]);
    d2 = __fmaf_rn(u, u, d2);
  }
  return d2 < 1.0f;
}

// Sorted points [x, y) to be marked in one half of a tube around `cell`.  The pass of
// a cell is the number whose bit d is the parity of its coordinate d, so the last
// coordinate decides first: from an even one both ends of a tube are later, from an odd
// one none is; the middle is later if the leading coordinates' bits are.  A tube that
// is later as a whole is its first half alone.  own: the cell itself counts as later.
template <int D>
__device__ __forceinline__ int2 later_points(int code, const int* cell, int batch, const int* nc,
                                             int total, bool own,
                                             const int32_t* __restrict__ start) {
  int base = 0, scale = 1, rem = code >> 1, mine = 0, theirs = 0;
  bool ok = true;
#pragma unroll
  for (int d = D - 2; d >= 0; --d) {
    const int c = cell[d] + rem % 3 - 1;
    rem /= 3;
    ok = ok && c >= 0 && c < nc[d];
    base += c * scale;
    scale *= nc[d];
    mine |= (cell[d] & 1) << d;
    theirs |= (c & 1) << d;
  }
  const int z = cell[D - 1];
  const bool second = code & 1, even = (z & 1) == 0;
  const bool later = theirs > mine || (own && code >> 1 == num_tubes<D>() / 2);
  int lo, hi;
  if (later) {
    lo = even ? max(z - 1, 0) : z;
    hi = even ? min(z + 1, nc[D - 1] - 1) : z;
    ok = ok && !second;
  } else {
    lo = hi = second ? z + 1 : z - 1;
    ok = ok && even && lo >= 0 && lo < nc[D - 1];
  }
  if (!ok) return make_int2(0, 0);
  base = (batch * scale + base) * nc[D - 1];
  return make_int2(__ldg(start + (total - (base + hi))), __ldg(start + (total - (base + lo)) + 1));
}

// Marks the neighbors of the taken points: the candidates of the cell, kSteps per lane
// at a time in registers, against all of them.  own: in the cell itself too.  Warp
// `part` of `parts` takes its share of the candidates.
template <int D>
__device__ __forceinline__ void mark_neighbors(const SampleArgs& a, Taken<D>& taken,
                                               const int* cell, int batch, const int* nc,
                                               int total, const float* inv_r, bool own,
                                               int part, int parts) {
  constexpr int kSteps = 4;
  constexpr int kHalves = 2 * num_tubes<D>();
  constexpr int kTop = kHalves > 16 ? 16 : kHalves > 8 ? 8 : 4;
  const int lane = lane_id();
  if (part == 0 && lane < taken.count) __stcg(a.state + taken.j, (uint8_t)2);
  for (int half0 = 0; half0 < kHalves; half0 += 32) {
    int2 r = make_int2(0, 0);
    if (half0 + lane < kHalves)
      r = later_points<D>(half0 + lane, cell, batch, nc, total, own, a.c.start);
    int before = r.y - r.x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += y;
    }
    const int candidates = __shfl_sync(0xffffffffu, before, 31);
    const int offset = r.y - before;
    for (int base = part * 32 * kSteps; base < candidates; base += parts * 32 * kSteps) {
      if (base >= kProgressMarks && base % kProgressMarks < parts * 32 * kSteps && lane == 0)
        show_progress(a.arrived + 2);
      float p[kSteps][D];
      int at[kSteps];
      bool hit[kSteps];
#pragma unroll
      for (int k = 0; k < kSteps; ++k) {
        const int i = base + 32 * k + lane;
        int t = 0;
#pragma unroll
        for (int o = kTop; o > 0; o >>= 1) {
          const int y = __shfl_sync(0xffffffffu, before, t + o - 1);
          if (y <= i) t += o;
        }
        at[k] = i + __shfl_sync(0xffffffffu, offset, t & 31);
        hit[k] = false;
#pragma unroll
        for (int d = 0; d < D; ++d) p[k][d] = INFINITY;
        if (i < candidates) load_coords<D>(a.c, at[k], p[k]);
      }
      for (int who = 0; who < taken.count; ++who) {
        float s[D];
#pragma unroll
        for (int d = 0; d < D; ++d) s[d] = __shfl_sync(0xffffffffu, taken.p[d], who);
        const int j = __shfl_sync(0xffffffffu, taken.j, who);
#pragma unroll
        for (int k = 0; k < kSteps; ++k) hit[k] = hit[k] || (within<D>(s, p[k], inv_r) && at[k] != j);
      }
#pragma unroll
      for (int k = 0; k < kSteps; ++k)
        if (hit[k]) __stcg(a.state + at[k], (uint8_t)1);
    }
  }
  taken.count = 0;
}

// Greedy selection in one cell.  Which of its points are taken depends on the marks of
// earlier passes and on its own points only, so it is settled first, 32 points at a
// time in registers; the marks of the (few) taken points follow together: the chain
// per taken point is a ballot, not a walk over its candidates.
template <int D>
__device__ __forceinline__ void poisson_cell(const SampleArgs& a, const int* cell, int batch,
                                             int begin, int end, const int* nc, int total,
                                             const float* inv_r) {
  const int lane = lane_id();
  Taken<D> taken;
  taken.count = 0;
  taken.j = -1;
#pragma unroll
  for (int d = 0; d < D; ++d) taken.p[d] = 0.0f;
  float p_next[D];
  bool free_next;
  auto load = [&](int q) {
#pragma unroll
    for (int d = 0; d < D; ++d) p_next[d] = INFINITY;
    free_next = false;
    if (q < end) {
      load_coords<D>(a.c, q, p_next);
      free_next = __ldcg(a.state + q) == 0;
    }
  };
  load(begin + lane);
  for (int q0 = begin; q0 < end; q0 += 32) {
    float p[D];
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = p_next[d];
    const bool free = free_next;
    load(q0 + 32 + lane);      // (again below if marks come in between)
    unsigned open = __ballot_sync(0xffffffffu, free);
    for (int k = 0; k < taken.count && open; ++k) {
      float s[D];
#pragma unroll
      for (int d = 0; d < D; ++d) s[d] = __shfl_sync(0xffffffffu, taken.p[d], k);
      open &= ~__ballot_sync(0xffffffffu, within<D>(s, p, inv_r));
    }
    while (open) {
      const int t = __ffs(open) - 1;
      float s[D];
#pragma unroll
      for (int d = 0; d < D; ++d) s[d] = __shfl_sync(0xffffffffu, p[d], t);
      open &= ~(__ballot_sync(0xffffffffu, within<D>(s, p, inv_r)) | (1u << t));
      if (lane == taken.count) {
#pragma unroll
        for (int d = 0; d < D; ++d) taken.p[d] = s[d];
        taken.j = q0 + t;
      }
      if (++taken.count == 32) {
        mark_neighbors<D>(a, taken, cell, batch, nc, total, inv_r, true, 0, 1);
        __syncwarp();          // these marks are visible to the next group's reads
        load(q0 + 32 + lane);
      }
    }
  }
  if (taken.count > 0) mark_neighbors<D>(a, taken, cell, batch, nc, total, inv_r, false, 0, 1);
}

// What the warps of a block tell each other about a crowded cell.
template <int D>
struct BlockCell {
  int first[2][kWarps];          // every warp's first open point (INT_MAX: none), of two turns
  float first_p[2][kWarps][D];
  int taken[32];
  float taken_p[32][D];
};

// The selection in a crowded cell by a whole block: its points stand in registers, kHeld per thread
// at a time, and a turn takes the first that is open and closes its neighbors, all at once.  A cell
// is then as many turns of one barrier as it has points to take, a dozen mostly, where a warp went
// through its points 32 at a time (and the block's others with it, to share the marks): first of
// four levels of 8 x 100 000 Gaussian-mixture points 217 -> 207 us, first of three of 60 000
// 102 -> 98; cells of three radii, with dozens to take, 363 -> 376.
template <int D>
__device__ __forceinline__ void poisson_crowded_cell(const SampleArgs& a, BlockCell<D>& s,
                                                     const int* cell, int batch, int begin,
                                                     int end, const int* nc, int total,
                                                     const float* inv_r) {
  constexpr int kHeld = 4;
  const int lane = lane_id(), w = threadIdx.x >> 5;
  int count = 0;
  auto mark = [&](bool own) {
    // (the list is complete, and nobody looks at states meanwhile)
    __syncthreads();
    Taken<D> taken;
    taken.count = count;
    taken.j = lane < count ? s.taken[lane] : -1;
#pragma unroll
    for (int d = 0; d < D; ++d) taken.p[d] = lane < count ? s.taken_p[lane][d] : 0.0f;
    mark_neighbors<D>(a, taken, cell, batch, nc, total, inv_r, own, w, kWarps);
    __syncthreads();
    count = 0;
  };
  int turn = 0;
  for (int q0 = begin; q0 < end; q0 += kHeld * kThreads) {
    float p[kHeld][D];
    unsigned open = 0;
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
      const int q = q0 + k * kThreads + (int)threadIdx.x;
#pragma unroll
      for (int d = 0; d < D; ++d) p[k][d] = INFINITY;
      if (q < end) {
        load_coords<D>(a.c, q, p[k]);
        open |= (unsigned)(__ldcg(a.state + q) == 0) << k;
      }
    }
    auto close = [&](const float* x) {
#pragma unroll
      for (int k = 0; k < kHeld; ++k)
        if (within<D>(x, p[k], inv_r)) open &= ~(1u << k);
    };
    for (int k = 0; k < count; ++k) close(s.taken_p[k]);      // (of the points before)
    while (true) {
      const int k = __ffs(open) - 1;
      const int mine = open ? q0 + k * kThreads + (int)threadIdx.x : INT32_MAX;
      const int least = __reduce_min_sync(0xffffffffu, mine);
      const int buf = turn++ & 1;
      if (mine == least && (open || lane == 0)) {
        s.first[buf][w] = least;
#pragma unroll
        for (int u = 0; u < kHeld; ++u)
#pragma unroll
          for (int d = 0; d < D; ++d)
            if (k == u) s.first_p[buf][w][d] = p[u][d];
      }
      __syncthreads();
      int first = INT32_MAX, who = 0;
#pragma unroll
      for (int u = 0; u < kWarps; ++u) {
        const int x = s.first[buf][u];
        if (x < first) {
          first = x;
          who = u;
        }
      }
      if (first == INT32_MAX) break;
      float x[D];
#pragma unroll
      for (int d = 0; d < D; ++d) x[d] = s.first_p[buf][who][d];
      close(x);
      if (mine == first) open &= ~(1u << k);          // (itself, should it be no number)
      if (threadIdx.x == 0) {
        s.taken[count] = first;
#pragma unroll
        for (int d = 0; d < D; ++d) s.taken_p[count][d] = x[d];
      }
      if (++count == 32) mark(true);
    }
    __syncthreads();           // (the list, to be read at the next points)
  }
  if (count > 0) mark(false);
}

// Sorted points [x, y) of earlier passes in one half of a tube around `cell` (see later_points):
// both ends from an odd last coordinate, the middle if the leading coordinates' bits are lower.
template <int D>
__device__ __forceinline__ int2 earlier_points(int code, const int* cell, int batch, const int* nc,
                                               int total, const int32_t* __restrict__ start) {
  int base = 0, scale = 1, rem = code >> 1, mine = 0, theirs = 0;
  bool ok = true;
#pragma unroll
  for (int d = D - 2; d >= 0; --d) {
    const int c = cell[d] + rem % 3 - 1;
    rem /= 3;
    ok = ok && c >= 0 && c < nc[d];
    base += c * scale;
    scale *= nc[d];
    mine |= (cell[d] & 1) << d;
    theirs |= (c & 1) << d;
  }
  const int z = cell[D - 1];
  const bool second = code & 1, odd = z & 1;
  int lo, hi;
  if (theirs < mine) {
    lo = odd ? z - 1 : z;
    hi = odd ? min(z + 1, nc[D - 1] - 1) : z;
    ok = ok && !second;
  } else {
    lo = hi = second ? z + 1 : z - 1;
    ok = ok && odd && lo < nc[D - 1];
  }
  if (!ok) return make_int2(0, 0);
  base = (batch * scale + base) * nc[D - 1];
  return make_int2(__ldg(start + (total - (base + hi))), __ldg(start + (total - (base + lo)) + 1));
}

// The team of a block: blocks [begin, begin + size) work on `cloud`; with too many clouds
// for teams, all blocks on all of them (cloud -1).  size 0: a block left over.
struct Team { int cloud, begin, size; };

// One block per cloud and the others in proportion to the clouds' points.
__device__ __forceinline__ Team team_of(const CellsView& c, int64_t n, int blocks, int total) {
  const int lane = lane_id();
  if (c.batch_size > kMaxTeams || c.batch_size * 2 > blocks) return Team{-1, 0, blocks};
  const int cells = total / c.batch_size;
  const long long spare = blocks - c.batch_size;
  int before = 0;
  for (int b0 = 0; b0 < c.batch_size; b0 += 32) {
    const int b = b0 + lane;
    int share = 0;
    if (b < c.batch_size) {
      const int points = __ldg(c.start + (total - b * cells) + 1) -
                         __ldg(c.start + (total - (b + 1) * cells) + 1);
      share = 1 + (int)(spare * points / n);
    }
    int upto = share;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += y;
    }
    upto += before;
    const unsigned m = __ballot_sync(0xffffffffu, upto > (int)blockIdx.x);
    if (m) {
      const int who = __ffs(m) - 1;
      const int size = __shfl_sync(0xffffffffu, share, who);
      return Team{b0 + who, __shfl_sync(0xffffffffu, upto, who) - size, size};
    }
    before = __shfl_sync(0xffffffffu, upto, 31);
  }
  return Team{0, 0, 0};
}

// Candidates of point i by sample: those before it in its cell, and as many times as there are halves
// those of one of them; very many where its cell is too full.  Over a block's threads, with points
// from all over the level, the mean is 12 % off (rms over 200 levels; at most 36 %).  (A call: as a
// part of settle_kernel it slows the search down by a third.)
template <int D>
__device__ __noinline__ int sampled_candidates(int i, const int64_t* keys, const int32_t* start,
                                               const int32_t* num_cells, int total) {
  constexpr int kHalves = 2 * num_tubes<D>();
  const int64_t key = __ldg(keys + i);
  if (key < 0 || key >= total) return 0;
  int cell[D], nc[D], rem = (int)key;
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    nc[d] = __ldg(num_cells + d);
    cell[d] = rem % nc[d];
    rem /= nc[d];
  }
  const int2 x = earlier_points<D>(threadIdx.x * 37 % kHalves, cell, rem, nc, total, start);
  const int begin = __ldg(start + (total - (int)key)), end = __ldg(start + (total - (int)key) + 1);
  return end - begin > kFlowCell ? 1 << 20 : min(i - begin + kHalves * (x.y - x.x), 1 << 20);
}

// The selection without passes: a point is settled as soon as its earlier neighbors (of earlier
// passes, or before it in its cell) are, not when all cells of their passes are.  Eight lanes find
// those neighbors, as words of 32 points and masks; then they look at the words until one of the
// neighbors is taken, or all are settled and none is.  All blocks are resident (a cooperative
// launch), and a point waits for earlier ones only.  What is taken is counted for the block that
// will write it (cells_sample_kernel, which follows and has nothing to wait for).  The chain of a
// level is a search and some twenty trips to L2, where the passes have ten barriers and a walk per
// cell between them: levels of 54 000, 10 600 and 2000 points take 81, 57 and 48 us by passes, 46,
// 23 and 21 so.
// Where cells are crowded the passes, which test around taken points only, are the faster ones.  All
// blocks of a level of more than kFlowFew points find that out from the same points, before they
// test any: 1.2 us of a settled level, 6 in all of one that is left.  (Blocks whose own points have
// less than an eighth of that need not ask: a quarter would make some test in vain, 7000 points
// with 260 neighbors 106 -> 124 us.  When each went by its own points, and few found it out, the
// others tested in vain for 16 to 43 us: levels of 30 000 and 60 000 points with 100 to 270
// candidates took 130 to 157 us, now 114 to 121, by passes alone 103 to 111.)  A block with far more
// candidates than that, a list that runs over and a cell that is too full leave the level to the
// passes as well, and a point of too full a cell is not searched for.  Then nothing of this counts
// (20 000 points in one cell, this kernel and the passes, without a look at a point's own cell
// 408 + 43 us, with it 4 + 43; in eight clouds of a cell each 190 + 31 and 4 + 31).
template <int D>
__global__ void __launch_bounds__(kThreads, 4)
settle_kernel(SampleArgs a) {
  constexpr int kGroups = kThreads / 8, kTurns = kFlowPer / kGroups, kPer = kFlowLists / 8;
  constexpr int kHalves = 2 * num_tubes<D>();
  constexpr int kMine = D <= 3 ? (kHalves + 7) / 8 : 1;       // halves of a lane looked up at once
  __shared__ uint2 lists[kFlowPer][kFlowLists];
  __shared__ int listed[kFlowPer], candidates_s, sampled_s;
  const int lane = lane_id(), eighth = lane & 7, group = threadIdx.x >> 3;
  int nc[D];
  float inv_r[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    nc[d] = __ldg(a.c.num_cells + d);
    inv_r[d] = __ldg(a.inv_radii + d);
  }
  const int total = total_cells<D>(nc, a.c.batch_size);
  if (total == 0) return;        // (a grid that got no cells: the call fails)
  const int64_t n = a.n_dev ? __ldg(a.n_dev) : a.c.n;
  volatile unsigned* const failed = a.arrived + 4;
  // (as few blocks as have a point for every eight lanes)
  const int blocks = (int)min((int64_t)gridDim.x, settle_blocks(n));
  if ((int)blockIdx.x >= blocks) return;
  if ((n + 3) / 4 > (int64_t)blocks * (kFlowPer / 4)) {       // (too few blocks are resident)
    *failed = 1u;
    return;
  }
  const int write_blocks = sample_blocks(n, a.write_blocks);
  const int per = (int)((n + write_blocks - 1) / write_blocks);    // points that a block writes
  const int turns = (int)((n + (int64_t)blocks * kGroups - 1) / ((int64_t)blocks * kGroups));
  // Point q of this block: four neighboring ones to a warp at a time (mostly of one cell), and
  // every blocks-th such four to a block: neighboring ones cost the same, and the slowest block
  // decides.
  auto point = [&](int q) { return ((int)blockIdx.x + (q >> 2) * blocks) * 4 + (q & 3); };
  for (int i = threadIdx.x; i < kFlowPer; i += kThreads) listed[i] = 0;
  if (threadIdx.x == 0) candidates_s = sampled_s = 0;
  __syncthreads();
  for (int turn = 0; turn < turns; ++turn) {
    const int q = group + turn * kGroups;
    const int j = point(q);
    const int64_t key = j < n ? __ldg(a.keys + j) : -1;
    const bool live = key >= 0 && key < total;         // (else in no cell: without neighbors)
    int cell[D], rem = live ? (int)key : 0;
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
      cell[d] = rem % nc[d];
      rem /= nc[d];
    }
    int begin = 0, end = 0;
    int2 r[kMine];
#pragma unroll
    for (int k = 0; k < kMine; ++k) r[k] = make_int2(0, 0);
    if (live) {
      begin = __ldg(a.c.start + (total - (int)key));
      end = __ldg(a.c.start + (total - (int)key) + 1);
#pragma unroll
      for (int k = 0; k < kMine; ++k)
        if (8 * k + eighth < kHalves)
          r[k] = earlier_points<D>(8 * k + eighth, cell, rem, nc, total, a.c.start);
    }
    if (turn == 0) {
      int mine = live && eighth == 0 ? j - begin : 0;
#pragma unroll
      for (int k = 0; k < kMine; ++k) mine += r[k].y - r[k].x;
      if (kMine * 8 < kHalves && live)
        for (int t = 8 * kMine + eighth; t < kHalves; t += 8) {
          const int2 x = earlier_points<D>(t, cell, rem, nc, total, a.c.start);
          mine += x.y - x.x;
        }
      mine = __reduce_add_sync(0xffffffffu, mine);
      if (lane == 0) atomicAdd(&candidates_s, mine);
      __syncthreads();
      const int limit = min(flow_work(D) / turns, kFlowMost);
      if (n > kFlowFew && candidates_s > limit * kGroups / 8) {
        const int i = (int)((threadIdx.x >> 2) * n / (kThreads / 4));      // (the same in all blocks)
        const int some = __reduce_add_sync(
            0xffffffffu, sampled_candidates<D>(i, a.keys, a.c.start, a.c.num_cells, total));
        if (lane == 0) atomicAdd(&sampled_s, some);
        __syncthreads();
      }
      if (sampled_s > limit * kThreads ||
          candidates_s > (n > kFlowFew ? 4 * limit : 448) * kGroups) {
        if (threadIdx.x == 0) *failed = 1u;
        return;
      }
    }
    if (end - begin > kFlowCell) {
      *failed = 1u;
      return;
    }
    if (*failed) return;
    if (!live) continue;
    float p[D];
    load_coords<D>(a.c, j, p);
    // the neighbors among the points [x, y), words w, w + step, ..
    auto search = [&](int2 r, int w, int step) {
      for (; r.x < r.y && w * 32 < r.y; w += step) {
        unsigned mask = 0;
        const int to = min(r.y, w * 32 + 32);
        // (four loads under way together, also of the last few)
        for (int i = max(r.x, w * 32); i < to; i += 4) {
          float o[4][D];
#pragma unroll
          for (int u = 0; u < 4; ++u) load_coords<D>(a.c, min(i + u, to - 1), o[u]);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (within<D>(p, o[u], inv_r)) mask |= 1u << (min(i + u, to - 1) & 31);
        }
        if (mask) {
          const int slot = atomicAdd(&listed[q], 1);
          if (slot < kFlowLists) lists[q][slot] = make_uint2((unsigned)w, mask);
          else *failed = 1u;
        }
      }
    };
#pragma unroll 1
    for (int k = 0; k < kMine; ++k) {
      int2 x = r[0];
#pragma unroll
      for (int u = 1; u < kMine; ++u) x = k == u ? r[u] : x;
      search(x, x.x >> 5, 1);
    }
    for (int t = 8 * kMine + eighth; t < kHalves; t += 8) {
      const int2 x = earlier_points<D>(t, cell, rem, nc, total, a.c.start);
      search(x, x.x >> 5, 1);
    }
    search(make_int2(begin, j), (begin >> 5) + eighth, 8);
  }
  __syncwarp();
  unsigned left = 0;          // turns whose point is not settled yet
#pragma unroll
  for (int k = 0; k < kTurns; ++k) left |= (k < turns && point(group + k * kGroups) < n) << k;
  unsigned long long t0 = 0;
  for (unsigned look = 1; __any_sync(0xffffffffu, left); ++look) {
    if ((look & 7u) == 0 && __any_sync(0xffffffffu, *failed != 0u)) return;
    if ((look & 255u) == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      if (__any_sync(0xffffffffu, t - t0 > 2 * a.period_ns)) {
        *(volatile unsigned*)(a.arrived + 1) = 1u;     // (no other block waits for long either)
        *failed = 1u;
        return;
      }
    }
#pragma unroll
    for (int k = 0; k < kTurns; ++k) {
      if (!__any_sync(0xffffffffu, left >> k & 1u)) continue;
      const int q = group + k * kGroups;
      const bool open = left >> k & 1u;
      const int count = open ? min(listed[q], kFlowLists) : 0;
      bool blocked = false, waits = false;
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const int slot = eighth + 8 * e;
        if (slot < count) {
          const uint2 l = lists[q][slot];
          const unsigned long long v =
              *(const volatile unsigned long long*)(a.settled + l.x);
          blocked = blocked || ((unsigned)v & l.y) != 0u;
          waits = waits || (l.y & ~(unsigned)(v >> 32)) != 0u;
        }
      }
      const unsigned any_blocked = __ballot_sync(0xffffffffu, blocked) >> (lane & 24) & 0xffu;
      const unsigned any_waits = __ballot_sync(0xffffffffu, waits) >> (lane & 24) & 0xffu;
      if (open && (any_blocked || !any_waits)) {
        left &= ~(1u << k);
        if (eighth == 0) {
          const int j = point(q);
          const unsigned long long bit = 1ull << (j & 31);
          atomicOr(a.settled + (j >> 5), any_blocked ? bit << 32 : bit << 32 | bit);
          if (!any_blocked) atomicAdd(a.block_total + j / per, 1);
        }
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(kThreads, 4)
cells_sample_kernel(SampleArgs a) {
  __shared__ int warp_total[kWarps], warp_all[kWarps], before_s;
  __shared__ int crowded[kMaxCrowded], num_crowded[2];     // (counters of this pass and the next)
  __shared__ BlockCell<D> block_cell;
  const int lane = lane_id(), w = threadIdx.x >> 5;
  int nc[D];
#pragma unroll
  for (int d = 0; d < D; ++d) nc[d] = __ldg(a.c.num_cells + d);
  const int total = total_cells<D>(nc, a.c.batch_size);
  if (total == 0) {              // (a grid that got no cells: the call fails)
    if (a.samples_dev && blockIdx.x == 0 && threadIdx.x == 0) *a.samples_dev = 0;
    return;
  }
  const int64_t n = a.n_dev ? __ldg(a.n_dev) : a.c.n;
  const int blocks = sample_blocks(n, (int)gridDim.x);
  if ((int)blockIdx.x >= blocks) return;      // (nobody waits for them)
  unsigned barriers = 0;
  bool ok = true, settled = false;
  if (a.mode == 0) {
    float inv_r[D];
#pragma unroll
    for (int d = 0; d < D; ++d) inv_r[d] = __ldg(a.inv_radii + d);
    // points outside every cell have no neighbors: all of them are taken
    const int lead = __ldg(a.c.start + 1), tail = __ldg(a.c.start + total + 1);
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < lead + (n - tail);
         i += (int64_t)blocks * kThreads)
      a.state[i < lead ? i : tail + (i - lead)] = 2;
    if (threadIdx.x == 0) num_crowded[0] = 0;
    __syncthreads();
    settled = a.settled != nullptr && a.arrived[4] == 0u;
    const Team team = settled ? Team{0, 0, 0} : team_of(a.c, n, blocks, total);
    const int warps = team.size * kWarps;
    // neighboring cells go to different blocks: crowded ones come side by side
    const int warp = w * team.size + (int)blockIdx.x - team.begin;
    unsigned* const counter = team.cloud < 0 ? a.arrived : a.arrived + kHeadWords + team.cloud;
    for (int pass = 0; pass < (1 << D) && team.size > 0; ++pass) {
      int half[D], cells = team.cloud < 0 ? a.c.batch_size : 1;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        half[d] = (nc[d] - ((pass >> d) & 1) + 1) >> 1;
        cells *= half[d];
      }
      int* const queued = num_crowded + (pass & 1);
      // the i-th cell of this pass
      auto cell_at = [&](int i, int* cell, int* batch, int* begin, int* end) {
        int rem = i, key = 0, scale = 1;
#pragma unroll
        for (int d = D - 1; d >= 0; --d) {
          cell[d] = 2 * (rem % half[d]) + ((pass >> d) & 1);
          rem /= half[d];
          key += cell[d] * scale;
          scale *= nc[d];
        }
        *batch = team.cloud < 0 ? rem : team.cloud;
        key += *batch * scale;
        *begin = __ldg(a.c.start + (total - key));
        *end = __ldg(a.c.start + (total - key) + 1);
      };
      // a lane looks at every `warps`-th cell: crowded regions spread over the warps
      for (int c0 = 0; c0 < cells; c0 += 32 * warps) {
        if (c0 >= 64 * 32 * warps && lane == 0) show_progress(a.arrived + 2);
        const int i = c0 + lane * warps + warp;
        int cell[D], batch = 0, begin = 0, end = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) cell[d] = 0;
        if (i < cells) cell_at(i, cell, &batch, &begin, &end);
        if (end - begin > kCrowded) {
          const int slot = atomicAdd(queued, 1);
          if (slot < kMaxCrowded) {
            crowded[slot] = i;
            end = begin;
          }
        }
        unsigned work = __ballot_sync(0xffffffffu, end > begin);
        while (work) {
          const int who = __ffs(work) - 1;
          work &= work - 1u;
          int cc[D];
#pragma unroll
          for (int d = 0; d < D; ++d) cc[d] = __shfl_sync(0xffffffffu, cell[d], who);
          poisson_cell<D>(a, cc, __shfl_sync(0xffffffffu, batch, who),
                          __shfl_sync(0xffffffffu, begin, who),
                          __shfl_sync(0xffffffffu, end, who), nc, total, inv_r);
        }
      }
      __syncthreads();
      const int shared_cells = min(*queued, kMaxCrowded);
      if (threadIdx.x == 0) num_crowded[(pass + 1) & 1] = 0;
      for (int k = 0; k < shared_cells; ++k) {
        int cell[D], batch, begin, end;
        cell_at(crowded[k], cell, &batch, &begin, &end);
        poisson_crowded_cell<D>(a, block_cell, cell, batch, begin, end, nc, total, inv_r);
      }
      if (pass + 1 == (1 << D)) break;     // (the compaction begins with a barrier)
      ok = grid_barrier(counter, (pass + 1) * team.size, a.arrived + 1, a.arrived + 2,
                        a.period_ns) && ok;
    }
    if (team.cloud < 0) barriers = (1 << D) - 1;
    if (!settled)
      ok = grid_barrier(a.arrived, ++barriers * blocks, a.arrived + 1, a.arrived + 2,
                        a.period_ns) && ok;
  }
  // ---- compaction: every block counts, then writes, its stretch of the points
  const int64_t per = (n + blocks - 1) / blocks;
  const int64_t first = min((int64_t)blockIdx.x * per, n), last = min(first + per, n);
  auto chosen = [&](int64_t i) {
    if (i >= last) return false;
    if (settled) return (__ldcg((const unsigned*)(a.settled + (i >> 5))) >> (i & 31) & 1u) != 0u;
    return a.mode == 0 ? __ldcg(a.state + i) == 2
                       : i == 0 || __ldg(a.keys + i) != __ldg(a.keys + i - 1);
  };
  if (!settled) {
    int mine = 0;
    for (int64_t i = first + threadIdx.x; i < last; i += kThreads) mine += chosen(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) warp_total[w] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int i = 0; i < kWarps; ++i) t += warp_total[i];
      __stcg(a.block_total + blockIdx.x, t);
    }
    ok = grid_barrier(a.arrived, ++barriers * blocks, a.arrived + 1, a.arrived + 2,
                      a.period_ns) && ok;
  }
  ok = ok && !any_gave_up(a.arrived + 1);
  {
    // samples of the blocks before this one, and all
    int t = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kMaxBlocks / kThreads; ++k) {
      const int i = (int)threadIdx.x + k * kThreads;
      const int v = i < blocks ? __ldcg(a.block_total + i) : 0;
      all += v;
      t += i < (int)blockIdx.x ? v : 0;
    }
    t = __reduce_add_sync(0xffffffffu, t);
    all = __reduce_add_sync(0xffffffffu, all);
    __syncthreads();
    if (lane == 0) {
      warp_total[w] = t;
      warp_all[w] = all;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      t = all = 0;
      for (int i = 0; i < kWarps; ++i) {
        t += warp_total[i];
        all += warp_all[i];
      }
      before_s = t;
      if (blockIdx.x == 0) {
        a.page[0] = all;
        a.page[1] = 0;
        a.page[2] = ok ? 0 : 1;
        if (a.samples_dev) *a.samples_dev = ok ? all : 0;
      }
    }
  }
  __syncthreads();
  int64_t out = before_s;
  if (!ok) return;
  for (int64_t i0 = first; i0 < last; i0 += kThreads) {
    const int64_t i = i0 + threadIdx.x;
    const bool take = chosen(i);
    const unsigned m = __ballot_sync(0xffffffffu, take);
    __syncthreads();
    if (lane == 0) warp_total[w] = __popc(m);
    __syncthreads();
    int ahead = 0, sum = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) {
      if (k < w) ahead += warp_total[k];
      sum += warp_total[k];
    }
    int64_t end = i;      // of the cell that begins at point i
    if (take) {
      const int64_t o = out + ahead + __popc(m & ((1u << lane) - 1u));
      if (a.mode == 0) {
#pragma unroll
        for (int d = 0; d < D; ++d) a.pts_out[o * D + d] = __ldg(a.c.points + i * D + d);
        a.batch_out[o] = __ldg(a.c.batch_ids + i);
        a.index_out[o] = __ldg(a.c.indices + i);
      } else {
        const int64_t key = __ldg(a.keys + i);
        float acc[D];
#pragma unroll
        for (int d = 0; d < D; ++d) acc[d] = 0.0f;
        if (key >= 0 && key < total) {
          end = __ldg(a.c.start + (total - (int)key) + 1);
        } else {
          while (end < n && __ldg(a.keys + end) == key) ++end;
        }
        if (end - i <= kLongCell) {
#pragma unroll 4
          for (int64_t q = i; q < end; ++q)
#pragma unroll
            for (int d = 0; d < D; ++d) acc[d] += __ldg(a.c.points + q * D + d);
          const float cnt = (float)(end - i);
#pragma unroll
          for (int d = 0; d < D; ++d) a.pts_out[o * D + d] = acc[d] / cnt;
        }
        a.batch_out[o] = (int32_t)(key / (total / a.c.batch_size));
      }
    }
    // cells of many points: read by their warp together, summed in the same order
    unsigned lengthy = __ballot_sync(0xffffffffu, a.mode == 1 && take && end - i > kLongCell);
    while (lengthy) {
      const int who = __ffs(lengthy) - 1;
      lengthy &= lengthy - 1u;
      const int64_t from = __shfl_sync(0xffffffffu, i, who), to = __shfl_sync(0xffffffffu, end, who);
      float acc[D], p[D];
      auto load = [&](int64_t q) {
#pragma unroll
        for (int d = 0; d < D; ++d) p[d] = q < to ? __ldg(a.c.points + q * D + d) : 0.0f;
      };
#pragma unroll
      for (int d = 0; d < D; ++d) acc[d] = 0.0f;
      load(from + lane);
      for (int64_t q = from; q < to; q += 32) {
        float now[D];
#pragma unroll
        for (int d = 0; d < D; ++d) now[d] = p[d];
        load(q + 32 + lane);
        const int have = (int)min(to - q, (int64_t)32);
        if (have == 32) {
#pragma unroll
          for (int k = 0; k < 32; ++k)
#pragma unroll
            for (int d = 0; d < D; ++d) acc[d] += __shfl_sync(0xffffffffu, now[d], k);
        } else {
          for (int k = 0; k < have; ++k)
#pragma unroll
            for (int d = 0; d < D; ++d) acc[d] += __shfl_sync(0xffffffffu, now[d], k);
        }
      }
      if (lane == who) {
        const int64_t o = out + ahead + __popc(m & ((1u << lane) - 1u));
        const float cnt = (float)(to - from);
#pragma unroll
        for (int d = 0; d < D; ++d) a.pts_out[o * D + d] = acc[d] / cnt;
      }
    }
    out += sum;
  }
}

// Blocks of a cooperative launch that are resident at once, at most 4 per SM.
template <auto kKernel>
int resident_blocks(int64_t wanted, unsigned* blocks) {
  static int per_sm = 0;     // (the same value whoever computes it)
  if (per_sm == 0) {
    int v = 0;
    TFGPC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kKernel, kThreads, 0));
    per_sm = v < 1 ? 1 : v;
  }
  const int64_t most = (int64_t)sm_count() * (per_sm < 4 ? per_sm : 4);
  if (wanted > most) wanted = most;
  *blocks = (unsigned)(wanted > kMaxBlocks ? kMaxBlocks : wanted);
  return TFGPC_OK;
}

template <int D>
int launch_sample(cudaStream_t st, SampleArgs a) {
  unsigned blocks = 0;
  int rc = resident_blocks<cells_sample_kernel<D>>(blocks_wanted(a.c.n), &blocks);
  if (rc) return rc;
  a.write_blocks = (int)blocks;
  void* args[] = {&a};
  if (a.settled) {
    unsigned first = 0;
    rc = resident_blocks<settle_kernel<D>>(settle_blocks(a.c.n), &first);
    if (rc) return rc;
    TFGPC_CUDA(cudaLaunchCooperativeKernel(settle_kernel<D>, dim3(first), dim3(kThreads), args, 0, st));
  }
  TFGPC_CUDA(cudaLaunchCooperativeKernel(cells_sample_kernel<D>, dim3(blocks), dim3(kThreads), args,
                                         0, st));
  return TFGPC_OK;
}

// The sampling's sequence of barriers without its work: two at the counter of a block's
// team (even and odd blocks), two of the grid.  Block late_block comes to barrier late_at
// after eight periods.  words: error, barrier counters, what block 0 would report, number
// of blocks that would return without writing, progress.
__global__ void barrier_probe_kernel(unsigned* words, int late_block, int late_at, int working,
                                     unsigned long long period_ns) {
  bool ok = true;
  for (int k = 0; k < 4; ++k) {
    if ((int)blockIdx.x == late_block && k == late_at && threadIdx.x == 0) {
      unsigned long long t0, t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      do {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (working) show_progress(words + 6);
      } while (t - t0 < 8 * period_ns);
    }
    unsigned* const counter = words + 1 + (k < 2 ? 1 + (blockIdx.x & 1) : 0);
    const unsigned blocks = k < 2 ? gridDim.x / 2 : gridDim.x;
    ok = grid_barrier(counter, (k % 2 + 1) * blocks, words, words + 6, period_ns) && ok;
  }
  ok = ok && !any_gave_up(words);
  if (threadIdx.x != 0) return;
  if (blockIdx.x == 0) words[4] = ok ? 0u : 1u;
  if (!ok) atomicAdd(words + 5, 1u);
}

// Barrier words, a byte of state per point, of a level that settle_kernel is tried on two bits, and
// the blocks' totals.
size_t settled_at(int64_t n) { return align_up((size_t)n + kHeadBytes, 8); }
size_t totals_at(int64_t n) {
  return settled_at(n) + (n <= kFlowPoints ? (size_t)((n + 31) / 32) * 8 : 0);
}

size_t sample_ws_bytes(int64_t n) { return align_up(totals_at(n) + (size_t)kMaxBlocks * 4, 256); }

// What has to be zero before the kernel starts.
size_t clear_bytes(int64_t n, int mode) {
  return mode != 0 ? kHeadBytes : totals_at(n) + (n <= kFlowPoints ? (size_t)kMaxBlocks * 4 : 0);
}

// Enqueues the sampling; the number of samples goes to words kReportTotal .. of the page.
int sample_async(cudaStream_t st, const tfgpc_cell_grid& g, int mode, const float* inv_radii,
                 float* pts_out, int32_t* batch_out, int32_t* index_out, void* ws, int32_t* page,
                 bool cleared, const int64_t* n_dev = nullptr, int64_t* samples_dev = nullptr) {
  SampleArgs a;
  a.c = view_of(g);
  a.keys = g.sorted_keys;
  a.mode = mode;
  a.inv_radii = inv_radii;
  a.arrived = (unsigned*)ws;
  a.state = (uint8_t*)ws + kHeadBytes;
  // (by passes where a caller's workspace is not aligned for words of 64 bits)
  const bool flow = mode == 0 && g.n <= kFlowPoints && (uintptr_t)ws % 8 == 0;
  a.settled = flow ? (unsigned long long*)((char*)ws + settled_at(g.n)) : nullptr;
  a.block_total = (int32_t*)((char*)ws + totals_at(g.n));
  a.pts_out = pts_out;
  a.batch_out = batch_out;
  a.index_out = index_out;
  a.page = page + kReportTotal;
  a.n_dev = n_dev;
  a.samples_dev = samples_dev;
  a.period_ns = barrier_period_ns(g.n);
  ProfScope prof(st, mode == 0 ? "sampling_poisson" : "sampling_cell_average");
  if (!cleared) TFGPC_CUDA(cudaMemsetAsync(ws, 0, clear_bytes(g.n, mode), st));
  switch (g.D) {
    case 2: return launch_sample<2>(st, a);
    case 3: return launch_sample<3>(st, a);
    case 4: return launch_sample<4>(st, a);
    case 5: return launch_sample<5>(st, a);
    default: return launch_sample<6>(st, a);
  }
}

int check_sample(const tfgpc_cell_grid* g, int mode, const float* inv_radii, const float* pts_out,
                 const int32_t* batch_out, const int32_t* index_out, const void* ws,
                 size_t ws_bytes, const int64_t* num_samples_out) {
  int rc = check_cell_grid("SamplingOp", g);
  if (rc) return rc;
  TFGPC_REQUIRE(mode == 0 || mode == 1, "SamplingOp expects mode 0 (poisson) or 1 (average)");
  TFGPC_REQUIRE(pts_out && batch_out && ws && num_samples_out &&
                (mode == 1 || (index_out && inv_radii)), "SamplingOp got a null pointer");
  TFGPC_REQUIRE((uintptr_t)ws % 4 == 0, "SamplingOp expects a workspace aligned to 4 bytes");
  if (ws_bytes < sample_ws_bytes(g->n)) return fail(TFGPC_ENOMEM, "SamplingOp workspace too small");
  return TFGPC_OK;
}

// The outputs of a blocking entry from the words that a level has left in the report page.
int level_report(const int32_t* host, const tfgpc_cell_grid& g, int32_t* num_cells_host_out,
                 int64_t* num_samples_out) {
  for (int d = 0; num_cells_host_out && d < g.D; ++d) num_cells_host_out[d] = host[d];
  if (num_cells_host_out && host[TFGPC_MAX_DIMS])
    return fail(TFGPC_ENOMEM, "SamplingOp: the grid needs more than max_cells = %d cells in a "
                "dimension; repeat the call with a larger bound", g.max_cells);
  if (host[kReportWords])
    return fail(TFGPC_ETIMEOUT, "a bounded wait inside the sampling kernel ran out");
  *num_samples_out = (int64_t)(uint32_t)host[kReportTotal] |
                     ((int64_t)host[kReportTotal + 1] << 32);
  return TFGPC_OK;
}

int finish_sample(cudaStream_t st, const tfgpc_cell_grid& g, int32_t* num_cells_host_out,
                  int64_t* num_samples_out) {
  int32_t host[kReportWords + 1];
  int rc = read_report(st, sizeof(host), host);
  return rc ? rc : level_report(host, g, num_cells_host_out, num_samples_out);
}

constexpr int kMaxLevels = TFGPC_MAX_CHAINED_LEVELS;
constexpr int kLevelWords = 16;          // of the report page, one level
static_assert(kReportWords + 1 <= kLevelWords && kMaxLevels * kLevelWords * 4 <= 4096, "page");

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

extern "C" size_t tfgpc_cells_sample_workspace_bytes(int64_t n) {
  return n > 0 ? sample_ws_bytes(n) : 256;
}

extern "C" int tfgpc_cells_sample(void* stream, const tfgpc_cell_grid* grid, int mode,
                                  const float* inv_radii, float* sample_pts_out,
                                  int32_t* sample_batch_ids_out, int32_t* sample_indices_out,
                                  void* ws, size_t ws_bytes, int64_t* num_samples_out) {
  int rc = check_sample(grid, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                        sample_indices_out, ws, ws_bytes, num_samples_out);
  if (rc) return rc;
  *num_samples_out = 0;
  cudaStream_t st = (cudaStream_t)stream;
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  rc = sample_async(st, *grid, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                    sample_indices_out, ws, (int32_t*)page, false);
  if (rc) return rc;
  return finish_sample(st, *grid, nullptr, num_samples_out);
}

extern "C" int tfgpc_cell_grid_sample(void* stream, const tfgpc_cell_grid* grid,
                                      const float* points, const int32_t* batch_ids,
                                      const float* cell_sizes, const int32_t* num_cells_in,
                                      int mode, const float* inv_radii, float* sample_pts_out,
                                      int32_t* sample_batch_ids_out, int32_t* sample_indices_out,
                                      void* ws, size_t ws_bytes, void* sample_ws,
                                      size_t sample_ws_bytes_given, int32_t* num_cells_host_out,
                                      int64_t* num_samples_out) {
  int rc = check_sample(grid, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                        sample_indices_out, sample_ws, sample_ws_bytes_given, num_samples_out);
  if (rc) return rc;
  const tfgpc_cell_grid& g = *grid;
  TFGPC_REQUIRE(points && batch_ids && cell_sizes && ws && num_cells_host_out,
                "SamplingOp got a null pointer");
  TFGPC_REQUIRE(num_cells_in != g.num_cells,
                "SamplingOp expects the given cell counts outside the output array");
  for (int d = 0; d < g.D; ++d)
    TFGPC_REQUIRE(cell_sizes[d] > 0.0f, "SamplingOp expects positive cell sizes");
  if (ws_bytes < tfgpc_cell_grid_workspace_bytes(g.D, g.n, 0, g.batch_size, g.max_cells))
    return fail(TFGPC_ENOMEM, "SamplingOp workspace too small");
  *num_samples_out = 0;
  cudaStream_t st = (cudaStream_t)stream;
  CellGridWs w = carve_cell_grid(ws, g.n, 0, g.D, g.batch_size, g.max_cells);
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  const AlsoClear also{(uint32_t*)sample_ws, (int64_t)(clear_bytes(g.n, mode) / 4)};
  rc = cell_grid_build(st, g, points, batch_ids, cell_sizes, num_cells_in, w, (int32_t*)page, also);
  if (rc) return rc;
  rc = sample_async(st, g, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                    sample_indices_out, sample_ws, (int32_t*)page, true);
  if (rc) return rc;
  return finish_sample(st, g, num_cells_host_out, num_samples_out);
}

extern "C" int64_t tfgpc_cell_grid_level_points(int D, int64_t batch_size, int max_cells) {
  if (!valid_dims(D) || batch_size < 1 || batch_size >= (int64_t)INT32_MAX || max_cells < 1) return 0;
  return cell_grid_cluster_points(D, batch_size, max_cells);
}

// With a blocking read per level the GPU waited 31 to 44 us between two levels of 10 to 80: for
// the host to see the number of points, to make the next level's arrays and for its first launch
// to arrive.
extern "C" int tfgpc_cell_grid_sample_level(
    void* stream, int level, const tfgpc_cell_grid* grid, const float* points,
    const int32_t* batch_ids, const int64_t* n_dev, const float* cell_sizes, int mode,
    const float* inv_radii, float* sample_pts_out, int32_t* sample_batch_ids_out,
    int32_t* sample_indices_out, int64_t* num_samples_dev_out, void* ws, size_t ws_bytes,
    void* sample_ws, size_t sample_ws_bytes_given) {
  TFGPC_REQUIRE(level >= 0 && level < kMaxLevels, "SamplingOp expects a level below %d", kMaxLevels);
  int64_t unused = 0;
  int rc = check_sample(grid, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                        sample_indices_out, sample_ws, sample_ws_bytes_given, &unused);
  if (rc) return rc;
  const tfgpc_cell_grid& g = *grid;
  TFGPC_REQUIRE(points && batch_ids && cell_sizes && ws && num_samples_dev_out,
                "SamplingOp got a null pointer");
  TFGPC_REQUIRE(n_dev != num_samples_dev_out, "SamplingOp expects two counts, not one");
  for (int d = 0; d < g.D; ++d)
    TFGPC_REQUIRE(cell_sizes[d] > 0.0f, "SamplingOp expects positive cell sizes");
  if (ws_bytes < tfgpc_cell_grid_workspace_bytes(g.D, g.n, 0, g.batch_size, g.max_cells))
    return fail(TFGPC_ENOMEM, "SamplingOp workspace too small");
  TFGPC_REQUIRE(!n_dev || g.n <= cell_grid_cluster_points(g.D, g.batch_size, g.max_cells),
                "SamplingOp: too large a level for points not counted yet");
  cudaStream_t st = (cudaStream_t)stream;
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  int32_t* words = (int32_t*)page + level * kLevelWords;
  const CellGridWs w = carve_cell_grid(ws, g.n, 0, g.D, g.batch_size, g.max_cells);
  const AlsoClear also{(uint32_t*)sample_ws, (int64_t)(clear_bytes(g.n, mode) / 4)};
  rc = cell_grid_build(st, g, points, batch_ids, cell_sizes, nullptr, w, words, also, n_dev);
  if (rc) return rc;
  return sample_async(st, g, mode, inv_radii, sample_pts_out, sample_batch_ids_out,
                      sample_indices_out, sample_ws, words, true, n_dev, num_samples_dev_out);
}

extern "C" int tfgpc_cell_grid_sample_report(void* stream, int levels, int D, int max_cells,
                                             int32_t* num_cells_host_out, int64_t* num_samples_out,
                                             int* levels_done_out) {
  TFGPC_REQUIRE(levels >= 1 && levels <= kMaxLevels && valid_dims(D),
                "SamplingOp expects 1 to %d levels and a valid dimension", kMaxLevels);
  TFGPC_REQUIRE(num_cells_host_out && num_samples_out && levels_done_out,
                "SamplingOp got a null pointer");
  int32_t host[kMaxLevels * kLevelWords];
  int rc = read_report((cudaStream_t)stream, (size_t)levels * kLevelWords * 4, host);
  if (rc) return rc;
  tfgpc_cell_grid g{};
  g.D = D;
  g.max_cells = max_cells;
  *levels_done_out = 0;
  for (int l = 0; l < levels; ++l) {
    rc = level_report(host + l * kLevelWords, g, num_cells_host_out + l * D, num_samples_out + l);
    if (rc == TFGPC_ENOMEM && l > 0) break;       // (the levels before it stand)
    if (rc) return rc;
    *levels_done_out = l + 1;
  }
  return TFGPC_OK;
}

extern "C" int tfgpc_debug_sampling_barrier(void* stream, void* ws, size_t ws_bytes,
                                            unsigned limit_us, int late_block, int late_at,
                                            int working, int* reported_out, int* gave_up_out) {
  TFGPC_REQUIRE(ws && reported_out && gave_up_out && ws_bytes >= 256 && (uintptr_t)ws % 256 == 0,
                "debug_sampling_barrier expects a 256-byte aligned workspace of 256 bytes");
  TFGPC_REQUIRE(limit_us >= 1 && limit_us <= 100000,
                "debug_sampling_barrier expects a limit between 1 us and 100 ms");
  cudaStream_t st = (cudaStream_t)stream;
  unsigned* words = (unsigned*)ws;
  TFGPC_CUDA(cudaMemsetAsync(words, 0, 7 * sizeof(unsigned), st));
  unsigned long long period_ns = (unsigned long long)limit_us * 500ull;
  void* args[] = {&words, &late_block, &late_at, &working, &period_ns};
  TFGPC_CUDA(cudaLaunchCooperativeKernel(barrier_probe_kernel, dim3(16), dim3(32), args, 0, st));
  int back[6];
  int rc = read_small(st, words, sizeof(back), back);
  if (rc) return rc;
  *reported_out = back[4];
  *gave_up_out = back[5];
  return TFGPC_OK;
}
