// Radius search and density estimate on the cell table of a grid (cells.cuh).
//
// All samples of a cell have the same candidates, the points of its 3^(D-1) tubes.  A
// warp takes up to 32 consecutive samples and, cell by cell among them, loads the
// candidates into registers (kSteps per lane) and tests them against the cell's samples
// one after the other: 32 tests per step and sample for about ten instructions (two
// candidates per packed fp32x2 operation), against some forty-five with one sample per
// warp and a loop over its tubes, which left a quarter of the lanes idle besides (a
// tube of a uniform cloud with 32 neighbors per point holds 23 candidates).  The passes
// are bound by issue slots, the fill pass by its output as well.
#include "cell_grid.cuh"

namespace tfgpc {
namespace {

constexpr int kThreads = 128;
constexpr int kMaxSpan = 16;    // samples of one warp

// What stands at the samples: mode 0 arrays of the caller; 1 the grid's own points in
// their unsorted order, visited in the sorted one; 2 the sorted points.
struct SampleSource {
  int mode;
  const float* samples;
  const int32_t* batch_ids;
};

template <int D>
struct Sample {
  float p[D];
  int cell[D];
  int batch;
  int key;        // of its cell, -1: no sample, or a batch id outside the batch
  int id;         // row of its results, -1: no sample
};

template <int D>
__device__ __forceinline__ void load_point(const CellsView& c, int64_t j, float* p, int* index) {
  if (D <= 3) {
    const float4 v = ld_global(c.packed + j);
    p[0] = v.x; p[1] = v.y;
    if (D == 3) p[D - 1] = v.z;
    *index = __float_as_int(v.w);
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) p[d] = ld_global(c.points + j * D + d);
    *index = ld_global(c.indices + j);
  }
}

template <int D>
__device__ __forceinline__ Sample<D> load_sample(const CellsView& c, const SampleSource& src,
                                                 int64_t v, bool live, const Grid<D>& g) {
  Sample<D> s;
  s.id = -1;
  s.key = -1;
  s.batch = -1;
#pragma unroll
  for (int d = 0; d < D; ++d) { s.p[d] = 0.0f; s.cell[d] = 0; }
  if (!live) return s;
  if (src.mode == 0) {
    s.id = (int)v;
    s.batch = ld_global(src.batch_ids + v);
#pragma unroll
    for (int d = 0; d < D; ++d) s.p[d] = ld_global(src.samples + v * D + d);
  } else {
    int index;
    load_point<D>(c, v, s.p, &index);
    s.id = src.mode == 1 ? index : (int)v;
    s.batch = ld_global(c.batch_ids + v);
  }
  if (s.batch < 0 || s.batch >= c.batch_size) return s;
  float smin[D];
#pragma unroll
  for (int d = 0; d < D; ++d) smin[d] = ld_global(c.scaled_min + (int64_t)s.batch * D + d);
  cell_of<D>(s.p, smin, g, s.cell);
  s.key = (int)key_of<D>(s.cell, g, s.batch);
  return s;
}

// Two fp32 operations per instruction, each rounded like the scalar one.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

enum { kCount = 0, kFill = 1, kDensity = 2, kFillBoth = 3 };

// *p = (a, b) under a condition, without a branch.  With two nested ones per candidate, and a
// look at whether the second list is wanted, the fill of one list took, us, before -> now: 665 -> 585
// on surfaces with 260 neighbors, 164 -> 150 and 211 -> 193 on 524 288 uniform points with 34 and 48,
// 85 -> 71 in two dimensions.
__device__ __forceinline__ void store_if(int2* p, int a, int b, bool ok) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n@p st.global.v2.u32 [%0], {%1, %2};\n}"
               ::"l"(p), "r"(a), "r"(b), "r"((uint32_t)ok) : "memory");
}

struct WalkArgs {
  CellsView c;
  SampleSource src;
  int64_t ns;
  int span;                     // samples per warp, 1 to kMaxSpan
  const float* inv_radii;
  int limit;                    // neighbors kept per sample
  int32_t* counts;              // kCount: [ns]
  const int32_t* ranges;        // the fills: [ns]
  int2* neigh;                  // the fills: [M]
  int2* ids;                    // kFillBoth: [M]
  const float* inv_bw;          // kDensity
  int bw_mode;
  float* density;               // kDensity: [ns]
  float4* packed;               // kDensity, D == 3: [ns] (point, 1 / density), or null
};

// kCount: number of neighbors.  kFill: the pairs in ascending sorted index, kFillBoth: also
// with the neighbor's original index.  kDensity: ComputePdf (compute_pdf_kernels.cu.cc:
// 107-128) over the points within the radius; the exponents of the D Gaussians are
// added before the one exponential, ex2.approx.  Their factor is kept in two parts and
// the terms are added with the norm of the density on them, rounded once: relative
// error against 64 bits 2.5e-8 to 6.7e-8 over 2 to 4 dimensions and bandwidths of 0.05
// to 1, where one expf per dimension over the list gives 4.6e-8 to 11e-8 (and the same
// sum with a factor of one part and the norm applied at the end up to 8.2e-8).  With expf
// in its place the pass loses 5 % of search and density on surfaces and gains nothing.
// The distance test is the reference's: t_d = (s_d - p_d) * inv_r_d, the fma chain from
// t_0 * t_0, sqrtf(d2) < 1 (count_neighbors_kernels.cu.cc:84-85), which a correctly
// rounded square root decides like d2 < 1.
template <int D, int MODE>
__global__ void
// (the fills' registers: given no bound, that of one list spills at 72, that of two takes 86)
__launch_bounds__(kThreads, MODE == kFill ? 1 : MODE == kFillBoth && D == 3 ? 6 : 0)
cells_walk_kernel(WalkArgs a) {
  chain_enter();
  constexpr int kSteps = D <= 3 ? 8 : 4;     // candidates per lane and round
  constexpr bool kFills = MODE == kFill || MODE == kFillBoth;
  constexpr int kTubes = num_tubes<D>();
  constexpr int kTop = kTubes > 16 ? 16 : kTubes > 8 ? 8 : kTubes > 4 ? 4 : 2;
  const CellsView& c = a.c;
  const int lane = lane_id();
  const int64_t v0 = (((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5) * a.span;
  if (v0 >= a.ns) return;
  const Grid<D> g = load_grid<D>(c.num_cells, c.inv_cell);
  const int total = total_cells<D>(g.nc, c.batch_size);
  if (total == 0) return;        // (a grid that got no cells: the call fails)
  float radius[D];       // its inverse
  f32x2 inv_r[D], scale[D], scale_lo[D];
  double norm_exact = 1.0;
  bool isotropic = true;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float r = ld_global(a.inv_radii + d);
    radius[d] = r;
    inv_r[d] = pack2(r, r);
    if (MODE == kDensity) {
      const float bw = a.bw_mode == 1 ? sqrtf((float)c.n) : ld_global(a.inv_bw + d);
      // of a base-2 exponential, in two parts: rounded once it would shift all
      // exponents of a sample the same way
      const double factor = (double)bw * bw * (-0.5 * 1.4426950408889634);
      const float hi = (float)factor, lo = (float)(factor - (double)hi);
      scale[d] = pack2(hi, hi);
      scale_lo[d] = pack2(lo, lo);
      norm_exact *= bw * 0.3989422804014327;
      isotropic = isotropic && scale[d] == scale[0] && scale_lo[d] == scale_lo[0];
    }
  }
  const float norm = (float)norm_exact;
  const bool live = lane < a.span && v0 + lane < a.ns;
  const Sample<D> s = load_sample<D>(c, a.src, v0 + lane, live, g);
  int my_count = 0, my_begin = 0;
  float my_density = 0.0f;
  if (kFills && s.id > 0) my_begin = ld_global(a.ranges + s.id - 1);
  unsigned open = __ballot_sync(0xffffffffu, s.key >= 0);
  while (open) {
    // the samples of one cell
    const int leader = __ffs(open) - 1;
    const int leader_key = __shfl_sync(0xffffffffu, s.key, leader);
    const unsigned members = __ballot_sync(0xffffffffu, s.key == leader_key);
    open &= ~members;
    int cell[D];
#pragma unroll
    for (int d = 0; d < D; ++d) cell[d] = __shfl_sync(0xffffffffu, s.cell[d], leader);
    const int batch = __shfl_sync(0xffffffffu, s.batch, leader);
    for (int tube0 = 0; tube0 < kTubes; tube0 += 32) {
      // lane t: the t-th tube in ascending sorted index, and how many candidates come before
      int2 r = make_int2(0, 0);
      if (tube0 + lane < kTubes)
        r = tube_points<D>(kTubes - 1 - (tube0 + lane), cell, batch, g.nc, total, c.start);
      int before = r.y - r.x;     // inclusive running count
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += y;
      }
      const int candidates = __shfl_sync(0xffffffffu, before, 31);
      const int offset = r.y - before;   // sorted index of candidate i of this tube: i + offset
      for (int base = 0; base < candidates; base += 32 * kSteps) {
        const int steps = (min(candidates - base, 32 * kSteps) + 31) >> 5;
        f32x2 np[D][kSteps / 2];         // negated coordinates of the lane's candidates
        int at[kSteps], index[kSteps];
#pragma unroll
        for (int k = 0; k < kSteps; k += 2) {
          // (few candidates: half the places stay empty.  524 288 points with 12 neighbors, three
          // dimensions: density 131 -> 108 us, list 144 -> 121; surfaces list 411 -> 400.  Count and
          // two lists gain as much there and lose 2 to 5 % with 34 neighbors and on surfaces; a branch
          // per pair of steps costs small clouds more than it saves, 10.6 -> 11.6 us, and four
          // dimensions 3 % here too)
          if ((MODE == kDensity || MODE == kFill) && D <= 3 && k >= kSteps / 2 && steps <= kSteps / 2)
            continue;
          float p[2][D];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int i = base + 32 * (k + u) + lane;
            int t = 0;
#pragma unroll
            for (int o = kTop; o > 0; o >>= 1) {
              const int y = __shfl_sync(0xffffffffu, before, t + o - 1);
              if (y <= i) t += o;
            }
            at[k + u] = i + __shfl_sync(0xffffffffu, offset, t & 31);
            index[k + u] = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) p[u][d] = INFINITY;    // too far away for any sample
            if (i < candidates) load_point<D>(c, at[k + u], p[u], &index[k + u]);
          }
#pragma unroll
          for (int d = 0; d < D; ++d) np[d][k / 2] = pack2(-p[0][d], -p[1][d]);
        }
        for (unsigned todo = members; todo; todo &= todo - 1u) {
          const int who = __ffs(todo) - 1;
          float one[D];
          f32x2 sp[D];
#pragma unroll
          for (int d = 0; d < D; ++d) {
            one[d] = __shfl_sync(0xffffffffu, s.p[d], who);
            sp[d] = pack2(one[d], one[d]);
          }
          int n_hit = 0, id = 0, begin = 0;
          float acc = 0.0f;
          if (kFills) {
            n_hit = __shfl_sync(0xffffffffu, my_count, who);
            id = __shfl_sync(0xffffffffu, s.id, who);
            begin = __shfl_sync(0xffffffffu, my_begin, who);
          }
#pragma unroll
          for (int k = 0; k < kSteps; k += 2) {
            if (MODE == kCount && D <= 3 && k < steps) {
              // One by one: where nothing follows the test the packed forms, which keep the
              // multiply-add pipes busy longer, are the slower ones.  Surfaces 366 -> 331 us, 524 288
              // uniform points with 34 neighbors 102 -> 96, with 16 105 and 105; four dimensions
              // 179 and 186.  (Density and fill of surfaces so: 503 -> 532, 665 -> 685.)
              float x[2][D];
#pragma unroll
              for (int d = 0; d < D; ++d) unpack2(np[d][k / 2], x[0][d], x[1][d]);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                float d2 = 0.0f;
#pragma unroll
                for (int d = 0; d < D; ++d) {
                  const float t = __fmul_rn(__fadd_rn(one[d], x[u][d]), radius[d]);
                  d2 = d == 0 ? __fmul_rn(t, t) : __fmaf_rn(t, t, d2);
                }
                n_hit += d2 < 1.0f;
              }
            } else if (k < steps) {
              f32x2 t2[D], d2;
#pragma unroll
              for (int d = 0; d < D; ++d) {
                t2[d] = mul2(add2(sp[d], np[d][k / 2]), inv_r[d]);
                d2 = d == 0 ? mul2(t2[d], t2[d]) : fma2(t2[d], t2[d], d2);
              }
              float dist[2], e[2];
              unpack2(d2, dist[0], dist[1]);
              if (MODE == kDensity) {
                f32x2 e2;
                if (isotropic) {
                  e2 = fma2(d2, scale[0], mul2(d2, scale_lo[0]));
                } else {
#pragma unroll
                  for (int d = 0; d < D; ++d) {
                    const f32x2 sq = mul2(t2[d], t2[d]);
                    const f32x2 low = d == 0 ? mul2(sq, scale_lo[d]) : fma2(sq, scale_lo[d], e2);
                    e2 = fma2(sq, scale[d], low);
                  }
                }
                unpack2(e2, e[0], e[1]);
              }
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const bool hit = dist[u] < 1.0f;
                if (MODE == kCount) n_hit += hit;
                if (kFills) {
                  const unsigned m = __ballot_sync(0xffffffffu, hit);
                  const int pos = n_hit + __popc(m & ((1u << lane) - 1u));
                  const bool ok = hit && pos < a.limit;
                  store_if(a.neigh + begin + (unsigned)pos, at[k + u], id, ok);
                  if (MODE == kFillBoth) store_if(a.ids + begin + (unsigned)pos, index[k + u], id, ok);
                  n_hit += __popc(m);
                }
                if (MODE == kDensity && hit) acc = fmaf(exp2_approx(e[u]), norm, acc);
              }
            }
          }
          if (MODE == kCount) {
            n_hit = __reduce_add_sync(0xffffffffu, n_hit);
            if (lane == who) my_count += n_hit;
          }
          if (kFills && lane == who) my_count = n_hit;
          if (MODE == kDensity) {
            acc = warp_sum(acc);
            if (lane == who) my_density += acc;
          }
        }
      }
    }
  }
  if (MODE == kCount && s.id >= 0) a.counts[s.id] = min(my_count, a.limit);
  if (MODE == kDensity && s.id >= 0) {
    const float density = (float)(my_density * (norm_exact / norm));
    a.density[s.id] = density;
    if (D == 3 && a.packed)
      a.packed[s.id] = make_float4(s.p[0], s.p[1], s.p[D - 1], 1.0f / density);
  }
}

// ---- densities of the grid's own points by half the tests ---------------------------
//
// The relation is symmetric, and so are the rounded differences: a pair is worked out once,
// at the point that comes first in the sorted order, and counts for both.

// A sum of exponentials as a whole number: sums of such numbers come out the same in any order.
// (A density of a point is at least the one of itself, the sum of a density 1: 2^-32 of that is
// 1/256 of the float's last place.)
constexpr float kDensityUnit = 4294967296.0f;
__device__ __forceinline__ void add_density(unsigned long long* sums, int j, float v) {
  atomicAdd(sums + j, __float2ull_rn(v * kDensityUnit));
}

struct DensityScale {
  float hi, lo;
};
__device__ __forceinline__ float density_bandwidth(const WalkArgs& a, int d) {
  return a.bw_mode == 1 ? sqrtf((float)a.c.n) : ld_global(a.inv_bw + d);
}
__device__ __forceinline__ DensityScale density_scale(float bw) {
  const double factor = (double)bw * bw * (-0.5 * 1.4426950408889634);
  const float hi = (float)factor;
  return DensityScale{hi, (float)(factor - (double)hi)};
}

// The walk of cells_walk_kernel over the sorted points, with the candidates behind a cell's first
// sample only: a lane keeps the sums of its candidates over the cell's samples beside theirs.
// Two tests in some 19 instructions count for four, where two of kDensity take 17.  530 366 points
// of surfaces (260 neighbors): 529 -> 320 us; the rule and more figures are at
// tfgpc_cells_density_workspace_bytes.  Error against 64 bits, rms over 2 to 4 dimensions and
// bandwidths of 0.05 to 1: 2.0e-8 to 5.3e-8, where kDensity has 1.8e-8 to 7.4e-8 (it rounds every
// term onto one sum; here half of them come in sums of at most 16, as whole numbers).  Bound by issue
// slots like the other walks; 16 more pairs of sums and places per lane, 78 registers.
template <int D>
__global__ void __launch_bounds__(kThreads)
cells_density_half_kernel(WalkArgs a, unsigned long long* sums) {
  chain_enter();
  constexpr int kSteps = D <= 3 ? 8 : 4;
  constexpr int kTubes = num_tubes<D>();
  constexpr int kTop = kTubes > 16 ? 16 : kTubes > 8 ? 8 : kTubes > 4 ? 4 : 2;
  const CellsView& c = a.c;
  const int lane = lane_id();
  const int64_t v0 = (((int64_t)blockIdx.x * kThreads + threadIdx.x) >> 5) * a.span;
  if (v0 >= a.ns) return;
  const Grid<D> g = load_grid<D>(c.num_cells, c.inv_cell);
  const int total = total_cells<D>(g.nc, c.batch_size);
  if (total == 0) return;
  f32x2 inv_r[D], scale[D], scale_lo[D];
  bool isotropic = true;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float r = ld_global(a.inv_radii + d);
    inv_r[d] = pack2(r, r);
    const DensityScale f = density_scale(density_bandwidth(a, d));
    scale[d] = pack2(f.hi, f.hi);
    scale_lo[d] = pack2(f.lo, f.lo);
    isotropic = isotropic && scale[d] == scale[0] && scale_lo[d] == scale_lo[0];
  }
  const bool live = lane < a.span && v0 + lane < a.ns;
  const Sample<D> s = load_sample<D>(c, SampleSource{2, nullptr, nullptr}, v0 + lane, live, g);
  float my_density = 0.0f;
  if (s.key >= 0) {          // the point itself, unless it is no neighbor of itself (no number)
    bool finite = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      float r, unused;
      unpack2(inv_r[d], r, unused);
      finite = finite && (s.p[d] - s.p[d]) * r == 0.0f;
    }
    my_density = finite ? 1.0f : 0.0f;
  }
  unsigned open = __ballot_sync(0xffffffffu, s.key >= 0);
  while (open) {
    const int leader = __ffs(open) - 1;
    const int leader_key = __shfl_sync(0xffffffffu, s.key, leader);
    const unsigned members = __ballot_sync(0xffffffffu, s.key == leader_key);
    open &= ~members;
    int cell[D];
#pragma unroll
    for (int d = 0; d < D; ++d) cell[d] = __shfl_sync(0xffffffffu, s.cell[d], leader);
    const int batch = __shfl_sync(0xffffffffu, s.batch, leader);
    const int after = (int)v0 + leader + 1;
    for (int tube0 = 0; tube0 < kTubes; tube0 += 32) {
      int2 r = make_int2(0, 0);
      if (tube0 + lane < kTubes)
        r = tube_points<D>(kTubes - 1 - (tube0 + lane), cell, batch, g.nc, total, c.start);
      r.x = min(max(r.x, after), r.y);       // (behind the cell's first sample only)
      int before = r.y - r.x;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += y;
      }
      const int candidates = __shfl_sync(0xffffffffu, before, 31);
      const int offset = r.y - before;
      for (int base = 0; base < candidates; base += 32 * kSteps) {
        const int steps = (min(candidates - base, 32 * kSteps) + 31) >> 5;
        f32x2 np[D][kSteps / 2], sum2[kSteps / 2];
        int at[kSteps];
#pragma unroll
        for (int k = 0; k < kSteps; k += 2) {
          if (k >= steps) continue;
          float p[2][D];
          sum2[k / 2] = 0ull;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int i = base + 32 * (k + u) + lane;
            int t = 0;
#pragma unroll
            for (int o = kTop; o > 0; o >>= 1) {
              const int y = __shfl_sync(0xffffffffu, before, t + o - 1);
              if (y <= i) t += o;
            }
            at[k + u] = i + __shfl_sync(0xffffffffu, offset, t & 31);
            int unused;
#pragma unroll
            for (int d = 0; d < D; ++d) p[u][d] = INFINITY;
            if (i < candidates) load_point<D>(c, at[k + u], p[u], &unused);
          }
#pragma unroll
          for (int d = 0; d < D; ++d) np[d][k / 2] = pack2(-p[0][d], -p[1][d]);
        }
        for (unsigned todo = members; todo; todo &= todo - 1u) {
          const int who = __ffs(todo) - 1;
          const int self = (int)v0 + who;
          f32x2 sp[D], acc2 = 0ull;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const float x = __shfl_sync(0xffffffffu, s.p[d], who);
            sp[d] = pack2(x, x);
          }
#pragma unroll
          for (int k = 0; k < kSteps; k += 2) {
            if (k < steps) {
              f32x2 t2[D], d2, e2;
#pragma unroll
              for (int d = 0; d < D; ++d) {
                t2[d] = mul2(add2(sp[d], np[d][k / 2]), inv_r[d]);
                d2 = d == 0 ? mul2(t2[d], t2[d]) : fma2(t2[d], t2[d], d2);
              }
              if (isotropic) {
                e2 = fma2(d2, scale[0], mul2(d2, scale_lo[0]));
              } else {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                  const f32x2 sq = mul2(t2[d], t2[d]);
                  const f32x2 low = d == 0 ? mul2(sq, scale_lo[d]) : fma2(sq, scale_lo[d], e2);
                  e2 = fma2(sq, scale[d], low);
                }
              }
              float dist[2], e[2];
              unpack2(d2, dist[0], dist[1]);
              unpack2(e2, e[0], e[1]);
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                bool hit = dist[u] < 1.0f;
                // (the sample's own cell begins the candidates: fewer than 16 of its warp's)
                if (k + u == 0) hit = hit && at[0] > self;
                e[u] = hit ? exp2_approx(e[u]) : 0.0f;
              }
              const f32x2 both = pack2(e[0], e[1]);
              acc2 = add2(acc2, both);
              sum2[k / 2] = add2(sum2[k / 2], both);
            }
          }
          float x, y;
          unpack2(acc2, x, y);
          x = warp_sum(x + y);
          if (lane == who) my_density += x;
        }
#pragma unroll
        for (int k = 0; k < kSteps; k += 2) {
          if (k < steps) {
            float x, y;
            unpack2(sum2[k / 2], x, y);
            if (x > 0.0f) add_density(sums, at[k], x);
            if (y > 0.0f) add_density(sums, at[k + 1], y);
          }
        }
      }
    }
  }
  if (my_density > 0.0f) add_density(sums, (int)v0 + lane, my_density);
}

// The densities from the sums: of sorted point v to its original place (mode 1) or to v (2).
template <int D>
__global__ void __launch_bounds__(256)
density_of_sums_kernel(WalkArgs a, const unsigned long long* sums) {
  chain_enter();
  const int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (v >= a.ns) return;
  if (total_cells<D>(load_grid<D>(a.c.num_cells, a.c.inv_cell).nc, a.c.batch_size) == 0)
    return;                  // (a grid that got no cells: its sorted arrays hold nothing)
  double norm = 1.0 / (double)kDensityUnit;
  float worst = 0.0f;        // (no number where an exponent's factor is none)
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float bw = density_bandwidth(a, d);
    const DensityScale f = density_scale(bw);
    worst += f.hi * 0.0f + f.lo * 0.0f;
    norm *= bw * 0.3989422804014327;
  }
  const int64_t row = a.src.mode == 1 ? ld_global(a.c.indices + v) : v;
  a.density[row] = (float)((double)ld_global(sums + v) * norm) + worst;
}

// Samples per warp: more of them share the candidates of a cell (a cell of a uniform
// cloud holds seven points), fewer spread dense regions over the SMs.  Fill pass at
// 32 / 16 / 8 / 4: 176 / 177 / 192 / 231 us on uniform clouds with 32 neighbors, 776 /
// 662 / 635 / 683 us on surfaces with 280; below 32 warps per SM it is the number of
// warps that decides.
int samples_per_warp(int64_t ns) {
  const int64_t s = ns / ((int64_t)sm_count() * 32);
  return (int)(s < 1 ? 1 : s > kMaxSpan ? kMaxSpan : s);
}

template <int MODE>
int launch_walk(cudaStream_t st, const char* name, int D, WalkArgs a) {
  a.span = samples_per_warp(a.ns);
  const int64_t warps = (a.ns + a.span - 1) / a.span;
  ProfScope prof(st, name);
  TFGPC_DIM_SWITCH(D, TFGPC_CUDA(launch_chained(st, blocks_for(warps, kThreads / 32), kThreads, 0,
      cells_walk_kernel<kD, MODE>, a)));
  return TFGPC_OK;
}

WalkArgs walk_args(const tfgpc_cell_grid& g, const SampleSource& src, int64_t ns,
                   const float* inv_radii, int max_neighs) {
  WalkArgs a{};
  a.c = view_of(g);
  a.src = src;
  a.ns = ns;
  a.inv_radii = inv_radii;
  a.limit = max_neighs > 0 ? max_neighs : INT32_MAX;
  return a;
}

}  // namespace

int check_cell_grid(const char* op, const tfgpc_cell_grid* g) {
  TFGPC_REQUIRE(g != nullptr, "%s got a null grid", op);
  TFGPC_REQUIRE(valid_dims(g->D), "%s expects a valid number of dimension (got %d)", op, g->D);
  TFGPC_REQUIRE(g->n > 0 && g->n < (int64_t)INT32_MAX && g->batch_size > 0 &&
                g->batch_size < (int64_t)INT32_MAX,
                "%s expects 0 < n, 0 < batch size, both below 2^31", op);
  TFGPC_REQUIRE(g->max_cells >= 1 && table_cells(g->D, g->batch_size, g->max_cells) > 0,
                "%s expects a grid whose cell table is small enough (tfgpc_cell_table_elems)", op);
  TFGPC_REQUIRE(g->aabb_min && g->aabb_max && g->num_cells && g->scaled_aabb_min &&
                g->inv_cell_sizes && g->keys && g->sorted_indices && g->sorted_keys &&
                g->sorted_points && g->sorted_batch_ids && (g->D > 3 || g->packed) &&
                g->cell_start && g->ds, "%s got a null pointer", op);
  TFGPC_REQUIRE((uintptr_t)g->packed % 16 == 0, "%s expects a 16-byte aligned packed table", op);
  return TFGPC_OK;
}

namespace {

int check_samples(const char* op, const tfgpc_cell_grid* g, int64_t ns, const float* samples,
                  const int32_t* sbatch, int mode, int max_neighs) {
  TFGPC_REQUIRE(ns >= 0 && ns < (int64_t)INT32_MAX && max_neighs >= 0,
                "%s expects 0 <= ns < 2^31 and max_neighs >= 0", op);
  TFGPC_REQUIRE(mode >= 0 && mode <= 2, "%s expects samples_are_points 0, 1 or 2", op);
  TFGPC_REQUIRE(mode != 0 || ns == 0 || (samples && sbatch), "%s got a null pointer", op);
  TFGPC_REQUIRE(mode == 0 || ns == g->n || ns == 0,
                "%s expects as many samples as points when the samples are the points", op);
  return TFGPC_OK;
}

// Counts and their scan; the total goes to `total` and to the report page.  room: where the
// counts may stand before they are scanned, [ns], or null.
int count_and_scan(cudaStream_t st, const tfgpc_cell_grid& g, const float* inv_radii, int64_t ns,
                   const SampleSource& src, int max_neighs, int32_t* ranges, int64_t* sums,
                   int64_t* total, int32_t* page, int32_t* room) {
  WalkArgs a = walk_args(g, src, ns, inv_radii, max_neighs);
  const bool apart = room && ns <= kDirectScan;
  a.counts = apart ? room : ranges;
  int rc = launch_walk<kCount>(st, "find_neighbors_count", g.D, a);
  if (rc) return rc;
  ScanReport rep;
  rep.dst = page + kReportTotal;
  if (apart) return inclusive_scan_apart(st, room, ranges, ns, total, rep);
  return inclusive_scan_i32(st, ranges, ranges, ns, sums, total, rep);
}

// Waits for the report (marked: see mark_report) and turns it into the outputs of a
// blocking entry.
int finish_report(cudaStream_t st, int D, int max_cells, bool with_total,
                  int32_t* num_cells_host_out, int64_t* total_out, bool marked = false) {
  int32_t host[kReportWords];
  int rc = marked ? read_marked_report(sizeof(host), host) : read_report(st, sizeof(host), host);
  if (rc) return rc;
  for (int d = 0; num_cells_host_out && d < D; ++d) num_cells_host_out[d] = host[d];
  if (num_cells_host_out && host[TFGPC_MAX_DIMS])
    return fail(TFGPC_ENOMEM, "GridNeighborhood: the grid needs more than max_cells = %d cells in "
                "a dimension; repeat the call with a larger bound", max_cells);
  if (!with_total) return TFGPC_OK;
  const int64_t total = (int64_t)(uint32_t)host[kReportTotal] |
                        ((int64_t)host[kReportTotal + 1] << 32);
  if (total > (int64_t)INT32_MAX)
    return fail(TFGPC_EINVAL, "FindNeighbors found %lld pairs; the int32 ranges of the op "
                "contract hold at most 2^31-1", (long long)total);
  *total_out = total;
  return TFGPC_OK;
}

// The density at every point in its own order, and the table of tfgpc_pack_points_density
// (or null).
struct DensityRequest {
  const float* inv_bandwidth;
  int mode;
  float* pdf;
  float4* packed;
};

// sums: [n] zeros, for the densities of the grid's own points (without a packed table), or null.
int enqueue_density(cudaStream_t st, const tfgpc_cell_grid& g, const SampleSource& src, int64_t ns,
                    const float* inv_radii, const DensityRequest& d, unsigned long long* sums) {
  WalkArgs a = walk_args(g, src, ns, inv_radii, 0);
  a.inv_bw = d.inv_bandwidth;
  a.bw_mode = d.mode;
  a.density = d.pdf;
  a.packed = d.packed;
  if (sums) {
    a.span = samples_per_warp(ns);
    const unsigned blocks = blocks_for((ns + a.span - 1) / a.span, kThreads / 32);
    ProfScope prof(st, "compute_pdf");
    TFGPC_DIM_SWITCH(g.D,
        TFGPC_CUDA(launch_chained(st, blocks, kThreads, 0, cells_density_half_kernel<kD>, a, sums));
        TFGPC_CUDA(launch_chained(st, blocks_for(ns, 256), 256, 0, density_of_sums_kernel<kD>, a,
                                  sums)));
    return TFGPC_OK;
  }
  return launch_walk<kDensity>(st, "compute_pdf", g.D, a);
}

int grid_neighborhood(cudaStream_t st, const tfgpc_cell_grid* grid, const float* points,
                      const int32_t* batch_ids, const float* cell_sizes,
                      const int32_t* num_cells_in, const float* inv_radii, int64_t ns,
                      const float* samples, const int32_t* samples_batch_ids,
                      int samples_are_points, int max_neighs, int32_t* ranges_out,
                      const DensityRequest* density, void* ws, size_t ws_bytes,
                      int32_t* num_cells_host_out, int64_t* total_out) {
  int rc = check_cell_grid("GridNeighborhood", grid);
  if (rc) return rc;
  const tfgpc_cell_grid& g = *grid;
  rc = check_samples("GridNeighborhood", grid, ns, samples, samples_batch_ids,
                     samples_are_points, max_neighs);
  if (rc) return rc;
  TFGPC_REQUIRE(points && batch_ids && cell_sizes && ws && num_cells_host_out && total_out &&
                (ns == 0 || (ranges_out && inv_radii)), "GridNeighborhood got a null pointer");
  TFGPC_REQUIRE(!density || ((density->mode == 0 || density->mode == 1) && density->pdf &&
                             inv_radii && (density->mode == 1 || density->inv_bandwidth) &&
                             (!density->packed || g.D == 3) && (uintptr_t)density->packed % 16 == 0),
                "GridNeighborhood: densities need mode 0 or 1, radii, a bandwidth and an output "
                "(packed: 16-byte aligned, three dimensions)");
  TFGPC_REQUIRE(num_cells_in != g.num_cells,
                "GridNeighborhood expects the given cell counts outside the output array");
  for (int d = 0; d < g.D; ++d)
    TFGPC_REQUIRE(cell_sizes[d] > 0.0f, "GridNeighborhood expects positive cell sizes");
  if (ws_bytes < tfgpc_cell_grid_workspace_bytes(g.D, g.n, ns, g.batch_size, g.max_cells))
    return fail(TFGPC_ENOMEM, "GridNeighborhood workspace too small");
  CellGridWs w = carve_cell_grid(ws, g.n, ns, g.D, g.batch_size, g.max_cells);
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  *total_out = 0;
  rc = cell_grid_build(st, g, points, batch_ids, cell_sizes, num_cells_in, w, (int32_t*)page);
  if (rc) return rc;
  if (ns > 0) {
    rc = count_and_scan(st, g, inv_radii, ns,
                        SampleSource{samples_are_points, samples, samples_batch_ids}, max_neighs,
                        ranges_out, w.sums, w.total, (int32_t*)page,
                        ns <= g.n ? w.arrival : nullptr);     // (free once the grid is built)
    if (rc) return rc;
  }
  if (density) {
    rc = mark_report(st);
    if (!rc) rc = enqueue_density(st, g, SampleSource{1, nullptr, nullptr}, g.n, inv_radii, *density,
                                  nullptr);
    if (rc) return rc;
  }
  return finish_report(st, g.D, g.max_cells, ns > 0, num_cells_host_out, total_out, density != nullptr);
}

}  // namespace
}  // namespace tfgpc

using namespace tfgpc;

extern "C" size_t tfgpc_cell_table_elems(int D, int64_t batch_size, int max_cells) {
  if (!valid_dims(D) || batch_size <= 0 || max_cells <= 0) return 0;
  const int64_t cells = table_cells(D, batch_size, max_cells);
  return cells > 0 ? (size_t)cells + 3 : 0;
}

extern "C" size_t tfgpc_cell_grid_workspace_bytes(int D, int64_t n, int64_t ns, int64_t batch_size,
                                                  int max_cells) {
  if (!valid_dims(D) || n < 0 || ns < 0 || batch_size <= 0 || max_cells <= 0) return 0;
  return carve_cell_grid(nullptr, n, ns, D, batch_size, max_cells).bytes + 256;
}

extern "C" int tfgpc_cell_grid_neighborhood(
    void* stream, const tfgpc_cell_grid* grid, const float* points, const int32_t* batch_ids,
    const float* cell_sizes, const int32_t* num_cells_in, const float* inv_radii, int64_t ns,
    const float* samples, const int32_t* samples_batch_ids, int samples_are_points,
    int max_neighs, int32_t* ranges_out, void* ws, size_t ws_bytes, int32_t* num_cells_host_out,
    int64_t* total_out) {
  return grid_neighborhood((cudaStream_t)stream, grid, points, batch_ids, cell_sizes, num_cells_in,
                           inv_radii, ns, samples, samples_batch_ids, samples_are_points,
                           max_neighs, ranges_out, nullptr, ws, ws_bytes, num_cells_host_out,
                           total_out);
}

extern "C" int tfgpc_cell_grid_neighborhood_pdf(
    void* stream, const tfgpc_cell_grid* grid, const float* points, const int32_t* batch_ids,
    const float* cell_sizes, const int32_t* num_cells_in, const float* inv_radii, int64_t ns,
    const float* samples, const int32_t* samples_batch_ids, int samples_are_points,
    int max_neighs, int32_t* ranges_out, const float* inv_bandwidth, int pdf_mode, float* pdf_out,
    float* packed_out, void* ws, size_t ws_bytes, int32_t* num_cells_host_out,
    int64_t* total_out) {
  const DensityRequest density{inv_bandwidth, pdf_mode, pdf_out, (float4*)packed_out};
  return grid_neighborhood((cudaStream_t)stream, grid, points, batch_ids, cell_sizes, num_cells_in,
                           inv_radii, ns, samples, samples_batch_ids, samples_are_points,
                           max_neighs, ranges_out, &density, ws, ws_bytes, num_cells_host_out,
                           total_out);
}

extern "C" int tfgpc_cells_count(void* stream, const tfgpc_cell_grid* grid, const float* inv_radii,
                                 int64_t ns, const float* samples,
                                 const int32_t* samples_batch_ids, int samples_are_points,
                                 int max_neighs, int32_t* ranges_out, void* ws, size_t ws_bytes,
                                 int64_t* total_out) {
  int rc = check_cell_grid("FindNeighbors", grid);
  if (rc) return rc;
  rc = check_samples("FindNeighbors", grid, ns, samples, samples_batch_ids, samples_are_points,
                     max_neighs);
  if (rc) return rc;
  TFGPC_REQUIRE(total_out, "FindNeighbors got a null pointer");
  *total_out = 0;
  if (ns == 0) return TFGPC_OK;
  TFGPC_REQUIRE(inv_radii && ranges_out && ws, "FindNeighbors got a null pointer");
  if (ws_bytes < tfgpc_find_neighbors_workspace_bytes(ns))
    return fail(TFGPC_ENOMEM, "FindNeighbors workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  int64_t* sums = (int64_t*)ws;
  rc = count_and_scan(st, *grid, inv_radii, ns,
                      SampleSource{samples_are_points, samples, samples_batch_ids}, max_neighs,
                      ranges_out, sums, sums + scan_block_sums_elems(ns), (int32_t*)page,
                      nullptr);
  if (rc) return rc;
  return finish_report(st, grid->D, grid->max_cells, true, nullptr, total_out);
}

extern "C" size_t tfgpc_cells_count_pdf_workspace_bytes(int64_t ns) {
  return ns < 0 ? 0 : align_up(tfgpc_find_neighbors_workspace_bytes(ns), 256) + (size_t)ns * 4;
}

extern "C" int tfgpc_cells_count_pdf(void* stream, const tfgpc_cell_grid* grid,
                                     const float* inv_radii, int64_t ns, const float* samples,
                                     const int32_t* samples_batch_ids, int samples_are_points,
                                     int max_neighs, int32_t* ranges_out,
                                     const float* inv_bandwidth, int pdf_mode, float* pdf_out,
                                     float* packed_out, void* ws, size_t ws_bytes,
                                     int64_t* total_out) {
  int rc = check_cell_grid("FindNeighbors", grid);
  if (rc) return rc;
  rc = check_samples("FindNeighbors", grid, ns, samples, samples_batch_ids, samples_are_points,
                     max_neighs);
  if (rc) return rc;
  TFGPC_REQUIRE(total_out && inv_radii && pdf_out && ws && (uintptr_t)ws % 16 == 0 &&
                (ns == 0 || ranges_out), "FindNeighbors got a null pointer");
  TFGPC_REQUIRE((pdf_mode == 0 || pdf_mode == 1) && (pdf_mode == 1 || inv_bandwidth) &&
                (!packed_out || (grid->D == 3 && (uintptr_t)packed_out % 16 == 0)),
                "FindNeighbors: densities need mode 0 or 1, a bandwidth and an output (packed: "
                "16-byte aligned, three dimensions)");
  if (ws_bytes < tfgpc_cells_count_pdf_workspace_bytes(ns))
    return fail(TFGPC_ENOMEM, "FindNeighbors workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  void* page = nullptr;
  rc = report_page(&page);
  if (rc) return rc;
  *total_out = 0;
  if (ns > 0) {
    int64_t* sums = (int64_t*)ws;
    rc = count_and_scan(st, *grid, inv_radii, ns,
                        SampleSource{samples_are_points, samples, samples_batch_ids}, max_neighs,
                        ranges_out, sums, sums + scan_block_sums_elems(ns), (int32_t*)page,
                        (int32_t*)((char*)ws + align_up(tfgpc_find_neighbors_workspace_bytes(ns), 256)));
    if (rc) return rc;
  }
  rc = mark_report(st);
  if (!rc)
    rc = enqueue_density(st, *grid, SampleSource{1, nullptr, nullptr}, grid->n, inv_radii,
                         DensityRequest{inv_bandwidth, pdf_mode, pdf_out, (float4*)packed_out}, nullptr);
  if (rc) return rc;
  return finish_report(st, grid->D, grid->max_cells, ns > 0, nullptr, total_out, true);
}

extern "C" int tfgpc_cells_fill(void* stream, const tfgpc_cell_grid* grid, const float* inv_radii,
                                int64_t ns, const float* samples,
                                const int32_t* samples_batch_ids, int samples_are_points,
                                int max_neighs, const int32_t* ranges, int64_t total,
                                int32_t* neigh_out, int32_t* ids_out) {
  int rc = check_cell_grid("FindNeighbors", grid);
  if (rc) return rc;
  rc = check_samples("FindNeighbors", grid, ns, samples, samples_batch_ids, samples_are_points,
                     max_neighs);
  if (rc) return rc;
  TFGPC_REQUIRE(total >= 0 && total <= (int64_t)INT32_MAX, "FindNeighbors expects 0 <= total < 2^31");
  if (ns == 0 || total == 0) return TFGPC_OK;
  TFGPC_REQUIRE(inv_radii && ranges && neigh_out, "FindNeighbors got a null pointer");
  WalkArgs a = walk_args(*grid, SampleSource{samples_are_points, samples, samples_batch_ids}, ns,
                         inv_radii, max_neighs);
  a.ranges = ranges;
  a.neigh = (int2*)neigh_out;
  a.ids = (int2*)ids_out;
  if (ids_out)
    return launch_walk<kFillBoth>((cudaStream_t)stream, "find_neighbors_fill_fused", grid->D, a);
  return launch_walk<kFill>((cudaStream_t)stream, "find_neighbors_fill", grid->D, a);
}

namespace {

int cells_density(cudaStream_t st, const tfgpc_cell_grid* grid, const float* inv_radii,
                  const float* inv_bandwidth, int mode, int64_t ns, const float* samples,
                  const int32_t* samples_batch_ids, int samples_are_points, void* ws,
                  size_t ws_bytes, float* pdf_out) {
  int rc = check_cell_grid("ComputePdf", grid);
  if (rc) return rc;
  rc = check_samples("ComputePdf", grid, ns, samples, samples_batch_ids, samples_are_points, 0);
  if (rc) return rc;
  TFGPC_REQUIRE(mode == 0 || mode == 1, "ComputePdf expects mode 0 or 1 (got %d)", mode);
  if (ns == 0) return TFGPC_OK;
  TFGPC_REQUIRE(inv_radii && pdf_out && (mode == 1 || inv_bandwidth), "ComputePdf got a null pointer");
  unsigned long long* sums = nullptr;
  if (ws && samples_are_points != 0) {
    if (ws_bytes < (size_t)ns * 8) return fail(TFGPC_ENOMEM, "ComputePdf workspace too small");
    TFGPC_REQUIRE((uintptr_t)ws % 8 == 0, "ComputePdf expects an 8-byte aligned workspace");
    sums = (unsigned long long*)ws;
    TFGPC_CUDA(cudaMemsetAsync(sums, 0, (size_t)ns * 8, st));
  }
  return enqueue_density(st, *grid, SampleSource{samples_are_points, samples, samples_batch_ids},
                         ns, inv_radii, DensityRequest{inv_bandwidth, mode, pdf_out, nullptr}, sums);
}

}  // namespace

extern "C" int tfgpc_cells_density(void* stream, const tfgpc_cell_grid* grid,
                                   const float* inv_radii, const float* inv_bandwidth, int mode,
                                   int64_t ns, const float* samples,
                                   const int32_t* samples_batch_ids, int samples_are_points,
                                   float* pdf_out) {
  return cells_density((cudaStream_t)stream, grid, inv_radii, inv_bandwidth, mode, ns, samples,
                       samples_batch_ids, samples_are_points, nullptr, 0, pdf_out);
}

// Half the tests pay where a cell's samples have many candidates: what a cell costs before its
// first test stays, each candidate's sum takes an atomic, and there are a launch and a memset
// more.  us, all tests / half of them: surfaces of 130 to 260 neighbors, 65 536 points 97 / 76,
// 524 288 471 / 315; four dimensions with 34 (560 candidates) 65 536 points 52 / 47, 524 288
// 307 / 241, with 12 (200) 37 / 35 and 229 / 183; three with 34 (220) 23 / 27 and 131 / 125, with
// 12 (77) 24 / 27 and 131 / 123; two with 34 (97) 15 / 20 and 73 / 79.  The candidates are
// estimated as those of a uniform cloud with `pairs` neighbors in all.
extern "C" size_t tfgpc_cells_density_workspace_bytes(int D, int64_t n, int64_t pairs) {
  constexpr int64_t kPoints = 65536;
  constexpr double kCandidates = 256.0;
  // 3^D cells over the unit ball's volume
  constexpr double kPerNeighbor[] = {2.86, 6.45, 16.4, 46.2, 141.0};
  if (!valid_dims(D) || n < kPoints || n >= (int64_t)INT32_MAX) return 0;
  return (double)pairs * kPerNeighbor[D - TFGPC_MIN_DIMS] >= kCandidates * (double)n ? (size_t)n * 8 : 0;
}

extern "C" int tfgpc_cells_density_ws(void* stream, const tfgpc_cell_grid* grid,
                                      const float* inv_radii, const float* inv_bandwidth, int mode,
                                      int64_t ns, const float* samples,
                                      const int32_t* samples_batch_ids, int samples_are_points,
                                      void* ws, size_t ws_bytes, float* pdf_out) {
  return cells_density((cudaStream_t)stream, grid, inv_radii, inv_bandwidth, mode, ns, samples,
                       samples_batch_ids, samples_are_points, ws, ws_bytes, pdf_out);
}
