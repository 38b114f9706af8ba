// Basis projection and its gradients in float32 for layers of few channels, where the
// tensor-core kernels do not go (K = 8, or C no multiple of 16) and a lane per few channels
// leaves most of the GPU idle.
//
// A warp owns a sample.  Its lanes tile one pair's C x K products, kKt basis functions by
// CT channels each, and what is left of the 32 lanes takes further pairs at the same time:
// lane = (pair slot * CL + channel block) * KL + basis block.  A step of the loop is one
// coalesced piece of the basis rows, one feature row per slot and kKt * CT multiply-adds a
// lane; the loads of the next step are under way meanwhile.  The slots' sums meet once per
// sample (forward), the lanes of a pair's tile once per pair (gradients), by halving
// butterflies: a lane hands over half of what it holds and keeps the other half.
//
// Before, a group of C / 4 (K = 64: C) lanes owned a sample and every lane all basis functions:
// one to eight lanes for a list of 33 pairs.  us before -> now on 4096 / 16 384 / 65 536
// samples of 16 / 31 / 33 pairs (launches of the op included):
//   forward    K =  8, C = 1  13 -> 7, 18 -> 9, 31 -> 31      C = 8  13 -> 7, 17 -> 13, 57 -> 51
//              K = 16, C = 8  13 -> 7, 19 -> 17, (71, 79)     C = 3  17 -> 7, 27 -> 15, (61, 69)
//              K = 32, C = 1  27 -> 7, 47 -> 17, 114 -> 91    C = 8  15 -> 7, 44 -> 28, 247 -> 127
//              K = 64, C = 1  48 -> 5, 103 -> 35, 228 -> 115  C = 8  21 -> 9, 201 -> 58, 729 -> 223
//              K = 32, C = 16 15 -> 10, 99 -> 68, 433 -> 275     C = 24 21 -> 15, 191 -> 132, 764 -> 519
//   gradients  K =  8, C = 1  42 -> 13, 74 -> 14, 158 -> 49   C = 8  29 -> 13, 46 -> 22, 148 -> 87
//              K = 16, C = 3  81 -> 13, 154 -> 24, 311 -> 109 C = 8  41 -> 13, 67 -> 31, 225 -> 133
//              K = 32, C = 1  153 -> 13, 308 -> 41, 624 -> 130   K = 64  294 -> 10, 577 -> 55, 1166 -> 214
//              K =  8, C = 64 29 -> 21, 101 -> 82, 373 -> 334    C = 128 (27, 31, 128, 161, 494, 605)
//              K = 16, C = 24 31 -> 20, 111 -> 90, 415 -> 350  K = 64  134 -> 51, 833 -> 246, 3385 -> 973
//              K = 32, C = 16 34 -> 17, 143 -> 98, 486 -> 366  C = 24 44 -> 28, 238 -> 228, 877 -> 858
// (bytes of K = 64, C = 1 at 6450 GB/s: 92 and 179 us.)
// Above eight channels the forward tiles are taken at K = 32 alone; elsewhere (us, the lanes of
// basis_proj.cu or the wide kernel, tiles in brackets, the same samples) they lose on many:
//              K =  8, C = 24 12, 29, 117 (7, 23, 140)         C = 64 13, 42, 190 (10, 44, 243)
//              K = 16, C = 24 12, 35, 158 (10, 44, 265)        C = 56 15, 65, 286 (15, 112, 461)
//              K = 64, C = 24 23, 119, 455 (23, 198, 778)
// (K = 64, C = 16, which only calls without scratch bring here: 34, 321, 1287 (15, 114, 443).)
// Bound by HBM for one channel, else by
// the latency of the gathers (10 to 17 warps an SM, issue 28 to 52 %) and the instructions
// around the multiply-adds.
#include "basis_proj.cuh"

namespace tfgpc {
namespace {

typedef unsigned long long f32x2;      // two floats for ffma2

constexpr int kTileThreads = 128;

// KT basis functions per lane; KL lanes cover K.  (K = 64 with four each would leave two
// channel blocks per warp.)
template <int K, int CT, int CL>
struct Tile {
  static constexpr int kKt = K == 64 ? 8 : 4;
  static constexpr int kKl = K / kKt;
  static constexpr int kSlots = 32 / (kKl * CL);      // pairs of a step
  static_assert(kKl * CL <= 32, "a pair's tile fits a warp");
};

constexpr int log2_of(int v) { return v <= 1 ? 0 : 1 + log2_of(v / 2); }

// Sums v[0 .. N) over the 2^STEPS lanes that differ in the lane bits from `bit` on.  Afterwards
// a lane holds max(N >> STEPS, LEAST) of the sums, from number *first on; owner: no other lane
// with a lower number holds the same ones.
template <int N, int STEPS, int LEAST>
__device__ __forceinline__ void fold(float* v, int lane, int bit, int* first, bool* owner) {
  *first = 0;
  *owner = true;
#pragma unroll
  for (int t = 0; t < STEPS; ++t) {
    const int at = bit << t;
    const bool upper = (lane & at) != 0;
    if ((N >> (t + 1)) >= LEAST) {
      const int width = N >> (t + 1);
#pragma unroll
      for (int i = 0; i < width; ++i) {
        const float send = upper ? v[i] : v[i + width];
        const float keep = upper ? v[i + width] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, at);
      }
      if (upper) *first += width;
    } else {
      constexpr int kLeft = (N < LEAST ? N : LEAST);
#pragma unroll
      for (int i = 0; i < kLeft; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], at);
      if (upper) *owner = false;
    }
  }
}

// Values that a lane is left with by fold<N, STEPS, LEAST>.
template <int N, int STEPS, int LEAST>
constexpr int folded() {
  int n = N;
  for (int t = 0; t < STEPS; ++t)
    if ((N >> (t + 1)) >= LEAST) n = N >> (t + 1);
  return n;
}

// What a slot without a pair reads.
__device__ __align__(16) const float kZeros[8] = {0.0f};

// What a lane holds of one pair: its basis values, its features and the neighbor.
template <int K, int CT, int CL>
struct Pair {
  static constexpr int kKt = Tile<K, CT, CL>::kKt;
  float w[kKt], f[CT];
  int j;
};

// The pairs of a warp's samples on their way to a lane's slot, a step of kSlots pairs after
// the other.  Neighbor indices are read 32 at a time, two such pieces ahead and the next
// sample's first one as well, and handed out by shuffle, so that a step's loads depend on
// nothing that is still under way.
template <int K, int CT, int CL>
struct PairStream {
  typedef Tile<K, CT, CL> tile;
  static constexpr int kKt = tile::kKt, kSlots = tile::kSlots;
  const float *basis, *feat;      // of this lane's basis functions and channels
  const int2* neigh;
  int stride, slot, lane;
  int have;                // this lane's channels that exist (0: none is ever read)
  bool vec;
  const float* w_at;       // basis row of the slot's pair of the next step
  unsigned a, total, at;   // first pair of the sample, how many, and how many are on their way
  int idx, idx_next, idx_after;

  __device__ __forceinline__ int neighbor_of(unsigned m, unsigned end) const {
    return m < end ? ld_global(&neigh[m].x) : 0;
  }
  __device__ __forceinline__ void init(unsigned begin, unsigned last) {
    idx_after = neighbor_of(begin + lane, last);
  }
  // the sample of the pairs [begin, end), those of the sample before ended at begin; none of
  // the warp's ends behind `last`.  (An end ahead of its begin is an empty list.)
  __device__ __forceinline__ void start(unsigned begin, unsigned end, unsigned last) {
    a = begin;
    total = (int)end > (int)begin ? end - begin : 0;
    at = 0;
    idx = idx_after;
    idx_next = neighbor_of(begin + 32 + lane, end);
    idx_after = neighbor_of(end + lane, last);
    w_at = basis + ((int64_t)begin + slot) * K;
  }
  // The next step's pair, zeros where the slot has none.  The whole warp calls.  (The loads are
  // made whatever the slot has, of zeros if need be: made on one side of a branch, they were
  // waited for where its sides meet.)
  __device__ __forceinline__ void load(Pair<K, CT, CL>& p) {
    p.j = __shfl_sync(0xffffffffu, idx, (at + slot) & 31);
    const bool live = at + slot < total;
    const float4* row = reinterpret_cast<const float4*>(live ? w_at : kZeros);
#pragma unroll
    for (int i = 0; i < kKt / 4; ++i) {
      const float4 v = ld_global(row + i);
      p.w[4 * i] = v.x; p.w[4 * i + 1] = v.y; p.w[4 * i + 2] = v.z; p.w[4 * i + 3] = v.w;
    }
    const float* src = live && have > 0 ? feat + (int64_t)p.j * stride : kZeros;
    if (CT == 1) {
      p.f[0] = ld_global(src);
    } else if (CT == 8 && (CL > 1 || vec)) {
#pragma unroll
      for (int i = 0; i < CT / 4; ++i) {
        const float4 v = ld_global(reinterpret_cast<const float4*>(src) + i);
        p.f[4 * i] = v.x; p.f[(4 * i + 1) % CT] = v.y;
        p.f[(4 * i + 2) % CT] = v.z; p.f[(4 * i + 3) % CT] = v.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < CT; ++c) p.f[c] = ld_global(c < have ? src + c : kZeros);
    }
    at += kSlots;
    w_at += kSlots * K;
    if ((at & 31) == 0) {
      idx = idx_next;
      idx_next = neighbor_of(a + at + 32 + lane, a + total);
    }
  }
};

// Samples [first, first + count) of a warp, count at most 32: lane i has the end of the i-th
// one's range, and the range before the first.
struct WarpSamples {
  int64_t first;
  int count, ends, before;
  __device__ __forceinline__ WarpSamples(const int32_t* ranges, int64_t ns, int per, int lane) {
    first = (((int64_t)blockIdx.x * kTileThreads + threadIdx.x) >> 5) * per;
    count = (int)(first >= ns ? 0 : ns - first < per ? ns - first : per);
    ends = lane < count ? ld_global(ranges + first + lane) : 0;
    before = count > 0 && first > 0 ? ld_global(ranges + first - 1) : 0;
  }
  __device__ __forceinline__ void range(int i, unsigned* a, unsigned* e) const {
    const int last = __shfl_sync(0xffffffffu, ends, (i + 31) & 31);
    *a = (unsigned)(i ? last : before);
    *e = (unsigned)__shfl_sync(0xffffffffu, ends, i);
  }
  __device__ __forceinline__ unsigned last() const {
    return (unsigned)__reduce_max_sync(0xffffffffu, max(ends, 0));
  }
};

// OUT = 0: fp32 [ns, C, K] (the op's output).  OUT = 1: the same values split into two bf16
// arrays [ns, C*K] (left operand of the tensor-core product), columns of block_offset.
template <int K, int CT, int CL, int OUT>
__global__ void __launch_bounds__(kTileThreads)
basis_proj_tile_kernel(int C, int64_t ns, int per, const float* basis, const float* feat,
                       const int2* neigh, const int32_t* ranges, float* __restrict__ out,
                       __nv_bfloat16* __restrict__ out_hi, __nv_bfloat16* __restrict__ out_mid,
                       int shift, bool vec) {
  chain_enter();
  typedef Tile<K, CT, CL> tile;
  constexpr int kKt = tile::kKt, kSlots = tile::kSlots;
  constexpr int kBatch = kSlots <= 2 ? 2 : 1;      // steps whose loads are made together
  constexpr int kAhead = 2 * kBatch;               // and are under way
  const int lane = lane_id();
  const int k0 = lane % tile::kKl * kKt, c0 = lane / tile::kKl % CL * CT;
  const int slot = lane / (tile::kKl * CL);
  const WarpSamples mine(ranges, ns, per, lane);
  if (mine.count == 0) return;
  const int have = min(max(C - c0, 0), CT);
  PairStream<K, CT, CL> pairs{basis + k0, feat + (have > 0 ? c0 : 0), neigh, C, slot, lane, have, vec};
  const unsigned last = mine.last();
  pairs.init((unsigned)mine.before, last);
  Pair<K, CT, CL> buf[kAhead];
  // the sample's first steps
  auto begin = [&](int i) {
    unsigned a, e;
    mine.range(i, &a, &e);
    pairs.start(a, e, last);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) pairs.load(buf[u]);
  };
  begin(0);
  for (int i = 0; i < mine.count; ++i) {
    // (CT == 1: two basis functions to a register pair, else two channels)
    constexpr int kAcc = CT * kKt;
    f32x2 sum[kAcc / 2];
#pragma unroll
    for (int v = 0; v < kAcc / 2; ++v) sum[v] = 0;
    const unsigned total = pairs.total;
    for (unsigned base = 0; base < total; base += kAhead * kSlots) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (u == kBatch && base + u * kSlots >= total) break;
        if constexpr (CT == 1) {
#pragma unroll
          for (int k = 0; k < kKt; k += 2)
            sum[k / 2] = ffma2(pack2(buf[u].f[0], buf[u].f[0]), pack2(buf[u].w[k], buf[u].w[k + 1]), sum[k / 2]);
        } else {
#pragma unroll
          for (int k = 0; k < kKt; ++k) {
            const f32x2 w = pack2(buf[u].w[k], buf[u].w[k]);
#pragma unroll
            for (int c = 0; c < CT / 2; ++c)
              sum[c * kKt + k] = ffma2(pack2(buf[u].f[2 * c], buf[u].f[2 * c + 1]), w, sum[c * kKt + k]);
          }
        }
        if (u % kBatch == kBatch - 1)
#pragma unroll
          for (int v = u + 1 - kBatch; v <= u; ++v) pairs.load(buf[v]);
      }
    }
    if (i + 1 < mine.count) begin(i + 1);
    float acc[kAcc];
#pragma unroll
    for (int v = 0; v < kAcc / 2; ++v) {
      if (CT == 1) unpack2(sum[v], acc[2 * v], acc[2 * v + 1]);
      else unpack2(sum[v], acc[v / kKt * 2 * kKt + v % kKt], acc[(v / kKt * 2 + 1) * kKt % kAcc + v % kKt]);
    }
    constexpr int kSteps = log2_of(kSlots);
    constexpr int kLeft = folded<CT * kKt, kSteps, 4>();
    int first;
    bool owner;
    fold<CT * kKt, kSteps, 4>(acc, lane, tile::kKl * CL, &first, &owner);
    const int64_t s = mine.first + i;
#pragma unroll
    for (int q = 0; q < kLeft; q += 4) {
      const int c = c0 + (first + q) / kKt, k = k0 + (first + q) % kKt;
      if (!owner || c >= C) continue;
      const int64_t o = block_offset<K>(s, C, c, k, shift);
      if (OUT == 0) {
        *reinterpret_cast<float4*>(out + o) =
            make_float4(acc[q], acc[q + 1], acc[q + 2], acc[q + 3]);
      } else {
        uint2 h, l;
        split2_bf16(acc[q], acc[q + 1], h.x, l.x);
        split2_bf16(acc[q + 2], acc[q + 3], h.y, l.y);
        *reinterpret_cast<uint2*>(out_hi + o) = h;
        *reinterpret_cast<uint2*>(out_mid + o) = l;
      }
    }
  }
}

// dst[0 .. N) += v under a condition, without a branch; have: values that exist.
template <int N>
__device__ __forceinline__ void add_values(float* dst, const float* v, int have, bool vec, bool ok) {
  if (N >= 4 && vec) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n"
                   "@p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"l"(dst + i), "f"(v[i]),
                   "f"(v[(i + 1) % N]), "f"(v[(i + 2) % N]), "f"(v[(i + 3) % N]),
                   "r"((uint32_t)(ok && have > i)) : "memory");
  } else if (N == 2 && vec) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n"
                 "@p red.global.add.v2.f32 [%0], {%1, %2};\n}" ::"l"(dst), "f"(v[0]), "f"(v[1 % N]),
                 "r"((uint32_t)(ok && have > 0)) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n"
                   "@p red.global.add.f32 [%0], %1;\n}" ::"l"(dst + i), "f"(v[i]),
                   "r"((uint32_t)(ok && i < have)) : "memory");
  }
}

template <int N>
__device__ __forceinline__ void store_values(float* dst, const float* v, bool vec, bool ok) {
  if (N % 4 == 0 && vec) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n"
                   "@p st.global.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"l"(dst + i), "f"(v[i]),
                   "f"(v[(i + 1) % N]), "f"(v[(i + 2) % N]), "f"(v[(i + 3) % N]), "r"((uint32_t)ok)
                   : "memory");
  } else if (N == 2 && vec) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n@p st.global.v2.f32 [%0], {%1, %2};\n}"
                 ::"l"(dst), "f"(v[0]), "f"(v[1 % N]), "r"((uint32_t)ok) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.global.f32 [%0], %1;\n}"
                   ::"l"(dst + i), "f"(v[i]), "r"((uint32_t)ok) : "memory");
  }
}

// Gradients: dfeat[nbr, c] += sum_k g[c, k] * basis[m, k] and (BASIS) dbasis[m, k] =
// sum_c g[c, k] * feat[nbr, c], g[s] in the lanes' registers.  dfeat is zero on entry.
template <int K, int CT, int CL, bool BASIS>
__global__ void __launch_bounds__(kTileThreads)
basis_proj_grads_tile_kernel(int C, int64_t ns, int64_t M, int per, const float* basis,
                             const float* feat, const int2* neigh, const int32_t* ranges,
                             const float* in_grads, float* __restrict__ dbasis,
                             float* __restrict__ dfeat, int shift, bool vec, bool vec_basis) {
  chain_enter();
  typedef Tile<K, CT, CL> tile;
  constexpr int kKt = tile::kKt, kSlots = tile::kSlots, kAhead = 2;
  const int lane = lane_id();
  const int k0 = lane % tile::kKl * kKt, c0 = lane / tile::kKl % CL * CT;
  const int slot = lane / (tile::kKl * CL);
  // pairs beyond the last range belong to no sample: their gradient is zero
  if (BASIS) {
    const int64_t thread = (int64_t)blockIdx.x * kTileThreads + threadIdx.x;
    for (int64_t i = (int64_t)ld_global(ranges + ns - 1) * K + thread; i < M * K;
         i += (int64_t)gridDim.x * kTileThreads)
      dbasis[i] = 0.0f;
  }
  const WarpSamples mine(ranges, ns, per, lane);
  if (mine.count == 0) return;
  const int have = min(max(C - c0, 0), CT);
  PairStream<K, CT, CL> pairs{basis + k0, feat + (have > 0 ? c0 : 0), neigh, C, slot, lane,
                              BASIS ? have : 0, vec};
  const unsigned last = mine.last();
  pairs.init((unsigned)mine.before, last);
  Pair<K, CT, CL> buf[kAhead];
  for (int i = 0; i < mine.count; ++i) {
    unsigned a, e;
    mine.range(i, &a, &e);
    pairs.start(a, e, last);
#pragma unroll
    for (int u = 0; u < kAhead; ++u) pairs.load(buf[u]);
    // the lane's tile of g
    float g[CT][kKt];
#pragma unroll
    for (int c = 0; c < CT; ++c) {
#pragma unroll
      for (int q = 0; q < kKt; q += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < have && pairs.total > 0)
          v = ld_global(reinterpret_cast<const float4*>(
              in_grads + block_offset<K>(mine.first + i, C, c0 + c, k0 + q, shift)));
        g[c][q] = v.x; g[c][q + 1] = v.y; g[c][q + 2] = v.z; g[c][q + 3] = v.w;
      }
    }
    const unsigned total = pairs.total;
    for (unsigned base = 0; base < total; base += kAhead * kSlots) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const unsigned done = base + u * kSlots;
        if (u > 0 && done >= total) break;
        const bool live = done + slot < total;
        const unsigned m = a + done + slot;
        float df[CT], db[kKt];
#pragma unroll
        for (int c = 0; c < CT; ++c) {
          df[c] = g[c][0] * buf[u].w[0];
#pragma unroll
          for (int k = 1; k < kKt; ++k) df[c] = fmaf(g[c][k], buf[u].w[k], df[c]);
        }
#pragma unroll
        for (int k = 0; k < (BASIS ? kKt : 0); ++k) {
          db[k] = g[0][k] * buf[u].f[0];
#pragma unroll
          for (int c = 1; c < CT; ++c) db[k] = fmaf(g[c][k], buf[u].f[c], db[k]);
        }
        const int j = buf[u].j;
        pairs.load(buf[u]);
        int at;
        bool owner;
        constexpr int kStepsF = log2_of(tile::kKl);
        fold<CT, kStepsF, 1>(df, lane, 1, &at, &owner);
        // (by predicate; where few lanes of a small K have something, those lanes branch first.
        // 65 536 samples, us, branch and predicate: one channel block K = 32, C = 8 256 / 214;
        // two K = 8, C = 16 136 / 129, K = 16 212 / 212, K = 32 376 / 366, K = 64 540 / 540; four
        // K = 8, C = 24 208 / 246, K = 16 350 / 440, K = 64 980 / 975.  K = 32 with four, 652 / 858,
        // would gain from the branch too, and is left as it is)
        constexpr bool kBranch = CL > 2 && K <= 16;
        if (!kBranch || (owner && live))
          add_values<folded<CT, kStepsF, 1>()>(dfeat + (int64_t)j * C + c0 + at, df, C - c0 - at, vec,
                                               kBranch || (owner && live));
        if (BASIS) {
          constexpr int kStepsB = log2_of(CL);
          fold<kKt, kStepsB, 1>(db, lane, tile::kKl, &at, &owner);
          if (!kBranch || (owner && live))
            store_values<folded<kKt, kStepsB, 1>()>(dbasis + (int64_t)m * K + k0 + at, db, vec_basis,
                                                    kBranch || (owner && live));
        }
      }
    }
  }
}

// Consecutive samples of a warp: several where there are enough for every SM's warps.
int samples_per_warp(int64_t ns) {
  const int64_t s = ns / ((int64_t)sm_count() * 32);
  return (int)(s < 1 ? 1 : s > 8 ? 8 : s);
}

unsigned tile_blocks(int64_t ns, int per) {
  return blocks_for((ns + per - 1) / per, kTileThreads / 32);
}

struct FwdCall {
  static constexpr int most_channels(int K) { return K == 32 ? 32 : 8; }
  cudaStream_t st;
  int C;
  int64_t ns;
  const float *basis, *feat;
  const int2* neigh;
  const int32_t* ranges;
  float* out;
  __nv_bfloat16 *hi, *mid;
  int shift;
  bool vec;
  template <int K, int CT, int CL>
  int run() const {
    const int per = samples_per_warp(ns);
    ProfScope prof(st, out ? "basis_proj" : "basis_proj_split");
    if (out)
      TFGPC_CUDA(launch_chained(st, tile_blocks(ns, per), kTileThreads, 0,
          basis_proj_tile_kernel<K, CT, CL, 0>, C, ns, per, basis, feat, neigh, ranges, out, hi,
          mid, shift, vec));
    else
      TFGPC_CUDA(launch_chained(st, tile_blocks(ns, per), kTileThreads, 0,
          basis_proj_tile_kernel<K, CT, CL, 1>, C, ns, per, basis, feat, neigh, ranges, out, hi,
          mid, shift, vec));
    return TFGPC_OK;
  }
};

struct GradCall {
  static constexpr int most_channels(int K) { return K <= 16 ? 64 : 32; }
  cudaStream_t st;
  int C;
  int64_t ns, M;
  const float *basis, *feat;
  const int2* neigh;
  const int32_t* ranges;
  const float* in_grads;
  float *dbasis, *dfeat;
  int shift;
  bool vec;
  template <int K, int CT, int CL>
  int run() const {
    const int per = samples_per_warp(ns);
    ProfScope prof(st, dbasis ? "basis_proj_grads" : "basis_proj_feature_grads");
    if (dbasis)
      TFGPC_CUDA(launch_chained(st, tile_blocks(ns, per), kTileThreads, 0,
          basis_proj_grads_tile_kernel<K, CT, CL, true>, C, ns, M, per, basis, feat, neigh, ranges,
          in_grads, dbasis, dfeat, shift, vec, (uintptr_t)dbasis % 16 == 0));
    else
      TFGPC_CUDA(launch_chained(st, tile_blocks(ns, per), kTileThreads, 0,
          basis_proj_grads_tile_kernel<K, CT, CL, false>, C, ns, M, per, basis, feat, neigh, ranges,
          in_grads, dbasis, dfeat, shift, vec, (uintptr_t)dbasis % 16 == 0));
    return TFGPC_OK;
  }
};

// The instance of a layer: one channel, up to four, else blocks of eight.
template <int K, typename Call>
int with_tile(const Call& call) {
  constexpr int kMost = Call::most_channels(K);
  if (call.C == 1) return call.template run<K, 1, 1>();
  if (call.C <= 4) return call.template run<K, 4, 1>();
  if (call.C <= 8) return call.template run<K, 8, 1>();
  if constexpr (kMost >= 16)
    if (call.C <= 16) return call.template run<K, 8, 2>();
  if constexpr (kMost >= 32)
    if (call.C <= 32) return call.template run<K, 8, 4>();
  if constexpr (kMost >= 64)
    if (call.C <= 64) return call.template run<K, 8, 8>();
  return fail(TFGPC_EINVAL, "projection tiles: too many channels");
}

template <typename Call>
int with_basis(int K, const Call& call) {
  switch (K) {
    case 8: return with_tile<8>(call);
    case 16: return with_tile<16>(call);
    case 32: return with_tile<32>(call);
    default: return with_tile<64>(call);
  }
}

}  // namespace

// Whether these kernels take a layer: where they were the faster ones (figures above).  Up to
// eight channels anything goes; more are read as 16-byte pieces.  Many samples fill the GPU
// with a few lanes each, and at K <= 16 those then spend fewer instructions on a pair (8 channels
// of 65 536 samples: lanes 57 and 70 us at K = 8 and 16, tiles 51 and 78; 3 channels 37 and 61, 43
// and 68).
bool basis_proj_tile_takes(int K, int C, int64_t ns, const float* feat) {
  if (C > 8) return C <= FwdCall::most_channels(K) && (uintptr_t)feat % 16 == 0;
  return K >= 32 || C == 1 || ns <= 32768;
}

bool basis_proj_grads_tile_takes(int K, int C, const float* feat) {
  return C <= 8 || (C <= GradCall::most_channels(K) && (uintptr_t)feat % 16 == 0);
}

int basis_proj_tile(cudaStream_t st, int K, int C, int64_t ns, const float* basis,
                    const float* feat, const int2* neigh, const int32_t* ranges, float* out,
                    __nv_bfloat16* hi, __nv_bfloat16* mid, int hidden) {
  const bool vec = C % 4 == 0 && (uintptr_t)feat % 16 == 0;
  return with_basis(K, FwdCall{st, C, ns, basis, feat, neigh, ranges, out, hi, mid,
                               hidden_shift(hidden), vec});
}

// dbasis null: the gradient of the features alone.
int basis_proj_grads_tile(cudaStream_t st, int K, int C, int64_t ns, int64_t M, const float* basis,
                          const float* feat, const int2* neigh, const int32_t* ranges,
                          const float* in_grads, float* dbasis, float* dfeat, int hidden) {
  const bool vec = C % 4 == 0 && (uintptr_t)feat % 16 == 0 && (uintptr_t)dfeat % 16 == 0;
  return with_basis(K, GradCall{st, C, ns, M, basis, feat, neigh, ranges, in_grads, dbasis, dfeat,
                                hidden_shift(hidden), vec});
}

}  // namespace tfgpc
