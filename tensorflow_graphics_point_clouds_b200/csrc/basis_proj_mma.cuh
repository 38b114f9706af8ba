// Basis projection and its gradients on warp-level tensor-core MMAs.
//
// Per sample the projection is a small ragged matrix product,
//   X[c, k] = sum_m feat[nbr(m), c] * basis[m, k],      m over the sample's pairs,
// and so are its two gradients,
//   dbasis[m, k]    = sum_c feat[nbr(m), c] * dX[c, k],
//   dfeat[nbr(m), c] += sum_k basis[m, k] * dX[c, k].
// A CTA-wide tcgen05 tile (128 rows) does not fit products with ~32 pairs per
// sample, so these kernels keep the one-warp-per-sample walk of the SIMT
// kernels and issue mma.sync.m16n8k16 on 16-pair chunks instead of FMAs.  fp32
// accuracy comes from the same 3-pass bf16 split as the big GEMMs:
//   x ~= hi + mid,   a*b ~= a_hi*b_mid + a_mid*b_hi + a_hi*b_hi  (fp32 accumulate).
// Features are pre-split once per call into [n, 2, C] bf16 (hi row, mid row), so
// a neighbor's operand row is gathered with one asynchronous 16-byte copy per
// lane and handed to the MMAs by ldmatrix, never touching registers in between.
//
// Shared-memory rows are padded by 16 bytes so that the eight row reads of one
// ldmatrix fall into distinct bank groups.  Column 2a + b of the tile t of a pair of basis
// tiles stands for basis function 4a + 2t + b: the two accumulator tiles then give every
// lane four consecutive k (or channels), i.e. 128-bit stores and reductions.
#pragma once

#include "basis_proj.cuh"
#include "list_parts.h"

namespace tfgpc {
namespace bpm {

constexpr int kChunk = 16;  // pairs per MMA step (the k or m extent of m16n8k16)

// CC: channels per pass.  A layer narrower than the widest pass takes a smaller one:
// shared memory and accumulators per warp shrink with it, so that more warps are
// resident to hide the gathers (C = 64, K = 16: 16 warps per SM instead of 11).
template <int K, int CC>
struct Cfg {
  static_assert(K == 16 || K == 32 || K == 64, "MMA projection: K in {16, 32, 64}");
  static_assert(CC % 32 == 0 && CC * K <= 2048, "at most 64 accumulators per lane");
  static constexpr int kCC = CC;
  static constexpr int kMT = kCC / 16;   // 16-channel tiles per pass
  static constexpr int kNT = K / 8;      // 8-wide basis tiles
  static constexpr int kNTP = K / 16;    // tile pairs
  static constexpr int kFeatStride = kCC * 4 + 16;  // bytes: hi[kCC] | mid[kCC] | pad
  static constexpr int kBasisStride = K + 4;        // floats of a basis row (+ pad)
  static constexpr int kFeatBytes = kChunk * kFeatStride;
  static constexpr int kBasisBytes = kChunk * kBasisStride * 4;
  static constexpr int kFwdWarpBytes = 2 * kFeatBytes + 2 * kBasisBytes;
  // warps per block (one block per SM): what 64 K registers and 227 KB allow
  static constexpr int kFwdRegWarps = CC * K >= 2048 ? 12 : CC * K >= 1024 ? 16 : 24;
  static constexpr int kMaxSmem = 227 * 1024;
  static constexpr int kFwdWarps = kFwdRegWarps < kMaxSmem / kFwdWarpBytes
                                       ? kFwdRegWarps : kMaxSmem / kFwdWarpBytes;
};

// ---- PTX helpers -----------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// d += a (16 x 16, row) * b (16 x 8, col), bf16 operands, fp32 accumulators
__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& mid) {
  split2_bf16(x, y, hi, mid);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// 16-byte asynchronous copy; copies nothing and writes zeros when !valid
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
               : "memory");
}

// What is done under a condition here is predicated, not branched around: with a branch each,
// and 64-bit products for the addresses, a copied row came to 28 instructions and a reduced one
// to 58, of 390 to 610 per chunk.  65 536 samples of 33 pairs, us before -> now: forward K = 16,
// C = 32 106 -> 84, C = 64 137 -> 122, K = 32, C = 64 218 -> 205; gradients 152 -> 140, 249 -> 237,
// 392 -> 385.
__device__ __forceinline__ void cp_async16_if(uint32_t dst, const void* src, bool ok) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n"
               "@p cp.async.cg.shared.global [%0], [%1], 16;\n}" ::"r"(dst), "l"(src),
               "r"((uint32_t)ok) : "memory");
}

// p + i * bytes, as one wide multiply-add
__device__ __forceinline__ const uint8_t* row_at(const uint8_t* p, int i, uint32_t bytes) {
  return p + (uint64_t)(uint32_t)i * bytes;
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- the walk over samples ---------------------------------------------------------
//
// A warp takes blocks of `bs` (1 to 32) consecutive samples, strided over all warps of
// the grid; the launcher makes blocks small enough that every warp gets several.  The
// range ends of a block are read with one coalesced load (the next block's are
// fetched while this one is processed) and handed out by shuffle, so moving from chunk
// to chunk and sample to sample costs no memory access.  A job is one chunk of up to
// 16 pairs; a sample without pairs still yields one empty job so that its (zero) result
// gets written.
struct Job {
  int64_t s;     // sample, -1 once the walk is over
  int base;      // first pair of the chunk
  int cnt;       // pairs in the chunk (0 .. 16)
  bool first, last;  // first / last chunk of the sample
  __device__ __forceinline__ bool valid() const { return s >= 0; }
};

struct Walker {
  const int32_t* ranges;
  int64_t ns, blk, stride;
  int lane, li, r_end, a0, nr_end, na0, base, e, bs;
  bool started;

  __device__ __forceinline__ void load_block(int64_t b, int& rend, int& first) const {
    const int64_t s0 = b * bs;
    rend = (lane < bs && s0 + lane < ns) ? ld_global(ranges + s0 + lane) : 0;
    first = (s0 > 0 && s0 < ns) ? ld_global(ranges + s0 - 1) : 0;
  }

  __device__ __forceinline__ void init(const int32_t* r, int64_t samples, int64_t warp,
                                       int64_t warps, int ln, int block) {
    ranges = r; ns = samples; blk = warp; stride = warps; lane = ln; bs = block;
    li = 0; base = 0; e = 0; started = false;
    load_block(blk, r_end, a0);
    load_block(blk + stride, nr_end, na0);
  }

  __device__ __forceinline__ Job next() {
    Job j;
    if (started && base + kChunk < e) {
      base += kChunk;
      j.s = blk * bs + li; j.base = base; j.cnt = min(kChunk, e - base);
      j.first = false; j.last = base + kChunk >= e;
      return j;
    }
    if (started) ++li;
    started = true;
    if (li == bs || blk * bs + li >= ns) {
      blk += stride; li = 0;
      r_end = nr_end; a0 = na0;
      load_block(blk + stride, nr_end, na0);
    }
    if (blk * bs >= ns) {
      j.s = -1; j.base = 0; j.cnt = 0; j.first = j.last = false;
      base = 0; e = 0; started = false; blk = ns;  // stay exhausted
      return j;
    }
    const int prev = __shfl_sync(0xffffffffu, r_end, (li + 31) & 31);
    e = __shfl_sync(0xffffffffu, r_end, li);
    base = li ? prev : a0;
    j.s = blk * bs + li; j.base = base; j.cnt = min(kChunk, e - base);
    j.first = true; j.last = base + kChunk >= e;
    return j;
  }
};

// ---- staging ---------------------------------------------------------------------------

// Neighbor (point) index of pair base + lane of a job, 0 beyond the chunk.
__device__ __forceinline__ int load_idx(const Job& j, const int2* neigh, int lane) {
  return (j.valid() && lane < j.cnt) ? ld_global(&neigh[j.base + lane].x) : 0;
}

// Starts the gather of a chunk's feature rows: row r of the tile receives
// hi[c0 .. c0+w) and mid[c0 .. c0+w) of point idx(r); rows beyond the chunk are
// zero-filled.  One commit group per call is left to the caller.
template <int K, int CC>
__device__ __forceinline__ void issue_features(uint32_t tile, const __nv_bfloat16* fs,
                                               int C, int c0, int w, int idx, int cnt, int lane) {
  typedef Cfg<K, CC> cfg;
  constexpr int kLph = cfg::kCC / 8;           // 16-byte segments per half row
  constexpr int kRpi = 32 / (2 * kLph);        // rows per warp instruction
  const int sub = lane % (2 * kLph), rsub = lane / (2 * kLph);
  const int half = sub / kLph, seg = sub % kLph;
  const int have = seg * 8 < w ? cnt : 0;      // (a lane without channels: zeros)
  const uint32_t dst0 = tile + half * (cfg::kCC * 2) + seg * 16 + rsub * cfg::kFeatStride;
  const uint8_t* const src0 = reinterpret_cast<const uint8_t*>(fs + (half * C + c0 + (seg * 8 < w ? seg * 8 : 0)));
  const uint32_t stride = 4u * (uint32_t)C;
#pragma unroll
  for (int it = 0; it < kChunk / kRpi; ++it) {
    const int j = __shfl_sync(0xffffffffu, idx, it * kRpi + rsub);
    cp_async16_zfill(dst0 + it * kRpi * cfg::kFeatStride, row_at(src0, j, stride),
                     it * kRpi + rsub < have);
  }
}

// Starts the copy of a chunk's basis rows, 16 x K floats contiguous in memory (zeros beyond
// the chunk).
template <int K>
__device__ __forceinline__ void issue_basis(uint32_t tile, const float* basis, int base, int cnt,
                                            int lane) {
  const float* src = basis + (int64_t)base * K + lane * 4;
#pragma unroll
  for (int t = 0; t < K / 8; ++t) {
    const int row = (lane + 32 * t) / (K / 4), a4 = lane % (K / 4);
    cp_async16_zfill(tile + (row * (K + 4) + a4 * 4) * 4, src + 128 * t, row < cnt);
  }
}

// The right operand of tile pair j out of a chunk's basis rows: rows 2q, 2q + 1 and, eight
// further on, of the column that the tiles' column g stands for, split.
template <int K>
__device__ __forceinline__ void basis_operand(const float* tile, int j, int g, int q, uint32_t* hi,
                                              uint32_t* mid) {
  const float* p = tile + 2 * q * (K + 4) + 16 * j + 4 * (g >> 1) + (g & 1);
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int half = 0; half < 2; ++half)
      split2(p[8 * half * (K + 4) + 2 * t], p[(8 * half + 1) * (K + 4) + 2 * t], hi[2 * t + half],
             mid[2 * t + half]);
}

// ---- forward ---------------------------------------------------------------------------
//
// X[s] as D[c, k] += A[c, pair] * B[pair, k] per chunk: A comes transposed out of
// the gathered feature rows (ldmatrix.trans), B out of the basis rows, split on the way to
// registers.  Features and basis rows of chunk i+1 are in flight, and the indices of chunk
// i+2 are on their way to registers, while chunk i is multiplied.  (The basis rows by
// registers, split and stored for ldmatrix at the end of a chunk, had the warp wait for them
// there.  65 536 samples of 33 pairs, us before -> now: forward K = 16, C = 32 84 -> 79, K = 32,
// C = 32 134 -> 114, C = 64 205 -> 183 to 203; gradients 140 -> 133, 212 -> 192, 385 -> 342 to 383.)
// OUT = 0: fp32 [ns, C, K] (the op's output).  OUT = 1: the same values split
// into two bf16 arrays [ns, C*K] (left operand of the tensor-core GEMM).
// The passes over the channels are dealt to gridDim.y.  The columns of a row lie in the
// order of block_offset: 2^shift = K is the op's (c, k), less are the blocks of several
// kernel MLPs, one after the other (BLOCKS: without them a row's places are constants).
template <int K, int CC, int OUT, bool BLOCKS>
__global__ void __launch_bounds__(Cfg<K, CC>::kFwdWarps * 32, 1)
basis_proj_mma_kernel(int bs, int shift, int C, int64_t ns, const float* basis,
                      const __nv_bfloat16* fs, const int2* neigh,
                      const int32_t* ranges, float* __restrict__ out,
                      __nv_bfloat16* __restrict__ out_hi, __nv_bfloat16* __restrict__ out_mid) {
  chain_enter(ns * 32, (int64_t)gridDim.x * blockDim.x);
  typedef Cfg<K, CC> cfg;
  extern __shared__ __align__(128) uint8_t bpm_smem[];
  const int lane = threadIdx.x & 31;
  const int warp_in_block = threadIdx.x >> 5;
  const int warps_per_block = blockDim.x >> 5;
  uint8_t* wsm = bpm_smem + (size_t)warp_in_block * cfg::kFwdWarpBytes;
  // two feature tiles, then two basis tiles
  auto feat_tile = [&](int b) { return wsm + b * cfg::kFeatBytes; };
  auto basis_tile = [&](int b) {
    return reinterpret_cast<float*>(wsm + 2 * cfg::kFeatBytes + b * cfg::kBasisBytes);
  };
  const int64_t warp = (int64_t)blockIdx.x * warps_per_block + warp_in_block;
  const int64_t warps = (int64_t)gridDim.x * warps_per_block;
  const int g = lane >> 2, q = lane & 3;
  const int mi = lane >> 3, r = lane & 7;
  // ldmatrix row addresses (bytes inside a tile) of this lane
  const uint32_t a_off = (r + 8 * (mi >> 1)) * cfg::kFeatStride + 8 * (mi & 1) * 2;

  for (int c0 = blockIdx.y * cfg::kCC; c0 < C; c0 += gridDim.y * cfg::kCC) {
    const int w = min(cfg::kCC, C - c0);
    const int mt_cnt = w >> 4;
    Walker walk;
    walk.init(ranges, ns, warp, warps, lane, bs);
    Job cur = walk.next(), n1 = walk.next(), n2 = walk.next();
    int idx1 = load_idx(n1, neigh, lane);
    __syncwarp();
    if (cur.valid()) {
      const int idx0 = load_idx(cur, neigh, lane);
      issue_features<K, CC>(smem_addr(feat_tile(0)), fs, C, c0, w, idx0, cur.cnt, lane);
      issue_basis<K>(smem_addr(basis_tile(0)), basis, cur.base, cur.cnt, lane);
    }
    cp_commit();
    float acc[cfg::kMT][cfg::kNT][4];
    int buf = 0;
    while (cur.valid()) {
      const int idx2 = load_idx(n2, neigh, lane);
      if (n1.valid()) {
        issue_features<K, CC>(smem_addr(feat_tile(buf ^ 1)), fs, C, c0, w, idx1, n1.cnt, lane);
        issue_basis<K>(smem_addr(basis_tile(buf ^ 1)), basis, n1.base, n1.cnt, lane);
      }
      cp_commit();
      cp_wait<1>();   // the rows of `cur` have landed
      __syncwarp();
      if (cur.first) {
#pragma unroll
        for (int mt = 0; mt < cfg::kMT; ++mt)
#pragma unroll
          for (int nt = 0; nt < cfg::kNT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[mt][nt][i] = 0.0f;
      }
      if (cur.cnt > 0) {
        const uint32_t ft = smem_addr(feat_tile(buf)) + a_off;
        const float* const bt = basis_tile(buf);
        // The basis operands, all at once where several channel tiles use them.  (Held for a
        // single pair of tiles, the 32 of K = 64 spilled: 241 us for 33 000 samples at C = 32,
        // 106 without.)
        constexpr bool kHold = cfg::kMT > 2;
        constexpr int kHeld = kHold ? cfg::kNTP : 1;
        uint32_t bh[kHeld][4], bm[kHeld][4];
#pragma unroll
        for (int j = 0; j < cfg::kNTP && kHold; ++j)
          basis_operand<K>(bt, j, g, q, bh[j % kHeld], bm[j % kHeld]);
        // Two 16-channel tiles at a time, and pass by pass over all their
        // accumulator tiles: consecutive MMAs never touch the same accumulator,
        // so none of them waits for the one before it.
#pragma unroll
        for (int mt = 0; mt < cfg::kMT; mt += 2) {
          if (mt < mt_cnt) {
            const bool two = mt + 1 < mt_cnt;
            uint32_t ah[2][4], am[2][4];
            ldsm_x4_t(ft + mt * 32, ah[0]);
            ldsm_x4_t(ft + cfg::kCC * 2 + mt * 32, am[0]);
            if (two) {
              ldsm_x4_t(ft + (mt + 1) * 32, ah[1]);
              ldsm_x4_t(ft + cfg::kCC * 2 + (mt + 1) * 32, am[1]);
            }
#pragma unroll
            for (int j0 = 0; j0 < cfg::kNTP; j0 += kHeld) {
              if (!kHold) basis_operand<K>(bt, j0, g, q, bh[0], bm[0]);
#pragma unroll
              for (int pass = 0; pass < 3; ++pass) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  if (u == 0 || two) {
                    const uint32_t* a = pass == 1 ? am[u] : ah[u];
#pragma unroll
                    for (int j = 0; j < kHeld; ++j) {
                      const uint32_t* b = pass == 0 ? bm[j] : bh[j];
                      mma16816(acc[mt + u][2 * (j0 + j)], a, b[0], b[1]);
                      mma16816(acc[mt + u][2 * (j0 + j) + 1], a, b[2], b[3]);
                    }
                  }
                }
              }
            }
          }
        }
      }
      if (cur.last) {
        // lane (g, q): channels c0 + 16*mt + g (+8), basis functions 16*j + 4*q .. +3
        const int sh = BLOCKS ? shift : K == 16 ? 4 : K == 32 ? 5 : 6;
        const int64_t obase = cur.s * C * K + ((c0 + g) << sh) + (BLOCKS ? 0 : 4 * q);
#pragma unroll
        for (int mt = 0; mt < cfg::kMT; ++mt) {
          if (mt < mt_cnt) {
#pragma unroll
            for (int j = 0; j < cfg::kNTP; ++j) {
#pragma unroll
              for (int h = 0; h < 2; ++h) {   // rows g and g + 8
                const int k = 16 * j + 4 * q;
                const int64_t o = obase + (BLOCKS ? (((k >> sh) * C + 16 * mt + 8 * h) << sh) +
                                                        (k & ((1 << sh) - 1))
                                                  : ((16 * mt + 8 * h) << sh) + 16 * j);
                if (OUT == 0) {
                  *reinterpret_cast<float4*>(out + o) =
                      make_float4(acc[mt][2 * j][2 * h], acc[mt][2 * j][2 * h + 1],
                                  acc[mt][2 * j + 1][2 * h], acc[mt][2 * j + 1][2 * h + 1]);
                } else {
                  uint2 hv, mv;
                  split2(acc[mt][2 * j][2 * h], acc[mt][2 * j][2 * h + 1], hv.x, mv.x);
                  split2(acc[mt][2 * j + 1][2 * h], acc[mt][2 * j + 1][2 * h + 1], hv.y, mv.y);
                  *reinterpret_cast<uint2*>(out_hi + o) = hv;
                  *reinterpret_cast<uint2*>(out_mid + o) = mv;
                }
              }
            }
          }
        }
      }
      __syncwarp();
      cur = n1; n1 = n2; n2 = walk.next();
      idx1 = idx2;
      buf ^= 1;
    }
    cp_wait<0>();
    __syncwarp();
  }
}

// ---- gradients ---------------------------------------------------------------------------
//
// The incoming gradient dX[s] (C x K floats) takes part in every chunk of a sample, so it
// is the LEFT operand of both products and stays in registers, split into bf16 hi / mid
// fragments once per sample, while the pairs stand in the columns, eight at a time:
//   (1) dbasis^T[k, pair] = A[k, c] * B[c, pair]: B straight out of the gathered feature rows;
//   (2) dfeat^T[c, pair]  = A[c, k] * B[k, pair]: B out of the staged basis rows; one 128-bit
//       reduction per lane and 4 channels into dfeat[nbr(pair)], 128 bytes in a row per pair.
// Both fragment sets together are C * K / 16 registers; where one warp cannot hold them a
// team of two shares a sample: both warps see all pairs, (1) is split by basis functions and
// (2) by channels, so that no sum crosses warps.
// While a chunk is multiplied the next one's feature and basis rows are on their way to the
// team's other stage, and dX of the next sample to the place that this one's has left for
// registers.
// What bounds it: the SM's L1 data path (62 % of its wavefronts, 69 % on the busiest SM:
// copies into shared memory, operand reads, reductions at ~24 B/clk) and the instructions
// around the MMAs (issue 51 %).  What teams and fragments gave, 65 536 samples of 28 pairs at
// C = 64, K = 32: 345 -> 290 us (now 54 500 of 32 pairs: 235, 0.9 GB: 3.8 TB/s); 41 000 at
// C = 64, K = 16: 166 -> 139, without the gradient of the basis 86 (the reductions of 1.15
// million rows: 60).  (One warp per sample with dX as bf16 rows in shared memory, read by
// ldmatrix again for every chunk, took 25 KB at C = 64, K = 32 -- 8 warps per SM -- and a chunk
// of nine pairs cost as much as one of sixteen.  Everything straight from global memory to
// registers, without shared memory, read each piece of dX twice through L1: 228 against 185 us
// on 33 000 samples.)
// dbasis is written, not accumulated (every pair belongs to exactly one sample; layers
// wider than a pass add to it pass by pass); dfeat must be zero on entry.
// BASIS false: dfeat alone, for layers whose basis is not trained: (1) is left out, and no
// features are gathered.
template <int K, int CC, bool BASIS>
struct GradCfg {
  static_assert(K * CC <= 2048 && CC % 32 == 0 && (K * CC <= 1024 || K >= 32), "fragments");
  static constexpr int kTeam = K * CC > 1024 ? 2 : 1;       // warps per sample
  static constexpr int kMt1 = K / 16 / kTeam;               // 16-row tiles of (1) per warp
  static constexpr int kKs1 = CC / 16;                      // its reduction steps
  static constexpr int kMt2 = CC / 16 / kTeam;              // tiles of (2)
  static constexpr int kKs2 = K / 16;
  static constexpr int kFeatStride = CC * 4 + 16;           // bytes: hi[CC] | mid[CC] | pad
  static constexpr int kBasisStride = K + 8;                // floats of a basis row (+ pad)
  static constexpr int kRawStride = K + 4;                  // floats, a row of dX over k
  static constexpr int kFeatBytes = BASIS ? kChunk * kFeatStride : 0;
  static constexpr int kStageBytes = kFeatBytes + kChunk * kBasisStride * 4;
  static constexpr int kRawBytes = CC * kRawStride * 4;
  static constexpr int kTeamBytes = kRawBytes + 2 * kStageBytes;
  static constexpr int kFit = 227 * 1024 / kTeamBytes * kTeam;      // warps: 16 of 128 registers
  static constexpr int kWarps = !BASIS && K * CC <= 512 ? 24                        // or 24 of 80
                                : kFit >= 16 && (kMt1 == 1 || !BASIS) ? 16 : 12;    // or 12 of 168
  static constexpr int kTeams = kWarps / kTeam;
  static constexpr int kThreads = kTeams * kTeam * 32;
  static constexpr int kBasisVecs = kChunk * K / 4 / (32 * kTeam);   // float4 per lane and chunk
  static_assert(kTeams * kTeamBytes <= 227 * 1024 && (kTeam == 1 || kTeams <= 15),
                "shared memory, and a named barrier per team");
};

// d = a * b
__device__ __forceinline__ void mma16816_first(float* d, const uint32_t* a, uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

template <int N>
__device__ __forceinline__ void red_add_if(float* dst, const float* v, bool ok) {
  if (N == 4)
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n"
                 "@p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"l"(dst), "f"(v[0]),
                 "f"(v[1]), "f"(v[N / 2]), "f"(v[N - 1]), "r"((uint32_t)ok) : "memory");
  else
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n"
                 "@p red.global.add.v2.f32 [%0], {%1, %2};\n}" ::"l"(dst), "f"(v[0]), "f"(v[1]),
                 "r"((uint32_t)ok) : "memory");
}

template <int N>
__device__ __forceinline__ void store_if(float* dst, const float* v, bool ok) {
  if (N == 4)
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n"
                 "@p st.global.v4.f32 [%0], {%1, %2, %3, %4};\n}" ::"l"(dst), "f"(v[0]), "f"(v[1]),
                 "f"(v[N / 2]), "f"(v[N - 1]), "r"((uint32_t)ok) : "memory");
  else
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %3, 0;\n"
                 "@p st.global.v2.f32 [%0], {%1, %2};\n}" ::"l"(dst), "f"(v[0]), "f"(v[1]),
                 "r"((uint32_t)ok) : "memory");
}

// The chunks of a team, one after the other (see Walker; an item without pairs is left out).
// Every sample is walked as `parts` items, each a run of its chunks: a sample's pairs are
// independent here.
struct Chunk {
  int item, base, end;     // item -1: no more
  bool first;
  __device__ __forceinline__ bool valid() const { return item >= 0; }
  __device__ __forceinline__ int cnt() const { return min(end - base, kChunk); }
};

struct ChunkWalk {
  const int32_t* ranges;
  int items, parts, bs, stride, lane;
  int blk, li, upto, begin, upto_next, begin_next;   // upto: end of the lane's item of the block

  __device__ __forceinline__ int item_end(int i) const {
    if (parts == 1) return ld_global(ranges + i);
    const int s = i / parts;
    return part_end(s > 0 ? ld_global(ranges + s - 1) : 0, ld_global(ranges + s), i - s * parts + 1, parts,
                    kChunk);
  }
  __device__ __forceinline__ void load(int64_t b, int* upto_b, int* begin_b) const {
    const int64_t s0 = b * bs;
    *upto_b = lane < bs && s0 + lane < items ? item_end((int)s0 + lane) : 0;
    *begin_b = s0 > 0 && s0 < items ? item_end((int)s0 - 1) : 0;
  }
  __device__ __forceinline__ Chunk start(const int32_t* r, int item_count, int team, int teams,
                                         int ln, int block, int part_count) {
    ranges = r; items = item_count; blk = team; stride = teams; lane = ln; bs = block;
    parts = part_count; li = -1;
    load(blk, &upto, &begin);
    load((int64_t)blk + stride, &upto_next, &begin_next);
    Chunk c;
    c.item = 0; c.base = c.end = 0; c.first = false;
    return next(c);
  }
  __device__ __forceinline__ Chunk next(Chunk c) {
    c.first = false;
    if (c.end - c.base > kChunk) {
      c.base += kChunk;
      return c;
    }
    do {
      ++li;
      if (li == bs || (int64_t)blk * bs + li >= items) {
        if ((int64_t)blk * bs >= items || ((int64_t)blk + stride) * bs >= items) {
          c.item = -1;
          c.base = c.end = 0;
          c.first = false;
          blk = items;        // (stays at the end)
          bs = 1;
          return c;
        }
        blk += stride;
        li = 0;
        upto = upto_next; begin = begin_next;
        load((int64_t)blk + stride, &upto_next, &begin_next);
      }
      c.end = __shfl_sync(0xffffffffu, upto, li);
      const int before = __shfl_sync(0xffffffffu, upto, (li + 31) & 31);
      c.base = li ? before : begin;
      c.item = blk * bs + li;
      c.first = true;
    } while (c.base >= c.end);
    return c;
  }
};

template <int K, int CC, bool BASIS>
__global__ void __launch_bounds__(GradCfg<K, CC, BASIS>::kThreads, 1)
basis_proj_grads_mma_kernel(int bs, int parts, int shift, int C, int64_t ns, int64_t M,
                            const float* basis,
                            const __nv_bfloat16* fs, const int2* neigh,
                            const int32_t* ranges,
                            const float* in_grads, float* __restrict__ dbasis,
                            float* __restrict__ dfeat) {
  typedef GradCfg<K, CC, BASIS> cfg;
  constexpr int W = cfg::kTeam;
  chain_enter(ns * parts * 32 * W, (int64_t)gridDim.x * blockDim.x);
  extern __shared__ __align__(128) uint8_t bpm_smem[];
  const int lane = threadIdx.x & 31;
  const int team = (threadIdx.x >> 5) / W, sub = (threadIdx.x >> 5) % W;
  const int tid = threadIdx.x % (32 * W);
  uint8_t* const mem = bpm_smem + (size_t)team * cfg::kTeamBytes;
  float* const raw = reinterpret_cast<float*>(mem);
  auto team_sync = [&]() {
    if (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(32 * W) : "memory");
  };
  const int g = lane >> 2, q = lane & 3;
  // ldmatrix rows of this lane: pair lane % 8 of a group; matrices 0 and 1 are the hi terms of
  // columns 0-7 and 8-15 of a 16-column step, 2 and 3 the mid terms
  const uint32_t f_off = (lane & 7) * cfg::kFeatStride + ((lane >> 3) & 1) * 16 + (lane >> 4) * (CC * 2);
  // The row order inside a tile gives a lane consecutive outputs: row g + 8h of a lone tile
  // is output 2g + h, of tile t of a pair output 4g + 2t + h of the pair's 32.
  constexpr int kVec1 = cfg::kMt1 % 2 == 0 ? 4 : 2, kVec2 = cfg::kMt2 % 2 == 0 ? 4 : 2;
  auto out_row = [&](int mt, int vec) {
    return vec == 4 ? 32 * (mt >> 1) + 4 * g + 2 * (mt & 1) : 16 * mt + 2 * g;
  };
  const int row1 = 16 * cfg::kMt1 * sub, row2 = 16 * cfg::kMt2 * sub;   // this warp's rows

  // pairs beyond the last range belong to no sample: their gradient is zero
  if (BASIS && blockIdx.x == 0 && threadIdx.x < 32) {
    const int64_t covered = ns > 0 ? ld_global(ranges + ns - 1) : 0;
    for (int64_t i = covered * K + lane; i < M * K; i += 32) dbasis[i] = 0.0f;
  }

  for (int c0 = 0; c0 < C; c0 += CC) {
    const int w = min(CC, C - c0);
    // ---- copies
    // dX: rows of K floats per channel, out of one piece of w * K floats per block of columns
    // 16-byte pieces of rows 8-15 of every 16 change places with those two further on: the
    // rows 4g that (2) reads then lie in different banks
    constexpr int kRowStep = 32 * W / (K / 4);      // rows of dX that a copy per lane covers
    static_assert(kRowStep == 8 || kRowStep == 4, "rows of one copy lie in half of 16");
    const uint32_t dx_row = smem_addr(raw) + tid / (K / 4) * cfg::kRawStride * 4;
    const uint32_t dx_dst[2] = {dx_row + tid % (K / 4) * 16, dx_row + (tid % (K / 4) ^ 2) * 16};
    auto issue_dx = [&](int item) {
      const float* src = in_grads + (int64_t)(parts == 1 ? item : item / parts) * C * K +
                         ((int64_t)c0 << shift);
      if ((1 << shift) == K && w == CC) {
        src += tid * 4;
#pragma unroll
        for (int i = 0; i < CC * K / 4 / (32 * W); ++i)
          cp_async16(dx_dst[i * kRowStep / 8 & 1] + i * kRowStep * cfg::kRawStride * 4,
                     src + i * 32 * W * 4);
      } else {
#pragma unroll 1
        for (int i = tid; i < w * (K / 4); i += 32 * W) {
          const int c = i / (K / 4), k = (i % (K / 4)) * 4;
          cp_async16(smem_addr(raw) + (c * cfg::kRawStride + (k ^ (c & 8))) * 4,
                     src + (((k >> shift) * C + c) << shift) + (k & ((1 << shift) - 1)));
        }
      }
    };
    // feature rows: hi[c0 .. c0 + w) and mid[c0 .. c0 + w) of the chunk's neighbors (a row
    // beyond them keeps what it held: it is a column of the products, and nobody takes it)
    constexpr int kSeg = CC / 8;             // 16-byte segments per half row
    constexpr int kRpi = 32 / (2 * kSeg);    // rows per warp instruction
    const int seg = lane % kSeg, half_row = lane / kSeg % 2, row0 = sub * kRpi + lane / (2 * kSeg);
    const uint32_t f_dst = smem_addr(mem) + cfg::kRawBytes + row0 * cfg::kFeatStride +
                           half_row * (CC * 2) + seg * 16;
    const uint8_t* const f_src = reinterpret_cast<const uint8_t*>(fs + ((int64_t)half_row * C + c0 + seg * 8));
    const int row_limit = seg * 8 < w ? row0 : kChunk;      // a lane without channels: no row
    auto issue_rows = [&](int st, const Chunk& j, int idx) {
      const uint32_t dst = f_dst + st * cfg::kStageBytes;
      const int cnt = j.cnt();
#pragma unroll
      for (int it = 0; it < kChunk / kRpi / W; ++it) {
        const int p = __shfl_sync(0xffffffffu, idx, it * W * kRpi + row0);
        cp_async16_if(dst + it * W * kRpi * cfg::kFeatStride, row_at(f_src, p, 4u * (uint32_t)C),
                      row_limit + it * W * kRpi < cnt);
      }
    };
    // basis rows: 16 bytes number tid + 32 W t of the chunk
    const uint32_t b_dst = smem_addr(mem) + cfg::kRawBytes + cfg::kFeatBytes +
                           (tid / (K / 4) * cfg::kBasisStride + tid % (K / 4) * 4) * 4;
    auto issue_basis = [&](int st, const Chunk& j) {
      const float* src = basis + (int64_t)j.base * K + tid * 4;
      const int have = j.cnt() * (K / 4) - tid;
#pragma unroll
      for (int t = 0; t < cfg::kBasisVecs; ++t)
        cp_async16_if(b_dst + st * cfg::kStageBytes + t * (32 * W / (K / 4)) * cfg::kBasisStride * 4,
                      src + 128 * W * t, 32 * W * t < have);
    };

    if (c0 > 0) team_sync();       // (the pass before has read its stages and dX)
    if (w < CC) {
      // channels that do not exist, on either side of (1)
      for (int i = tid; i < (CC - w) * cfg::kRawStride; i += 32 * W) raw[w * cfg::kRawStride + i] = 0.0f;
      for (int i = tid; BASIS && i < 2 * kChunk * 2 * (CC - w) / 8; i += 32 * W) {
        const int r = i / (2 * (CC - w) / 8), e = i % (2 * (CC - w) / 8), h = e / ((CC - w) / 8);
        uint8_t* row = mem + cfg::kRawBytes + (r / kChunk) * cfg::kStageBytes + (r % kChunk) * cfg::kFeatStride;
        *reinterpret_cast<uint4*>(row + h * (CC * 2) + (w + e % ((CC - w) / 8) * 8) * 2) =
            make_uint4(0, 0, 0, 0);
      }
    }
    ChunkWalk walk;
    Chunk cur = walk.start(ranges, (int)(ns * parts), (int)blockIdx.x * cfg::kTeams + team,
                           (int)gridDim.x * cfg::kTeams, lane, bs, parts);
    Chunk n1 = walk.next(cur), n2 = walk.next(n1);
    auto load_idx = [&](const Chunk& j) {
      return j.valid() && lane < j.cnt() ? ld_global(&neigh[j.base + lane].x) : 0;
    };
    int idx0 = load_idx(cur), idx1 = load_idx(n1);
    if (cur.valid()) {
      issue_dx(cur.item);
      if (BASIS) issue_rows(0, cur, idx0);
      issue_basis(0, cur);
    }
    cp_commit();
    uint32_t a1h[cfg::kMt1][cfg::kKs1][4], a1m[cfg::kMt1][cfg::kKs1][4];
    uint32_t a2h[cfg::kMt2][cfg::kKs2][4], a2m[cfg::kMt2][cfg::kKs2][4];
    float* const db_lane = dbasis + row1 + out_row(0, kVec1) + 2 * q * K;
    float* const df_lane = dfeat + c0 + row2 + out_row(0, kVec2);
    const int channels = w - (row2 + out_row(0, kVec2));      // from the lane's first one on
    int st = 0;
    while (cur.valid()) {
      // the rows of this chunk have landed, and dX if it is the item's first; the other
      // stage has been read
      cp_wait<0>();
      team_sync();
      if (cur.first) {
#pragma unroll
        for (int mt = 0; mt < (BASIS ? cfg::kMt1 : 0); ++mt) {
          const int k = row1 + out_row(mt, kVec1);
#pragma unroll
          for (int ks = 0; ks < cfg::kKs1; ++ks) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const float* r = raw + (16 * ks + 8 * half + 2 * q) * cfg::kRawStride + (k ^ (8 * half));
              const float2 x = *reinterpret_cast<const float2*>(r);
              const float2 y = *reinterpret_cast<const float2*>(r + cfg::kRawStride);
              split2(x.x, y.x, a1h[mt][ks][2 * half], a1m[mt][ks][2 * half]);
              split2(x.y, y.y, a1h[mt][ks][2 * half + 1], a1m[mt][ks][2 * half + 1]);
            }
          }
        }
#pragma unroll
        for (int mt = 0; mt < cfg::kMt2; ++mt) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int c = row2 + out_row(mt, kVec2) + h;
            const float* r = raw + c * cfg::kRawStride + 2 * q;
#pragma unroll
            for (int ks = 0; ks < cfg::kKs2; ++ks) {
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                const float2 x = *reinterpret_cast<const float2*>(r + 16 * ks + ((8 * half) ^ (c & 8)));
                split2(x.x, x.y, a2h[mt][ks][2 * half + h], a2m[mt][ks][2 * half + h]);
              }
            }
          }
        }
        team_sync();     // dX has been read: the next item's may come
        const Chunk& following = n1.first ? n1 : n2;      // (further ahead: at the next chunk)
        if (following.valid() && following.first) issue_dx(following.item);
      } else if (!n1.first && n2.valid() && n2.first) {
        issue_dx(n2.item);
      }
      if (n1.valid()) {
        if (BASIS) issue_rows(st ^ 1, n1, idx1);
        issue_basis(st ^ 1, n1);
      }
      cp_commit();
      const int idx2 = load_idx(n2);
      // ---- the products, eight pairs at a time
      const uint32_t tile = smem_addr(mem) + cfg::kRawBytes + st * cfg::kStageBytes;
      const float* const rows_of = reinterpret_cast<const float*>(mem + cfg::kRawBytes + st * cfg::kStageBytes +
                                                                  cfg::kFeatBytes) +
                                   g * cfg::kBasisStride + 2 * q;
      const int cnt = cur.cnt();
      float* const db = db_lane + (int64_t)cur.base * K;
#pragma unroll
      for (int p = 0; p < kChunk; p += 8) {
        if (p >= cnt) break;
        float d1[cfg::kMt1][4], d2[cfg::kMt2][4];
#pragma unroll
        for (int ks = 0; ks < (BASIS ? cfg::kKs1 : 0); ++ks) {
          uint32_t b[4];
          ldsm_x4(tile + f_off + p * cfg::kFeatStride + ks * 32, b);
#pragma unroll
          for (int mt = 0; mt < cfg::kMt1; ++mt) {
            if (ks == 0) mma16816_first(d1[mt], a1h[mt][ks], b[2], b[3]);
            else mma16816(d1[mt], a1h[mt][ks], b[2], b[3]);
            mma16816(d1[mt], a1m[mt][ks], b[0], b[1]);
            mma16816(d1[mt], a1h[mt][ks], b[0], b[1]);
          }
        }
#pragma unroll
        for (int ks = 0; ks < cfg::kKs2; ++ks) {
          uint32_t b[4];      // hi terms of columns 2q, 2q + 1 and, eight further on; mid terms
          const float* row = rows_of + p * cfg::kBasisStride + 16 * ks;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const float2 x = *reinterpret_cast<const float2*>(row + 8 * half);
            split2(x.x, x.y, b[half], b[2 + half]);
          }
#pragma unroll
          for (int pass = 0; pass < 3; ++pass)
#pragma unroll
            for (int mt = 0; mt < cfg::kMt2; ++mt) {
              const uint32_t* a = pass == 1 ? a2m[mt][ks] : a2h[mt][ks];
              const uint32_t b0 = pass == 0 ? b[2] : b[0], b1 = pass == 0 ? b[3] : b[1];
              if (ks == 0 && pass == 0) mma16816_first(d2[mt], a, b0, b1);
              else mma16816(d2[mt], a, b0, b1);
            }
        }
        // lane (g, q): pairs 2q and 2q + 1 of the eight
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int pt = __shfl_sync(0xffffffffu, idx0, p + 2 * q + e);
          const bool ok = p + 2 * q + e < cnt;
          float* const df = (float*)row_at((const uint8_t*)df_lane, pt, 4u * (uint32_t)C);
#pragma unroll
          for (int mt = 0; mt < cfg::kMt2; mt += kVec2 / 2) {
            float v[kVec2];
#pragma unroll
            for (int i = 0; i < kVec2; ++i) v[i] = d2[mt + i / 2][2 * (i % 2) + e];
            const int c = out_row(mt, kVec2) - out_row(0, kVec2);
            red_add_if<kVec2>(df + c, v, ok && c < channels);
          }
#pragma unroll
          for (int mt = 0; mt < (BASIS ? cfg::kMt1 : 0); mt += kVec1 / 2) {
            float v[kVec1];
#pragma unroll
            for (int i = 0; i < kVec1; ++i) v[i] = d1[mt + i / 2][2 * (i % 2) + e];
            float* dst = db + (p + e) * K + (out_row(mt, kVec1) - out_row(0, kVec1));
            if (c0 > 0)      // (a load of the pass before's sum would stall the warp)
              red_add_if<kVec1>(dst, v, ok);
            else
              store_if<kVec1>(dst, v, ok);
          }
        }
      }
      st ^= 1;
      cur = n1; n1 = n2; n2 = walk.next(n1);
      idx0 = idx1; idx1 = idx2;
    }
    cp_wait<0>();
  }
}

}  // namespace bpm
}  // namespace tfgpc
