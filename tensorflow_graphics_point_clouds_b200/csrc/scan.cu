// Device-wide scan of int32 counts.
// Takes the place of the reference's recursive Blelloch scan with its host
// loop (find_neighbors/cc/kernels/scan_alg_kernels.cu.cc:41-266): one launch for
// inputs that one block can take (kOneBlock elements), else two -- tile sums, then a
// pass in which every block first adds up the sums of the tiles before its own (up to
// kDirectTiles values out of L2, cheaper than a third launch) --, and above that three,
// the tile sums scanned by one block in between; no host synchronisation, 64-bit tile
// sums so that totals beyond 2^31 are detected by the caller instead of wrapping silently.
#include "scan.cuh"

namespace tfgpc {

int64_t scan_block_sums_elems(int64_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

namespace {

template <int THREADS>
__device__ __forceinline__ int64_t block_sum(int64_t v, int64_t* smem) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane_id() == 0) smem[threadIdx.x >> 5] = v;
  __syncthreads();
  v = threadIdx.x < THREADS / 32 ? smem[threadIdx.x] : 0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) smem[0] = v;
  }
  __syncthreads();
  v = smem[0];
  __syncthreads();
  return v;  // in every thread
}

__device__ __forceinline__ int64_t elems_of(const ScanSize& s) {
  if (!s.num_cells) return s.n;
  int64_t t = s.batch_size;
  for (int d = 0; d < s.dims; ++d) t *= ld_global(s.num_cells + d);
  return t + 3;
}

__global__ void __launch_bounds__(kScanThreads)
scan_reduce_kernel(const int32_t* in, ScanSize size, int64_t* __restrict__ tile_sums) {
  chain_enter();
  __shared__ int64_t smem[32];
  const int64_t n = elems_of(size);
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  if (base >= n) return;
  int64_t v = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t idx = base + (int64_t)i * kScanThreads + threadIdx.x;
    if (idx < n) v += in[idx];
  }
  v = block_sum<kScanThreads>(v, smem);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = v;
}

// Tile sums to the sums of the tiles before each, by one block.
__global__ void __launch_bounds__(1024)
scan_sums_kernel(ScanSize size, int64_t* tile_sums) {
  chain_enter();
  __shared__ int64_t smem[32];
  const int64_t n = elems_of(size);
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  const int w = threadIdx.x >> 5;
  int64_t run = 0;
  for (int64_t t0 = 0; t0 < tiles; t0 += 1024) {
    const int64_t t = t0 + threadIdx.x;
    const int64_t own = t < tiles ? tile_sums[t] : 0;
    int64_t x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane_id() >= o) x += y;
    }
    if (lane_id() == 31) smem[w] = x;
    __syncthreads();
    int64_t before = 0, all = 0;
    for (int i = 0; i < 32; ++i) {
      if (i < w) before += smem[i];
      all += smem[i];
    }
    if (t < tiles) tile_sums[t] = run + before + x - own;
    run += all;
    __syncthreads();
  }
}

// One tile per block.  EXCLUSIVE: out[i] = sum of in[0..i), else of in[0..i].  The
// last tile's block also delivers the report.
template <int THREADS, int ITEMS, bool EXCLUSIVE>
__global__ void __launch_bounds__(THREADS)
scan_tiles_kernel(const int32_t* in, int32_t* __restrict__ out, ScanSize size,
                  const int64_t* tile_sums, bool sums_scanned,
                  int64_t* __restrict__ total, ScanReport rep) {
  chain_enter();
  constexpr int kTile = THREADS * ITEMS;
  __shared__ int64_t smem[32];
  __shared__ int32_t stage[kTile];
  const int64_t n = elems_of(size);
  const int64_t tile0 = (int64_t)blockIdx.x * kTile;
  if (tile0 >= n) return;
  int64_t before = 0;
  if (sums_scanned) {
    before = ld_global(tile_sums + blockIdx.x);
  } else if (blockIdx.x > 0) {
    for (int64_t t = threadIdx.x; t < blockIdx.x; t += THREADS) before += ld_global(tile_sums + t);
    before = block_sum<THREADS>(before, smem);
  }
  // coalesced in, through shared memory to runs of ITEMS per thread and back
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int64_t idx = tile0 + (int64_t)i * THREADS + threadIdx.x;
    stage[i * THREADS + threadIdx.x] = idx < n ? in[idx] : 0;
  }
  __syncthreads();
  int32_t item[ITEMS];
  int64_t local = 0;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    item[i] = stage[threadIdx.x * ITEMS + i];
    local += item[i];
  }
  int64_t x = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane_id() >= o) x += y;
  }
  const int w = threadIdx.x >> 5;
  if (lane_id() == 31) smem[w] = x;
  __syncthreads();
  if (w == 0) {
    const int64_t t = lane_id() < THREADS / 32 ? smem[lane_id()] : 0;
    int64_t s = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane_id() >= o) s += y;
    }
    smem[lane_id()] = s - t;
  }
  __syncthreads();
  int64_t run = before + smem[w] + (x - local);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    if (EXCLUSIVE) {
      stage[threadIdx.x * ITEMS + i] = (int32_t)run;
      run += item[i];
    } else {
      run += item[i];
      stage[threadIdx.x * ITEMS + i] = (int32_t)run;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int64_t idx = tile0 + (int64_t)i * THREADS + threadIdx.x;
    if (idx < n) out[idx] = stage[i * THREADS + threadIdx.x];
  }
  if (tile0 + kTile >= n && threadIdx.x == THREADS - 1) {
    if (total) *total = run;
    if (rep.dst) {
      for (int i = 0; i < rep.words; ++i) rep.dst[i] = __ldcg(rep.src + i);
      rep.dst[rep.words] = (int32_t)(uint32_t)run;
      rep.dst[rep.words + 1] = (int32_t)(run >> 32);
    }
  }
}

// Up to kDirectScan elements that do not lie where the result goes: every block adds up all
// elements before its tile itself, at most 32 loads a thread out of L2, in place of a launch
// for the tile sums (41 000 elements, from the end of the kernel before: 9.9 us with that
// launch, 6.5 so), and 4096 are two blocks' work, not one's (7.6 -> 3.5).
constexpr int kDirectThreads = 512;
constexpr int kDirectTile = 4 * kDirectThreads;

__global__ void __launch_bounds__(kDirectThreads)
scan_direct_kernel(const int32_t* in, int32_t* __restrict__ out, int64_t n,
                   int64_t* __restrict__ total, ScanReport rep) {
  chain_enter();
  constexpr int kWarps = kDirectThreads / 32;
  __shared__ int64_t tile_s[kWarps], before_s[kWarps];
  const int4* in4 = reinterpret_cast<const int4*>(in);
  const int64_t tile0 = (int64_t)blockIdx.x * kDirectTile;
  int64_t before = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < (int)(tile0 / 4); i += kDirectThreads) {
    const int4 v = ld_global(in4 + i);
    before += ((int64_t)v.x + v.y) + ((int64_t)v.z + v.w);
  }
  const int64_t at = tile0 + 4 * threadIdx.x;
  int v[4];
  if (at + 4 <= n) {
    const int4 q = ld_global(in4 + at / 4);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = at + e < n ? ld_global(in + at + e) : 0;
  }
  const int64_t own = ((int64_t)v[0] + v[1]) + ((int64_t)v[2] + v[3]);
  const int lane = lane_id(), w = threadIdx.x >> 5;
  int64_t x = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
    before += __shfl_xor_sync(0xffffffffu, before, o);
  }
  if (lane == 31) {
    tile_s[w] = x;
    before_s[w] = before;
  }
  __syncthreads();
  int64_t run = 0;
#pragma unroll
  for (int k = 0; k < kWarps; ++k) run += before_s[k] + (k < w ? tile_s[k] : 0);
  run += x - own;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    run += v[e];
    v[e] = (int)run;
  }
  if (at + 4 <= n && (uintptr_t)out % 16 == 0) {
    *reinterpret_cast<int4*>(out + at) = make_int4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (at + e < n) out[at + e] = v[e];
  }
  if (tile0 + kDirectTile >= n && threadIdx.x == kDirectThreads - 1) {
    if (total) *total = run;
    if (rep.dst) {
      for (int i = 0; i < rep.words; ++i) rep.dst[i] = __ldcg(rep.src + i);
      rep.dst[rep.words] = (int32_t)(uint32_t)run;
      rep.dst[rep.words + 1] = (int32_t)(run >> 32);
    }
  }
}

constexpr int kOneThreads = 1024;
constexpr int kOneItems = 8;
constexpr int64_t kOneBlock = (int64_t)kOneThreads * kOneItems;   // 8192
// Tiles up to which every block adds up the sums before its own: 33 million elements.
constexpr unsigned kDirectTiles = 8192;

template <bool EXCLUSIVE>
int scan_impl(cudaStream_t st, const int32_t* in, int32_t* out, const ScanSize& size,
              int64_t capacity, int64_t* block_sums, int64_t* total, const ScanReport& rep) {
  ProfScope prof(st, "scan_i32");
  if (capacity <= kOneBlock) {
    TFGPC_CUDA(launch_chained(st, 1, kOneThreads, 0,
        scan_tiles_kernel<kOneThreads, kOneItems, EXCLUSIVE>, in, out, size, nullptr, false, total,
        rep));
    return TFGPC_OK;
  }
  const unsigned tiles = (unsigned)((capacity + kScanTile - 1) / kScanTile);
  TFGPC_CUDA(launch_chained(st, tiles, kScanThreads, 0, scan_reduce_kernel, in, size, block_sums));
  const bool scanned = tiles > kDirectTiles;
  if (scanned) {
    TFGPC_CUDA(launch_chained(st, 1, 1024, 0, scan_sums_kernel, size, block_sums));
  }
  TFGPC_CUDA(launch_chained(st, tiles, kScanThreads, 0,
      scan_tiles_kernel<kScanThreads, kScanItems, EXCLUSIVE>, in, out, size, block_sums, scanned,
      total, rep));
  return TFGPC_OK;
}

}  // namespace

int inclusive_scan_i32(cudaStream_t stream, const int32_t* in, int32_t* out, int64_t n,
                       int64_t* block_sums, int64_t* total, ScanReport rep) {
  if (n <= 0) {
    TFGPC_CUDA(cudaMemsetAsync(total, 0, sizeof(int64_t), stream));
    return TFGPC_OK;
  }
  return scan_impl<false>(stream, in, out, ScanSize{n, nullptr, 0, 0}, n, block_sums, total, rep);
}

int inclusive_scan_apart(cudaStream_t stream, const int32_t* in, int32_t* out, int64_t n,
                         int64_t* total, ScanReport rep) {
  TFGPC_REQUIRE(n > 0 && n <= kDirectScan && in != out && (uintptr_t)in % 16 == 0,
                "scan of too many elements for one launch");
  ProfScope prof(stream, "scan_i32");
  TFGPC_CUDA(launch_chained(stream, blocks_for(n, kDirectTile), kDirectThreads, 0,
      scan_direct_kernel, in, out, n, total, rep));
  return TFGPC_OK;
}

int exclusive_scan_cells(cudaStream_t stream, int32_t* table, const int32_t* num_cells, int dims,
                         int batch_size, int64_t capacity, int64_t* block_sums) {
  return scan_impl<true>(stream, table, table, ScanSize{0, num_cells, dims, batch_size}, capacity,
                         block_sums, nullptr, ScanReport{});
}

}  // namespace tfgpc
