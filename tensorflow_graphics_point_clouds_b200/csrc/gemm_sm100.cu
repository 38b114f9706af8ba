// tcgen05 / TMEM / TMA GEMM with 3-pass bf16 operand splitting (see
// gemm_sm100.cuh).  Persistent kernel, one CTA per SM, warp-specialised:
//   warp 0     TMA producer: streams 128 x 64 tiles of A (hi, mid) and
//              BN x 64 tiles of B (hi, mid) into a shared-memory ring;
//   warp 1     allocates tensor memory and issues the tcgen05.mma instructions
//              (one elected lane); completion is tracked with tcgen05.commit
//              on mbarriers, which also hands ring slots back to the producer;
//   warps 2-5  epilogue: tcgen05.ld the 128 x BN fp32 accumulator out of
//              tensor memory, stage it in swizzled 32 x 32 boxes and hand those
//              to TMA stores, while the MMA warp already works on the next tile
//              in the second accumulator buffer.
// Every wait is bounded: after about a second without progress the kernel sets
// the caller's error flag, stops waiting and drains, so it always terminates
// and frees its tensor memory.
#include <cuda.h>

#include "gemm_sm100.cuh"
#include "basis_proj.cuh"
#include "tc_common.cuh"

namespace tfgpc {

namespace {

constexpr int kBM = 128;           // rows of C per tile (TMEM lanes)
constexpr int kBNMax = 256;        // columns of C per tile (TMEM columns per buffer)
constexpr int kBK = 64;            // reduction elements per ring slot: 128 bytes of bf16
constexpr int kMaxStages = 4;
constexpr int kUmmaK = 16;         // reduction elements per tcgen05.mma (kind::f16)
constexpr int kThreads = 192;
constexpr int kTmemCols = 512;     // two accumulator buffers of 256 columns
constexpr uint32_t kABytes = kBM * kBK * 2;        // one A tile (hi or mid)
constexpr uint32_t kOutBoxBytes = 32 * 32 * 4;     // one 32 x 32 fp32 box of the epilogue
constexpr uint32_t kOutStageBytes = 4 * 2 * kOutBoxBytes;  // 4 epilogue warps, double buffered
constexpr uint32_t kFixedBytes = kOutStageBytes + 1024 /*alignment*/ + 256 /*barriers*/;

// One ring slot holds the A and B tiles (hi and mid) of 64 reduction elements; narrow
// tiles leave room for more slots.
inline uint32_t stage_bytes(int bn) { return 2 * kABytes + 2 * (uint32_t)bn * kBK * 2; }
inline int stages_for(int bn) {
  const int s = (int)((227u * 1024u - kFixedBytes) / stage_bytes(bn));
  return s < kMaxStages ? s : kMaxStages;
}

using namespace tc;

// One 32-byte store (sm_100: 256-bit vector access to global memory).
__device__ __forceinline__ void st_global_256(void* p, const uint4& lo, const uint4& hi) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y),
                 "r"(hi.z), "r"(hi.w) : "memory");
}

// Writes 2 channels x 16 basis functions (v[0..31]) of sample `row` into the
// operand image of the tensor-core gradient kernel (basis_proj_grads_tc.cu).
// The row's two chunks (k 0-7, k 8-15) of a channel share one 32-byte sector,
// in swapped order when the channel is odd: one 256-bit store per part, and the
// lanes of neighboring samples fill whole 128-byte lines.
__device__ __forceinline__ void store_image_row(uint8_t* image, int channels, int group_size,
                                                int64_t row, int ch0, const uint32_t* v) {
  const int64_t part = (int64_t)channels * 128;   // bytes of the hi (or mid) rows of a group
  const int64_t gi = row / group_size;
  uint8_t* group = image + gi * (2 * part);
  const int sl = (int)(row - gi * group_size);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int ch = ch0 + u;
    uint4 hv[2], mv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int b = 16 * u + 8 * h;
      split2_bf16(__uint_as_float(v[b]), __uint_as_float(v[b + 1]), hv[h].x, mv[h].x);
      split2_bf16(__uint_as_float(v[b + 2]), __uint_as_float(v[b + 3]), hv[h].y, mv[h].y);
      split2_bf16(__uint_as_float(v[b + 4]), __uint_as_float(v[b + 5]), hv[h].z, mv[h].z);
      split2_bf16(__uint_as_float(v[b + 6]), __uint_as_float(v[b + 7]), hv[h].w, mv[h].w);
    }
    const bool swap = (ch & 1) != 0;
    const uint4 h_lo = swap ? hv[1] : hv[0], h_hi = swap ? hv[0] : hv[1];
    const uint4 m_lo = swap ? mv[1] : mv[0], m_hi = swap ? mv[0] : mv[1];
    uint8_t* dst = group + (int64_t)ch * 128 + (((2 * sl) ^ (ch & 6)) << 4);
    st_global_256(dst, h_lo, h_hi);
    st_global_256(dst + part, m_lo, m_hi);
  }
}

struct TileSchedule {
  int m_tiles, n_tiles, batches, k_splits;
  int k_blocks;         // ring slots over the whole reduction
  int k_blocks_per_split;
  int add_slices;       // 1: every slice of the reduction is added into the one output
  int slice_batches;    // > 0: slice s of batch b goes to matrix s * slice_batches + b of C
};

struct Barriers {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

// OUT = 0: C as fp32 through TMA stores.  OUT = 2: the map of C describes C^T ([N, M]
// row-major): boxes are transposed on their way through shared memory, for products
// whose natural left operand is the small matrix.  OUT = 3: C^T is the gradient of a
// [rows, channels, 16] projection and is written as the bf16 hi/mid operand image the
// tensor-core gradient kernel loads with one bulk copy per group of four rows
// (basis_proj_grads_tc.cu describes the layout).
// OUT = 4: like 2, but row j of C^T goes to row row_order[j] of the output
// (`image` is then the fp32 output, image_channels its row length): the rows of a
// product computed in another sequence than the caller's are put back in place.
template <bool A_MN, bool B_MN, int OUT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16x3_kernel(const __grid_constant__ CUtensorMap tm_a_hi,
                   const __grid_constant__ CUtensorMap tm_a_mid,
                   const __grid_constant__ CUtensorMap tm_b_hi,
                   const __grid_constant__ CUtensorMap tm_b_mid,
                   const __grid_constant__ CUtensorMap tm_c, int64_t m_total, int64_t n_total,
                   int bn, int stages, uint32_t idesc, TileSchedule sch, int* err_flag,
                   const float* bias, uint8_t* image, int image_channels,
                   int image_group, const int32_t* row_order) {
  extern __shared__ uint8_t smem_raw[];
  // the swizzled tiles need 1024-byte alignment
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t b_bytes = (uint32_t)bn * kBK * 2;            // one B tile (hi or mid)
  const uint32_t slot_bytes = 2 * kABytes + 2 * b_bytes;
  uint8_t* out_stage = smem + (size_t)stages * slot_bytes;    // 1024-byte aligned
  Barriers* bars = (Barriers*)(out_stage + kOutStageBytes);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int total_tiles = sch.m_tiles * sch.n_tiles * sch.batches * sch.k_splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&bars->full[s]), 1);
      mbar_init(smem_u32(&bars->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bars->acc_full[b]), 1);
      mbar_init(smem_u32(&bars->acc_empty[b]), 4);
    }
    bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(&bars->tmem_base), kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_enter((int64_t)total_tiles * 4, gridDim.x);
  const uint32_t tmem_base = *(volatile uint32_t*)&bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;

  // tile -> (m, n, batch, split); m fastest so that CTAs running together share B/k-slices
  auto decode = [&](int t, int& m, int& n, int& bt, int& sp) {
    m = t % sch.m_tiles;
    int r = t / sch.m_tiles;
    n = r % sch.n_tiles;
    r /= sch.n_tiles;
    bt = r % sch.batches;
    sp = r / sch.batches;
  };

  if (warp == 0) {
    // ---------------------------------------------------------- TMA producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        int m, n, bt, sp;
        decode(t, m, n, bt, sp);
        const int kb0 = sp * sch.k_blocks_per_split;
        const int kb1 = min(kb0 + sch.k_blocks_per_split, sch.k_blocks);
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(smem_u32(&bars->empty[s]), ph ^ 1, abort_flag, err_flag);
          const uint32_t full = smem_u32(&bars->full[s]);
          mbar_expect_tx(full, slot_bytes);
          uint8_t* st = smem + (size_t)s * slot_bytes;
          if (++s == stages) { s = 0; ph ^= 1; }
          const uint32_t a_hi = smem_u32(st), a_mid = a_hi + kABytes;
          const uint32_t b_hi = a_mid + kABytes, b_mid = b_hi + b_bytes;
          if (!A_MN) {
            tma_load_3d(a_hi, &tm_a_hi, kb * kBK, m * kBM, bt, full);
            tma_load_3d(a_mid, &tm_a_mid, kb * kBK, m * kBM, bt, full);
          } else {
            // two boxes of 64 (M) x 64 (K rows): 8 KB each
            for (int j = 0; j < kBM / 64; ++j) {
              tma_load_3d(a_hi + j * 8192, &tm_a_hi, m * kBM + j * 64, kb * kBK, bt, full);
              tma_load_3d(a_mid + j * 8192, &tm_a_mid, m * kBM + j * 64, kb * kBK, bt, full);
            }
          }
          if (!B_MN) {
            tma_load_3d(b_hi, &tm_b_hi, kb * kBK, n * bn, bt, full);
            tma_load_3d(b_mid, &tm_b_mid, kb * kBK, n * bn, bt, full);
          } else {
            for (int j = 0; j < bn / 64; ++j) {
              tma_load_3d(b_hi + j * 8192, &tm_b_hi, n * bn + j * 64, kb * kBK, bt, full);
              tma_load_3d(b_mid + j * 8192, &tm_b_mid, n * bn + j * 64, kb * kBK, bt, full);
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      int tile_iter = 0;
      for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++tile_iter) {
        int m, n, bt, sp;
        decode(t, m, n, bt, sp);
        const int kb0 = sp * sch.k_blocks_per_split;
        const int kb1 = min(kb0 + sch.k_blocks_per_split, sch.k_blocks);
        const int buf = tile_iter & 1;
        mbar_wait(smem_u32(&bars->acc_empty[buf]), ((tile_iter >> 1) & 1) ^ 1, abort_flag, err_flag);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)buf * kBNMax;
        uint32_t accumulate = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(smem_u32(&bars->full[s]), ph, abort_flag, err_flag);
          tc_fence_after();
          uint8_t* st = smem + (size_t)s * slot_bytes;
          const uint32_t a_hi = smem_u32(st), a_mid = a_hi + kABytes;
          const uint32_t b_hi = a_mid + kABytes, b_mid = b_hi + b_bytes;
          // K-major: rows of 128 bytes, 8-row swizzle atoms 1024 bytes apart;
          // one UMMA_K step is 32 bytes inside the row.
          // MN-major: 64 (MN) x 8 (K) atoms of 1024 bytes; atoms along K are
          // 1024 bytes apart (stride offset), blocks of 64 along MN are 8192
          // bytes apart (leading offset); one UMMA_K step is 16 K rows.
          const uint32_t a_step = A_MN ? 16 * 128 : 32;
          const uint32_t b_step = B_MN ? 16 * 128 : 32;
          const uint32_t a_lbo = A_MN ? 8192 : 16, b_lbo = B_MN ? 8192 : 16;
#pragma unroll
          for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
            const uint64_t da_hi = make_desc(a_hi + kk * a_step, a_lbo, 1024);
            const uint64_t da_mid = make_desc(a_mid + kk * a_step, a_lbo, 1024);
            const uint64_t db_hi = make_desc(b_hi + kk * b_step, b_lbo, 1024);
            const uint64_t db_mid = make_desc(b_mid + kk * b_step, b_lbo, 1024);
            umma_bf16(d_tmem, da_hi, db_mid, idesc, accumulate);
            umma_bf16(d_tmem, da_mid, db_hi, idesc, 1u);
            umma_bf16(d_tmem, da_hi, db_hi, idesc, 1u);
            accumulate = 1u;
          }
          umma_commit(smem_u32(&bars->empty[s]));  // slot free once these MMAs have read it
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        umma_commit(smem_u32(&bars->acc_full[buf]));
      }
    }
  } else {
    // -------------------------------------------------------------- epilogue
    // Each warp drains its 32 accumulator rows 32 columns at a time: tcgen05.ld
    // to registers, a 128-byte-swizzled 32 x 32 box in shared memory (lane =
    // row, so the swizzle makes the 16-byte writes of a quarter warp hit
    // distinct banks), then one TMA store per box, double buffered.  TMA clips
    // the rows and columns beyond the edge of C.
    const int quarter = warp & 3;  // TMEM lanes this warp may read: 32*quarter ...
    uint8_t* my_stage = out_stage + (size_t)quarter * 2 * kOutBoxBytes;
    uint32_t box_iter = 0;
    int tile_iter = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++tile_iter) {
      int m, n, bt, sp;
      decode(t, m, n, bt, sp);
      const int buf = tile_iter & 1;
      mbar_wait(smem_u32(&bars->acc_full[buf]), (tile_iter >> 1) & 1, abort_flag, err_flag);
      tc_fence_after();
      const int row0 = m * kBM + quarter * 32;
      for (int c0 = 0; c0 < bn; c0 += 32, ++box_iter) {
        // Boxes beyond the last column or row hold nothing to store.  They must
        // not touch the staging buffers either: the wait below only covers the
        // buffer's previous store if every box written here also issues one.
        if ((int64_t)n * bn + c0 >= n_total || row0 >= m_total) break;
        uint32_t r[32];
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) +
                               (uint32_t)(buf * kBNMax + c0);
        tmem_ld_32x32(taddr, r);
        if (OUT == 4) {
          // as OUT == 3 below: after the transposition this thread holds columns
          // row0 .. row0 + 31 of C^T's row n * bn + c0 + lane, 128 contiguous bytes
          uint8_t* box = my_stage;
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            *reinterpret_cast<uint32_t*>(box + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) +
                                         (lane & 3) * 4) = r[i];
          __syncwarp();
          const int64_t j = (int64_t)n * bn + c0 + lane;
          if (j < n_total && !*abort_flag) {
            float* dst = reinterpret_cast<float*>(image) +
                         (int64_t)ld_global(row_order + j) * image_channels + row0;
            if (row0 + 32 <= m_total) {
#pragma unroll
              for (int q = 0; q < 8; q += 2)   // whole 32-byte sectors per store
                st_global_256(dst + 4 * q,
                              *reinterpret_cast<const uint4*>(box + lane * 128 + ((q ^ (lane & 7)) << 4)),
                              *reinterpret_cast<const uint4*>(box + lane * 128 + (((q + 1) ^ (lane & 7)) << 4)));
            } else {
              for (int e = 0; row0 + e < m_total; ++e)
                dst[e] = *reinterpret_cast<const float*>(box + lane * 128 +
                                                         (((e >> 2) ^ (lane & 7)) << 4) + (e & 3) * 4);
            }
          }
          continue;
        }
        if (OUT == 3) {
          // C^T tile: this thread holds 32 rows (samples c0 .. c0+31 of the tile)
          // of column row0 + lane.  Transposed through the warp's staging box, it
          // holds 32 consecutive columns (2 channels x 16) of sample c0 + lane.
          uint8_t* box = my_stage;
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            *reinterpret_cast<uint32_t*>(box + i * 128 + (((lane >> 2) ^ (i & 7)) << 4) +
                                         (lane & 3) * 4) = r[i];
          __syncwarp();
          uint32_t v[32];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 t4 = *reinterpret_cast<const uint4*>(box + lane * 128 + ((q ^ (lane & 7)) << 4));
            v[4 * q] = t4.x; v[4 * q + 1] = t4.y; v[4 * q + 2] = t4.z; v[4 * q + 3] = t4.w;
          }
          const int64_t sample = (int64_t)n * bn + c0 + lane;
          if (sample < n_total && !*abort_flag)
            store_image_row(image, image_channels, image_group, sample, row0 / 16, v);
          continue;
        }
        if (OUT == 0 && bias && sp == 0) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int64_t col = (int64_t)n * bn + c0 + i;
            if (col < n_total) r[i] = __float_as_uint(__uint_as_float(r[i]) + ld_global(bias + col));
          }
        }
        if (OUT == 2 && bias && sp == 0 && row0 + lane < m_total) {
          const float v = ld_global(bias + row0 + lane);
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + v);
        }
        uint8_t* box = my_stage + (size_t)(box_iter & 1) * kOutBoxBytes;
        if (lane == 0) tma_store_wait_read<1>();  // the store that last used this box has read it
        __syncwarp();
        if (OUT == 2) {
          // box row i = column c0 + i of the tile, box column = this lane's row:
          // a warp store fills one (swizzled) 128-byte row, no bank conflicts
#pragma unroll
          for (int i = 0; i < 32; ++i)
            *reinterpret_cast<uint32_t*>(box + i * 128 + ((((lane >> 2) ^ (i & 7))) << 4) +
                                         (lane & 3) * 4) = r[i];
        } else {
          float4* rowp = reinterpret_cast<float4*>(box + lane * 128);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            rowp[q ^ (lane & 7)] =
                make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                            __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
        fence_proxy_async();
        __syncwarp();
        const int col0 = n * bn + c0;
        if (lane == 0 && row0 < m_total && col0 < n_total && !*abort_flag) {
          const int x = OUT == 2 ? row0 : col0, y = OUT == 2 ? col0 : row0;
          if (sch.add_slices)
            tma_reduce_add_3d(&tm_c, smem_u32(box), x, y, bt);
          else
            tma_store_3d(&tm_c, smem_u32(box), x, y, bt + sp * sch.slice_batches);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[buf]));
    }
    if (lane == 0) tma_store_wait_read<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---- host side ---------------------------------------------------------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 3-D bf16 tensor map: dim0 (contiguous) x dim1 rows x batches, 128-byte swizzle, zero
// fill beyond the edges of a batch's own matrix.
int make_map(CUtensorMap* map, const __nv_bfloat16* base, const GemmOperand& op, int64_t dim0,
             int64_t dim1, int batches, int box0, int box1) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(TFGPC_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
  if ((uintptr_t)base % 16 != 0 || (op.ld * 2) % 16 != 0 || (op.batch_stride * 2) % 16 != 0)
    return fail(TFGPC_EINVAL, "tensor-core GEMM operands need 16-byte aligned rows (ld %lld)",
                (long long)op.ld);
  cuuint64_t dims[3] = {(cuuint64_t)dim0, (cuuint64_t)dim1, (cuuint64_t)batches};
  cuuint64_t strides[2] = {(cuuint64_t)op.ld * 2,
                           (cuuint64_t)(batches > 1 ? op.batch_stride : dim1 * op.ld) * 2};
  cuuint32_t box[3] = {(cuuint32_t)box0, (cuuint32_t)box1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TFGPC_ECUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  return TFGPC_OK;
}

// 3-D fp32 tensor map of C: (columns, rows, batches), boxes of 32 x 32 x 1 with the
// 128-byte swizzle the epilogue writes its staging boxes in.
int make_map_c(CUtensorMap* map, float* base, int64_t n, int64_t m, int batches, int64_t ldc,
               int64_t batch_stride) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(TFGPC_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
  if ((uintptr_t)base % 16 != 0 || ldc % 4 != 0 || batch_stride % 4 != 0)
    return fail(TFGPC_EINVAL, "tensor-core GEMM output needs 16-byte aligned rows (ld %lld)",
                (long long)ldc);
  cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)m, (cuuint64_t)batches};
  cuuint64_t strides[2] = {(cuuint64_t)ldc * 4,
                           (cuuint64_t)(batches > 1 ? batch_stride : m * ldc) * 4};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TFGPC_ECUDA, "cuTensorMapEncodeTiled (C) failed with %d", (int)r);
  return TFGPC_OK;
}

// Columns of C per tile: a multiple of 32 (epilogue chunk), of 64 for MN-major B boxes.
int tile_columns(int64_t N, bool b_mn) {
  const int gran = b_mn ? 64 : 32;
  const int bn = (int)(N < kBNMax ? N : kBNMax);
  return (bn + gran - 1) / gran * gran;
}

// The four operand maps of a product with M x N tiles of kBM x bn.
int operand_maps(CUtensorMap* maps, const GemmOperand& a, const GemmOperand& b, int64_t M,
                 int64_t N, int64_t K, int batches, int bn) {
  const __nv_bfloat16* ap[2] = {a.hi, a.mid};
  const __nv_bfloat16* bp[2] = {b.hi, b.mid};
  for (int i = 0; i < 2; ++i) {
    int rc = a.major == Major::MN ? make_map(&maps[i], ap[i], a, M, K, batches, 64, kBK)
                                  : make_map(&maps[i], ap[i], a, K, M, batches, kBK, kBM);
    if (rc) return rc;
    rc = b.major == Major::MN ? make_map(&maps[2 + i], bp[i], b, N, K, batches, 64, kBK)
                              : make_map(&maps[2 + i], bp[i], b, K, N, batches, kBK, bn);
    if (rc) return rc;
  }
  return TFGPC_OK;
}

TileSchedule schedule(int64_t M, int64_t N, int64_t K, int batches, int bn, int k_splits) {
  TileSchedule sch;
  sch.m_tiles = (int)((M + kBM - 1) / kBM);
  sch.n_tiles = (int)((N + bn - 1) / bn);
  sch.batches = batches;
  sch.k_blocks = (int)((K + kBK - 1) / kBK);
  sch.k_splits = k_splits < sch.k_blocks ? k_splits : sch.k_blocks;
  sch.k_blocks_per_split = (sch.k_blocks + sch.k_splits - 1) / sch.k_splits;
  // drop empty trailing slices
  sch.k_splits = (sch.k_blocks + sch.k_blocks_per_split - 1) / sch.k_blocks_per_split;
  sch.add_slices = sch.k_splits > 1 ? 1 : 0;
  sch.slice_batches = 0;
  return sch;
}

// Instruction descriptor of tcgen05.mma kind::f16: D fp32, A and B bf16.
uint32_t make_idesc(int m, int n, bool a_mn, bool b_mn) {
  uint32_t d = 0;
  d |= 1u << 4;                       // D format: f32
  d |= 1u << 7;                       // A format: bf16
  d |= 1u << 10;                      // B format: bf16
  d |= (a_mn ? 1u : 0u) << 15;        // A major: 0 = K, 1 = MN
  d |= (b_mn ? 1u : 0u) << 16;        // B major
  d |= (uint32_t)(n >> 3) << 17;      // N / 8
  d |= (uint32_t)(m >> 4) << 24;      // M / 16
  return d;
}

template <bool A_MN, bool B_MN, int OUT = 0>
int launch(cudaStream_t st, const CUtensorMap* maps, int64_t M, int64_t N, int bn,
           TileSchedule sch, int* err_flag, const float* bias = nullptr, uint8_t* image = nullptr,
           int image_channels = 0, int image_group = 4, const int32_t* row_order = nullptr) {
  auto kern = gemm_bf16x3_kernel<A_MN, B_MN, OUT>;
  const int stages = stages_for(bn);
  const size_t smem = (size_t)stages * stage_bytes(bn) + kFixedBytes;
  TFGPC_CUDA((allow_shared<gemm_bf16x3_kernel<A_MN, B_MN, OUT>>((int)smem)));
  const int64_t tiles = (int64_t)sch.m_tiles * sch.n_tiles * sch.batches * sch.k_splits;
  const int grid = tiles < sm_count() ? (int)tiles : sm_count();
  ProfScope prof(st, OUT == 4 ? "gemm_bf16x3_mn_k_scatter" : OUT == 3 ? "gemm_bf16x3_mn_k_image"
                     : OUT == 2 ? "gemm_bf16x3_mn_k_t"
                     : A_MN ? (B_MN ? "gemm_bf16x3_mn_mn" : "gemm_bf16x3_mn_k")
                            : (B_MN ? "gemm_bf16x3_k_mn" : "gemm_bf16x3_k_k"));
  TFGPC_CUDA(launch_chained(st, grid, kThreads, smem, kern, maps[0], maps[1], maps[2], maps[3],
      maps[4], M, N, bn, stages, make_idesc(kBM, bn, A_MN, B_MN), sch, err_flag, bias, image,
      image_channels, image_group, row_order));
  return TFGPC_OK;
}

// One warp that waits, through the same bounded wait as every role of the
// GEMM, for a barrier phase that nothing ever completes: the wait gives up after
// `limit_ns`, records that in the status word and the kernel returns.
__global__ void wait_probe_kernel(int* err_flag, unsigned long long limit_ns, int* returned) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_wait_limit(smem_u32(&bar), 0, &abort_flag, err_flag, limit_ns);
    *returned = 1;
  }
}

// out = the sum of `slices` slices, one after the other (and the bias, [cols] or
// null), four values per thread.
__global__ void __launch_bounds__(256)
sum_slices_kernel(const float* partials, int slices, int batches, int64_t rows,
                  int cols, const float* bias, float* __restrict__ out, int64_t ldc,
                  int64_t c_batch_stride) {
  chain_enter();
  const int quads = cols / 4;
  const int64_t per_slice = (int64_t)batches * rows * quads;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= per_slice) return;
  const float4* src = reinterpret_cast<const float4*>(partials) + i;
  float4 v = ld_global(src);
#pragma unroll 4
  for (int s = 1; s < slices; ++s) {
    const float4 t = ld_global(src + (int64_t)s * per_slice);
    v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
  }
  const int64_t r = i / quads;
  const int c = (int)(i - r * quads) * 4;
  if (bias) {
    v.x += ld_global(bias + c); v.y += ld_global(bias + c + 1);
    v.z += ld_global(bias + c + 2); v.w += ld_global(bias + c + 3);
  }
  const int64_t b = r / rows;
  *reinterpret_cast<float4*>(out + b * c_batch_stride + (r - b * rows) * ldc + c) = v;
}

// hi_t, mid_t [cols, rows] = the split of the transpose of x, whose rows and columns are
// padded with zeros as in split_block (prepare.cu).
__global__ void split_transpose_kernel(const float* x, int64_t rows, int64_t cols,
                                       int cols_src, int k_src, int k_dst,
                                       __nv_bfloat16* __restrict__ hi_t,
                                       __nv_bfloat16* __restrict__ mid_t) {
  chain_enter();
  __shared__ float tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, c0 = (int64_t)blockIdx.x * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int64_t r = r0 + j, cc = c0 + threadIdx.x;
    const int64_t ch = r / k_dst;
    const int k = (int)(r - ch * k_dst);
    tile[j][threadIdx.x] = (r < rows && cc < cols_src && k < k_src)
                               ? ld_global(x + (ch * k_src + k) * cols_src + cc) : 0.0f;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    int64_t cc = c0 + j, r = r0 + threadIdx.x;
    if (cc < cols && r < rows) {
      __nv_bfloat16 h, l;
      split_bf16(tile[threadIdx.x][j], h, l);
      hi_t[cc * rows + r] = h;
      mid_t[cc * rows + r] = l;
    }
  }
}

}  // namespace

// The tensor cores add into their fp32 accumulator by truncation, so the error of
// a sum grows with the number of terms one accumulator takes: measured on the
// weight-gradient product of the layer (K = 524 288 samples in 9 slices) it was
// 7e-4 of the result's rms, against 9e-5 for K = 65 536 and 2e-5 for an fp32
// FMA loop; with slices of 8192 / 4096 / 2048 terms 9.6e-5 / 5.9e-5 / 3.4e-5.
// K is therefore cut into slices of at most kMaxChain terms, whose results are
// summed in round-to-nearest fp32.
constexpr int64_t kMaxChain = 2048;

static int pick_k_splits(int64_t tiles, int64_t K) {
  const int64_t sms = sm_count(), k_blocks = (K + kBK - 1) / kBK;
  const int64_t chain = (K + kMaxChain - 1) / kMaxChain;
  // As many slices as the last wave of tiles has room for (a slice of eight slots or
  // more pays for its share of the output): 8 tiles of a 41 000-sample weight gradient
  // ran as 168 slices in two waves, the second of 20.
  const int64_t waves = (tiles * chain + sms - 1) / sms;
  int64_t splits = waves <= 4 ? waves * sms / tiles : chain;
  const int64_t most = k_blocks / 8;
  if (splits > most) splits = most;
  if (splits < chain) splits = chain;
  return (int)(splits < 1 ? 1 : splits);
}

int64_t gemm_partial_elems(int64_t M, int64_t N, int64_t K, bool b_mn) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int bn = tile_columns(N, b_mn);
  const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn);
  const int splits = schedule(M, N, K, 1, bn, pick_k_splits(tiles, K)).k_splits;
  return splits > 2 ? splits * M * N : 0;
}

int gemm_bf16x3_grad_image_tn(cudaStream_t stream, int channels, int64_t N, int64_t K,
                              const GemmOperand& a, const GemmOperand& b, void* image, int group,
                              int* err_flag) {
  const int64_t M = (int64_t)channels * 16;
  TFGPC_REQUIRE(channels > 0 && N > 0 && K > 0 && N < (int64_t)INT32_MAX && K < (int64_t)INT32_MAX,
                "GEMM expects positive sizes below 2^31");
  TFGPC_REQUIRE(a.major == Major::MN && b.major == Major::K && channels % 2 == 0 &&
                (uintptr_t)image % 32 == 0 && group >= 1 && group <= 4,
                "gradient-image GEMM (transposed form) expects an MN-major left and a K-major "
                "right operand and groups of 1 to 4 rows");
  const int bn = tile_columns(N, false);
  CUtensorMap maps[5] = {};
  int rc = operand_maps(maps, a, b, M, N, K, 1, bn);
  if (rc) return rc;
  return launch<true, false, 3>(stream, maps, M, N, bn, schedule(M, N, K, 1, bn, 1), err_flag,
                                nullptr, (uint8_t*)image, channels, group);
}

int gemm_bf16x3_tn_scatter(cudaStream_t stream, int64_t M, int64_t N, int64_t K,
                           const GemmOperand& a, const GemmOperand& b, float* out, int64_t ld_out,
                           const int32_t* row_order, int* err_flag) {
  TFGPC_REQUIRE(M > 0 && N > 0 && K > 0 && M < (int64_t)INT32_MAX && N < (int64_t)INT32_MAX &&
                K < (int64_t)INT32_MAX && ld_out < (int64_t)INT32_MAX,
                "GEMM expects positive sizes below 2^31");
  TFGPC_REQUIRE(a.major == Major::MN && b.major == Major::K && row_order && out &&
                (uintptr_t)out % 32 == 0 && ld_out % 8 == 0,
                "row-scattering GEMM expects an MN-major left and a K-major right operand and "
                "32-byte aligned output rows");
  const int bn = tile_columns(N, false);
  CUtensorMap maps[5] = {};
  int rc = operand_maps(maps, a, b, M, N, K, 1, bn);
  if (rc) return rc;
  return launch<true, false, 4>(stream, maps, M, N, bn, schedule(M, N, K, 1, bn, 1), err_flag,
                                nullptr, (uint8_t*)out, (int)ld_out, 4, row_order);
}

// Tiles and slices of a product; slice_batches > 0: its slices are kept apart.
static TileSchedule schedule_of(const GemmProblem& p) {
  const int bn = tile_columns(p.N, p.b.major == Major::MN);
  const int64_t tiles = ((p.M + kBM - 1) / kBM) * ((p.N + bn - 1) / bn) * p.batches;
  const int64_t cols = p.transposed ? p.M : p.N;
  int splits = pick_k_splits(tiles, p.K);
  if (p.ordered && splits > 2) {
    const int64_t room = cols % 4 == 0 ? p.partial_elems / (p.M * p.N * p.batches) : 0;
    splits = (int)(room > 2 ? (room < splits ? room : splits) : 2);
  }
  TileSchedule sch = schedule(p.M, p.N, p.K, p.batches, bn, splits);
  if (p.ordered && sch.k_splits > 2) {
    sch.add_slices = 0;
    sch.slice_batches = p.batches;
  }
  return sch;
}

bool gemm_adds_slices(const GemmProblem& p) { return schedule_of(p).add_slices != 0; }

int gemm_bf16x3(cudaStream_t stream, const GemmProblem& p, int* err_flag) {
  TFGPC_REQUIRE(p.M > 0 && p.N > 0 && p.K > 0 && p.batches > 0, "GEMM expects positive sizes");
  TFGPC_REQUIRE(p.M < (int64_t)INT32_MAX && p.N < (int64_t)INT32_MAX && p.K < (int64_t)INT32_MAX,
                "GEMM sizes must stay below 2^31");
  const bool a_mn = p.a.major == Major::MN, b_mn = p.b.major == Major::MN;
  TFGPC_REQUIRE(!p.transposed || (a_mn && !b_mn),
                "transposed-output GEMM expects an MN-major left and a K-major right operand");
  const int bn = tile_columns(p.N, b_mn);
  CUtensorMap maps[5] = {};
  int rc = operand_maps(maps, p.a, p.b, p.M, p.N, p.K, p.batches, bn);
  if (rc) return rc;
  const int64_t rows = p.transposed ? p.N : p.M, cols = p.transposed ? p.M : p.N;
  const TileSchedule sch = schedule_of(p);
  const bool apart = sch.slice_batches > 0;
  if (sch.add_slices && !p.cleared) {
    // the slices are added into c, which starts from zero, by the store unit (the order
    // of the additions, and with it the last bits of the sums, varies from run to run)
    const bool dense = p.batches == 1 ? p.ldc == cols
                                      : (p.c_batch_stride == cols && p.ldc == cols * p.batches) ||
                                            (p.ldc == cols && p.c_batch_stride == cols * rows);
    if (dense) {
      TFGPC_CUDA(cudaMemsetAsync(p.c, 0, sizeof(float) * (size_t)rows * cols * p.batches, stream));
    } else {
      for (int b = 0; b < p.batches; ++b)
        TFGPC_CUDA(cudaMemset2DAsync(p.c + b * p.c_batch_stride, sizeof(float) * (size_t)p.ldc, 0,
                                     sizeof(float) * (size_t)cols, (size_t)rows, stream));
    }
  }
  rc = apart ? make_map_c(&maps[4], p.partials, cols, rows, sch.k_splits * p.batches, cols,
                          rows * cols)
             : make_map_c(&maps[4], p.c, cols, rows, p.batches, p.ldc, p.c_batch_stride);
  if (rc) return rc;
  const float* bias = apart ? nullptr : p.bias;
  if (p.transposed)
    rc = launch<true, false, 2>(stream, maps, p.M, p.N, bn, sch, err_flag, bias);
  else if (a_mn && b_mn)
    rc = launch<true, true>(stream, maps, p.M, p.N, bn, sch, err_flag, bias);
  else if (a_mn)
    rc = launch<true, false>(stream, maps, p.M, p.N, bn, sch, err_flag, bias);
  else if (b_mn)
    rc = launch<false, true>(stream, maps, p.M, p.N, bn, sch, err_flag, bias);
  else
    rc = launch<false, false>(stream, maps, p.M, p.N, bn, sch, err_flag, bias);
  if (rc || !apart) return rc;
  ProfScope prof(stream, "sum_slices");
  TFGPC_CUDA(launch_chained(stream, blocks_for(p.batches * rows * (cols / 4), 256), 256, 0,
      sum_slices_kernel, p.partials, sch.k_splits, p.batches, rows, (int)cols, p.bias, p.c, p.ldc,
      p.c_batch_stride));
  return TFGPC_OK;
}

int split_transpose_to_bf16(cudaStream_t stream, const float* x, int64_t rows, int64_t cols,
                            int cols_src, int k_src, int k_dst, __nv_bfloat16* hi_t,
                            __nv_bfloat16* mid_t) {
  if (rows <= 0 || cols <= 0) return TFGPC_OK;
  dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
  TFGPC_CUDA(launch_chained(stream, grid, dim3(32, 8), 0, split_transpose_kernel, x, rows, cols,
      cols_src, k_src, k_dst, hi_t, mid_t));
  return TFGPC_OK;
}

}  // namespace tfgpc

// Exercises the bounded wait of the tensor-core kernels (see include/tfgpc.h).
extern "C" int tfgpc_debug_bounded_wait(void* stream, void* ws, size_t ws_bytes,
                                        unsigned limit_us, int* returned_out) {
  using namespace tfgpc;
  TFGPC_REQUIRE(ws && returned_out && ws_bytes >= 1024 && (uintptr_t)ws % 256 == 0,
                "debug_bounded_wait expects a 256-byte aligned workspace of at least 1024 bytes");
  TFGPC_REQUIRE(limit_us >= 1 && limit_us <= 100000,
                "debug_bounded_wait expects a limit between 1 us and 100 ms");
  cudaStream_t st = (cudaStream_t)stream;
  // word 0 is the status word tfgpc_mcconv_status reads, word 1 the kernel's
  // "I returned" mark
  int* words = (int*)ws;
  TFGPC_CUDA(cudaMemsetAsync(words, 0, 2 * sizeof(int), st));
  wait_probe_kernel<<<1, 32, 0, st>>>(words, (unsigned long long)limit_us * 1000ull, words + 1);
  TFGPC_LAUNCH_CHECK();
  int back[2] = {0, 0};
  int rc = read_small(st, words, sizeof(back), back);
  if (rc) return rc;
  *returned_out = back[1];
  return TFGPC_OK;
}

