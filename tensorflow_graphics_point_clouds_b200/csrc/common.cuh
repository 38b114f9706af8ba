// Shared host/device helpers of the tfgpc library (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "granted.h"
#include "tfgpc.h"

namespace tfgpc {

// ---- status handling -------------------------------------------------------
// Stores a printf-formatted message for tfgpc_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);
void clear_error();

#define TFGPC_REQUIRE(cond, ...)                          \
  do {                                                    \
    if (!(cond)) return ::tfgpc::fail(TFGPC_EINVAL, __VA_ARGS__); \
  } while (0)

#define TFGPC_CUDA(expr)                                                      \
  do {                                                                        \
    cudaError_t e__ = (expr);                                                 \
    if (e__ != cudaSuccess)                                                   \
      return ::tfgpc::fail(TFGPC_ECUDA, "%s failed: %s (%s:%d)", #expr,       \
                           cudaGetErrorString(e__), __FILE__, __LINE__);      \
  } while (0)

#define TFGPC_LAUNCH_CHECK() TFGPC_CUDA(cudaGetLastError())

// Dispatch on the point dimension, D in [2, 6] (the reference's
// DIMENSION_SWITCH_CALL, shared/cc/kernels/defines.hpp:42-49).
#define TFGPC_DIM_SWITCH(D, ...)                         \
  switch (D) {                                           \
    case 2: { constexpr int kD = 2; __VA_ARGS__; } break; \
    case 3: { constexpr int kD = 3; __VA_ARGS__; } break; \
    case 4: { constexpr int kD = 4; __VA_ARGS__; } break; \
    case 5: { constexpr int kD = 5; __VA_ARGS__; } break; \
    case 6: { constexpr int kD = 6; __VA_ARGS__; } break; \
    default: break;                                      \
  }

inline bool valid_dims(int D) { return D >= TFGPC_MIN_DIMS && D <= TFGPC_MAX_DIMS; }

// Optional per-launch timing (tfgpc_profile_enable): when on, a ProfScope
// brackets the launches made inside its lifetime with two CUDA events on the
// launching stream; tfgpc_profile_collect returns name and duration of every
// scope.  When off it costs one thread-local load.
struct ProfScope {
  ProfScope(cudaStream_t st, const char* name);
  ~ProfScope();
  int slot;
  cudaStream_t st;
};

// While one of these lives, the ProfScopes of this host thread record nothing
// (and so create no events and grow no record table): for entry points that
// promise to allocate nothing.
struct ProfPause {
  ProfPause();
  ~ProfPause();
  bool was_on;
};

// Number of SMs of the current device (cached per device).
int sm_count();

// Lets a kernel take `bytes` of dynamic shared memory: asked of the driver once per device
// and larger size (every launch of a product or projection asked again, 0.6 us each).
template <auto kKernel>
cudaError_t allow_shared(int bytes) {
  static Granted granted[64];
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  auto ask = [](int size) {
    return (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, size);
  };
  return (cudaError_t)(dev >= 0 && dev < 64 ? granted[dev].reach(bytes, ask) : ask(bytes));
}

// Blocking read of a few values (4 .. 4096 bytes, a multiple of 4) from device
// memory, through mapped pinned host memory instead of a copy engine: it does
// not queue behind bulk transfers on other streams.
int read_small(cudaStream_t st, const void* dev_src, size_t bytes, void* host_dst);

// The same page for kernels that deliver their results themselves: its device address
// and, once `st` has been synchronised, its contents on the host.
int report_page(void** dev_page);
int read_report(cudaStream_t st, size_t bytes, void* host_dst);

// For what is enqueued between a report and its reading, and need not be waited for:
// mark_report behind the report, read_marked_report in place of read_report.
int mark_report(cudaStream_t st);
int read_marked_report(size_t bytes, void* host_dst);

// ---- launches ----------------------------------------------------------------
//
// A layer is a chain of some twenty kernels of a few microseconds each, every one reading
// what the one before it wrote.  launch_chained lets the GPU set a kernel up (its blocks,
// their shared and tensor memory) while its predecessor still runs; the kernel calls
// chain_enter() before it touches global memory, which waits until the predecessor has
// finished and its writes are visible.  A kernel that waits there has also waited for
// everything before its predecessor, since that one waited too: chains hold, whatever else
// is on the stream.
template <typename T> struct SameType { typedef T type; };

template <typename... P>
cudaError_t launch_chained(cudaStream_t st, dim3 grid, dim3 block, size_t smem, void (*kern)(P...),
                           typename SameType<P>::type... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Every load of a chained kernel is a plain one: the kernel begins before its inputs are
// written, so that a load on the read-only path (__ldg, or a const __restrict__ parameter,
// which gets it by itself) may be made before the wait.
template <typename T>
__device__ __forceinline__ T ld_global(const T* p) { return *p; }

// Waits for the kernel before this one and, unless the launch is a long one, lets the next
// kernel be set up at once (else that happens as the blocks end).  Nothing but the kernel's own
// parameters, shared memory and tensor memory is touched before it.  Long: more than 4096
// blocks or, in a kernel that states its work, more than eight turns of the grid over `items`,
// per_turn at a time.  (A kernel that states none, like the walks of the grid search, goes by
// its blocks alone, however long each of them works: the kernels behind the walks are small.)
// Set up early beside a long kernel that takes an SM's whole shared memory, the next one
// lives with what is left of the L1 cache, and blocks take their places in another order:
// 524 288 points, us, 1.3 ms kernels before them: kernel-MLP gradients 347 -> 578, dX product
// 1560 -> 1752, projection gradients 2380 -> 2527.
// A kernel with tensor memory calls it behind the barrier that follows its allocation: a
// successor that may come while a block still waits for its columns could take them first and
// then wait for that block.  (With the call before the barrier nothing but the size of these
// kernels' shared memory, 169 KB or more, kept two of them off one SM.)
__device__ __forceinline__ void chain_enter(int64_t items = 0, int64_t per_turn = 0) {
  if (items <= 8 * per_turn && (uint64_t)gridDim.x * gridDim.y * gridDim.z <= 4096)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The wait alone: the next kernel comes as the blocks end.  For kernels of a few blocks per
// SM that all run at once: a successor of the same kind that comes early finds the SMs
// unevenly full and keeps its uneven places (general kernel MLP, four of 8-16 on 94 000 pairs of
// two dimensions: 26 us behind itself with the early release, 19.4 without).
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline unsigned blocks_for(int64_t work, int per_block) {
  int64_t b = (work + per_block - 1) / per_block;
  return (unsigned)(b < 1 ? 1 : b);
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// ---- device helpers --------------------------------------------------------

template <int D>
struct Grid {
  int nc[D];      // cells per dimension
  float inv[D];   // inverse cell size
};

// Loads the D cell counts / inverse cell sizes that the reference keeps in
// device tensors (they are op inputs, so the host never reads them).
template <int D>
__device__ __forceinline__ Grid<D> load_grid(const int32_t* num_cells,
                                             const float* inv_cell) {
  Grid<D> g;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    g.nc[d] = ld_global(num_cells + d);
    g.inv[d] = ld_global(inv_cell + d);
  }
  return g;
}

// Cell of a point: clamp(floor(fma(p, inv_cell, -scaled_min)), 0, cells-1).
// The explicit fma is what the reference's `p*inv - min` compiles to under
// nvcc's default -fmad=true (shared/cc/kernels/grid_utils.h:63-74).
template <int D>
__device__ __forceinline__ void cell_of(const float* p, const float* smin,
                                        const Grid<D>& g, int* cell) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    float rel = __fmaf_rn(p[d], g.inv[d], -smin[d]);
    int c = (int)floorf(rel);
    c = max(c, 0);
    c = min(c, g.nc[d] - 1);
    cell[d] = c;
  }
}

// Key of a cell (shared/cc/kernels/grid_utils.h:85-100).
template <int D>
__device__ __forceinline__ int64_t key_of(const int* cell, const Grid<D>& g,
                                          int batch) {
  int64_t key = 0, acc = 1;
#pragma unroll
  for (int d = D - 1; d >= 0; --d) {
    key += (int64_t)cell[d] * acc;
    acc *= g.nc[d];
  }
  return key + acc * (int64_t)batch;
}

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace tfgpc
