// Device-wide scans (scan.cu).
#pragma once

#include "common.cuh"

namespace tfgpc {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Length of a scan: n, or, with num_cells set, the number of cells of a grid (the
// product of the batch size and the D counts, known on the device only) plus 3.
struct ScanSize {
  int64_t n;
  const int32_t* num_cells;
  int dims, batch_size;
};

// Where the scan's last block writes `words` words of src followed by the 64-bit total
// (mapped host memory, see report_page in common.cuh); dst null: nowhere.
struct ScanReport {
  const int32_t* src = nullptr;
  int32_t* dst = nullptr;
  int words = 0;
};

// int64 elements of scratch for a scan of n elements.
int64_t scan_block_sums_elems(int64_t n);

// out[i] = sum_{j<=i} in[j] (int32, as the reference's ranges are), and the 64-bit
// total to *total (device).  `in` may alias `out`.
int inclusive_scan_i32(cudaStream_t stream, const int32_t* in, int32_t* out, int64_t n,
                       int64_t* block_sums, int64_t* total, ScanReport rep = ScanReport());

// The same of at most kDirectScan counts in one launch; `in` (16-byte aligned) is not `out`.
constexpr int64_t kDirectScan = 65536;
int inclusive_scan_apart(cudaStream_t stream, const int32_t* in, int32_t* out, int64_t n,
                         int64_t* total, ScanReport rep = ScanReport());

// table[i] = sum_{j<i} table[j], in place, over the cells of a grid + 3 (at most
// `capacity` elements).
int exclusive_scan_cells(cudaStream_t stream, int32_t* table, const int32_t* num_cells, int dims,
                         int batch_size, int64_t capacity, int64_t* block_sums);

}  // namespace tfgpc
