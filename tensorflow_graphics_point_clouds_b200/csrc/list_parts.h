// How a sample's list of pairs is dealt to several warps (basis_proj_mma.cuh).
// Host and device: the formula alone, without CUDA headers.
#pragma once

#ifdef __CUDACC__
#define TFGPC_HD __host__ __device__ __forceinline__
#else
#define TFGPC_HD inline
#endif

namespace tfgpc {

// End of part p (1 to parts) of the pairs [begin, end): whole chunks, dealt evenly.
// In 64 bits: the product of chunks and parts passes 2^31 from a list of some seven
// million pairs in 4736 parts on.
TFGPC_HD int part_end(int begin, int end, int p, int parts, int chunk) {
  if (p == parts) return end;
  const long long chunks = ((long long)end - begin + chunk - 1) / chunk;
  const long long upto = begin + chunks * p / parts * chunk;
  return upto < end ? (int)upto : end;
}

}  // namespace tfgpc
