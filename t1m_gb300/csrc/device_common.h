// Device helpers of every kernel file: offset lookup, and finding and copying
// the descriptor of a block of a grouped launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace t1m {
namespace gb300 {
namespace {

__device__ __forceinline__ int64_t offs(const int64_t* v, int64_t u, int64_t i) {
  return u >= 0 ? i * u : __ldg(v + i);
}

// Last of n descriptors (sorted by begin(i)) whose begin is at most x, found by
// the whole block at once: a binary search is a chain of dependent loads that
// a short block waits for (seven for a batch of 128).
template <class F>
__device__ __forceinline__ int block_find(int n, int64_t x, F begin) {
  int found = 0;
  for (int b = 0; b < n; b += static_cast<int>(blockDim.x)) {
    const int i = b + static_cast<int>(threadIdx.x);
    found += __syncthreads_count(i < n && begin(i) <= x);
  }
  return found - 1;
}

// Copy a descriptor to shared memory by words (whole block; callers
// synchronise before reading it).
template <class D>
__device__ __forceinline__ void block_copy(D* dst, const D* src) {
  static_assert(sizeof(D) % 4 == 0, "copied by words");
  for (int i = threadIdx.x; i < static_cast<int>(sizeof(D) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
}

}  // namespace
}  // namespace gb300
}  // namespace t1m
