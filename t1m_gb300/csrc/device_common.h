// Device helpers of every kernel file: offset lookup, and finding and copying
// the descriptor of a block of a grouped launch.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

namespace t1m {
namespace gb300 {
namespace {

__device__ __forceinline__ int64_t offs(const int64_t* v, int64_t u, int64_t i) {
  return u >= 0 ? i * u : __ldg(v + i);
}

// Launches under programmatic dependent launch: the kernel may be resident
// before the one ahead of it in the stream has finished (its launch and its
// prologue overlap that one's end), and waits in begin_dependent before it
// touches global memory.
__device__ __forceinline__ void begin_dependent() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Lets the kernel behind this one become resident as soon as every block of
// this one has started, instead of ended.  Only ahead of kernels with one block
// per SM: others gather on the SMs with the most room (a split-K reduction
// behind a product that left 8 SMs free ran mostly on those, 38 -> 51 us).
__device__ __forceinline__ void release_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                             cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // Not on the default streams, which order themselves with other streams.
  const bool own = stream && stream != cudaStreamLegacy && stream != cudaStreamPerThread;
  cfg.numAttrs = own ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Global -> shared copy of one element (4, 8 or 16 bytes) that does not pass
// through registers; src_bytes 0 writes zeros (operands past the tile edge).
template <int kBytes>
__device__ __forceinline__ void cp_async_elem(void* dst, const void* src, bool in) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  const uint32_t n = in ? kBytes : 0u;
  if constexpr (kBytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src),
                 "n"(kBytes), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
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
