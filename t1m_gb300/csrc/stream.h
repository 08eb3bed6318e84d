// Streamed products of small outputs over long contracted bundles (stream.cu).
#pragma once

#include "internal.h"

namespace t1m {
namespace gb300 {

// How the operands are read: unit stride along their rows (M, N) or not; the
// K order to use instead of the plan's (both null: the plan's); the epilogue
// store flags of C in the order of launch_stream (rows = the smaller side).
struct StreamLayout {
  bool a_rows, b_rows;
  const int64_t *a_k, *b_k;
  uint32_t store_flags;
};

// K ranges of a product that runs streamed (complex64, BF16x6) and their
// length, or 0 where it does not.
int stream_splits(int64_t M, int64_t N, int64_t K, int64_t* k_per_split);
cudaError_t launch_stream(const GemmArgs& g, const StreamLayout& lay, int splits,
                          cudaStream_t stream, int* err_flag);
// tc.cu: the layout of a product's operands and output.
StreamLayout stream_layout(const GemmArgs& g, const HostPlan& plan);

}  // namespace gb300
}  // namespace t1m
