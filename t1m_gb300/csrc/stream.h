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

// How the operands of a product can be fetched, for stream_pays.
enum : int {
  kStreamGathered = 0,  // not loaded by TMA, but unit stride along rows, the first
                        // K mode or both K modes (interleaved order)
  kStreamTma = 1,       // both are plain views that the one-tile kernels load by TMA
  kStreamSectors = 2    // one is read 8 bytes of each 32-byte sector at a time
};
// Whether a product for which stream_splits gives `splits` ranges of `kps` runs
// streamed; `other`, `other_kps`: the K ranges it has otherwise (tiles of 64
// x 128).  Measured as speed against the other form, calls queued among others
// over 260 MB of inputs:
//   gathered: always (96 x 64, K = 36864 interleaved 1.7; 500 x 33 1.6; 64 x
//     129 over 40000 2.1);
//   TMA, more than 64 rows of A (the other form runs over pieces): always (96 x
//     96 over 40000 1.5, 4000 x 33 over 1024 1.8; worst 65 x 4000 0.9);
//   TMA, otherwise: outputs of one tile (64 x 128 over 40000 1.1) and up to
//     seven stages of an SM (64 x 1000 over 4096 1.1, 8 x 4000 over 1024 1.5),
//     beyond only while the k that the busiest SM goes through, 1.1 (one row) to
//     1.8 (64 rows) times as long each, are fewer than in the other form (64 x
//     1000 over 8192 0.8, 64 x 16000 over 1024 0.4, 8 x 4000 over 8192 1.5);
//   sectors: outputs of one tile (64 x 64 over 40425 1.1; 95 x 63 over 16983 1.0,
//     33511 0.9, kept for its error, 1.7e-7 against 1.9e-7), larger ones over K
//     up to 14000 (70 x 70 over 13824 1.2, 23693 0.9; 97 x 65 1.0 over 8645,
//     0.8 over 16983; 500 x 33 1.1 over 13824, 0.5 over 23693).
bool stream_pays(int fetch, int64_t M, int64_t N, int64_t K, int splits, int64_t kps, int other,
                 int64_t other_kps);

// K ranges of a product that runs streamed (complex64, BF16x6) and their
// length, or 0 where it does not.
int stream_splits(int64_t M, int64_t N, int64_t K, int64_t* k_per_split);
cudaError_t launch_stream(const GemmArgs& g, const StreamLayout& lay, int splits,
                          cudaStream_t stream, int* err_flag);
// tc.cu: the kStream* of a product, the layout of its operands and output.
int stream_fetch(const GemmArgs& g, const HostPlan& plan);
StreamLayout stream_layout(const GemmArgs& g, const HostPlan& plan);

}  // namespace gb300
}  // namespace t1m
