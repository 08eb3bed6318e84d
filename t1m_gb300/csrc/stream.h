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
// x 128).  Measured in us, other form / streamed, cold:
//   gathered: always (96 x 64, K = 36864 interleaved 84 / 59; 500 x 33 210 / 140;
//     63 x 1001 over 40001 593 / 223; 8 x 16001 over 8191 1980 / 421);
//   TMA: outputs of one tile (64 x 128 over 40000 51 / 51, 8 x 64 over 1024 1.2
//     times), and larger ones while the k that the busiest SM goes through,
//     1.25 (one row) to 2 (64 rows) times as long each as in the other form,
//     cost no more than the launch saves (140 k): 64 x 1000 over 2048
//     1.04 times, over 40000 131 / 220; 64 x 16000 over 1024 62 / 147,
//     16000 x 33 over 1024 124 / 113;
//   sectors: outputs of one tile, over K up to 20000 where they are large
//     (95 x 63: 48 / 49 over 6061, 82 / 90 over 33511; 64 x 64 67 / 57 there),
//     larger ones up to 8192 (97 x 65: 48 / 46 over 6061, 56 / 75 over 16983;
//     500 x 33: 64 / 67, 125 / 179).
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
