// Tile of a plain product with a forced number of K ranges: the tile of the
// same product with as many ranges as it has k steps, where more are forced.
#include <cstdio>

#include "internal.h"
#include "t1m_capi.h"

using namespace t1m::gb300;

int main() {
  int failures = 0;
  for (int dtype : {T1M_FLOAT32, T1M_COMPLEX64, T1M_FLOAT64, T1M_COMPLEX128})
    for (int64_t mn : {8, 100, 1000, 4096})
      for (int64_t K : {5, 16, 64, 200}) {
        const int64_t steps = (K + 15) / 16;
        const int at = small_form(dtype, mn, mn, K, steps).tile;
        for (int64_t forced : {steps + 1, 2 * steps, 4 * steps})
          if (small_form(dtype, mn, mn, K, forced).tile != at) {
            std::printf("dtype %d, %ld^2 over %ld: tile %d of %ld ranges, %d of %ld\n", dtype,
                        long(mn), long(K), at, long(steps),
                        small_form(dtype, mn, mn, K, forced).tile, long(forced));
            ++failures;
          }
      }
  // A large FP32 product keeps the large tile.
  if (small_form(T1M_FLOAT32, 4096, 4096, 64, 8).tile != 0) ++failures;
  // Float64 over at most 8 k: large outputs on the large tile, small ones not.
  if (small_form(T1M_FLOAT64, 4000, 4000, 8, 0).tile != 0) ++failures;
  if (small_form(T1M_FLOAT64, 1000, 1000, 1, 0).tile != 0) ++failures;
  if (small_form(T1M_FLOAT64, 200, 300, 8, 0).tile == 0) ++failures;
  if (small_form(T1M_FLOAT64, 4000, 4000, 9, 0).tile == 0) ++failures;
  if (small_form(T1M_COMPLEX128, 4000, 4000, 8, 0).tile == 0) ++failures;
  std::printf("%d failures\n", failures);
  return failures != 0;
}
