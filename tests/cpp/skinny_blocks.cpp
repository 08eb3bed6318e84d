// Blocks of a grouped launch's skinny items: tall ones only where they still
// give every SM two blocks; K ranges shorter than usual only up to a block
// per SM.
#include <algorithm>
#include <cstdio>

#include "internal.h"

using namespace t1m::gb300;

int main() {
  constexpr int kSms = 152;
  int failures = 0, tall_cases = 0;
  for (int64_t M : {1, 32, 255, 256, 257, 300, 1000, 4096, 65536})
    for (int count : {1, 2, 4, 8, 16, 40, 64, 128})
      for (int splits : {1, 4}) {
        GemmArgs g{};
        g.M = M;
        g.N = 4;
        g.uA_k = 1;
        g.flags = kFlagSkinnyAsync;
        const int64_t low = skinny_tiles(g, splits, 4) * count;  // 32-row blocks
        if (skinny_may_tall(g) && skinny_tall(skinny_tall_blocks(g, splits) * count, kSms))
          g.flags |= kFlagSkinnyTall;
        const int64_t blocks = skinny_tiles(g, splits, 4) * count;
        const bool tall = g.flags & kFlagSkinnyTall;
        tall_cases += tall;
        const int64_t rows = skinny_async_rows(g.flags);
        const bool ok = blocks == count * splits * ((M + rows - 1) / rows) &&
                        blocks >= std::min<int64_t>(low, 2 * kSms) && (!tall || M >= 256);
        if (ok) continue;
        std::printf("%d items of %ld rows, %d ranges: %ld blocks of %ld rows, %ld of 32\n", count,
                    long(M), splits, long(blocks), long(rows), long(low));
        ++failures;
      }
  if (tall_cases == 0) ++failures;
  // K ranges of `count` equal items.
  int split_cases = 0;
  for (int nmax : {4, 16})
    for (int64_t unit : {1, 64})
      for (int64_t M : {1, 40, 64, 65, 256, 1000})
        for (int64_t K : {64, 500, 2048, 4096, 20000, 32768})
          for (int count : {1, 3, 8, 16, 64}) {
            GemmArgs g{};
            g.M = M;
            g.N = nmax;
            g.K = K;
            g.uA_k = unit;
            const int64_t rows = skinny_tiles(g, 1, nmax) * count;
            const int64_t cap = skinny_k_cap(false, g, double(rows) * double(K), kSms);
            const int64_t steps = (K + 15) / 16, ranges = (steps + cap / 16 - 1) / (cap / 16);
            const int64_t usual = (K + kGroupKCap - 1) / kGroupKCap;
            split_cases += ranges > usual;
            if (ranges >= usual && cap >= 128 && cap <= kGroupKCap &&
                rows * ranges <= std::max<int64_t>(kSms, rows * usual))
              continue;
            std::printf("%d items of %ld rows over %ld: %ld ranges, %ld blocks\n", count, long(M),
                        long(K), long(ranges), long(rows * ranges));
            ++failures;
          }
  if (split_cases == 0) ++failures;
  std::printf("%d failures, %d tall\n", failures, tall_cases);
  return failures != 0;
}
