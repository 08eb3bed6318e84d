// Blocks of a grouped launch's asynchronous skinny items: tall ones only where
// they still give every SM two blocks.
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
  std::printf("%d failures, %d tall\n", failures, tall_cases);
  return failures != 0;
}
