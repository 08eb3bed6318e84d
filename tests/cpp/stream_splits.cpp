// The K ranges of streamed products cover K, and their partial products stay
// within the split-K workspace's cap and half of the operands' bytes.
#include <cstdio>

#include "stream.h"

using namespace t1m::gb300;

int main() {
  int failures = 0, streamed = 0;
  const int64_t sides[] = {1, 9, 17, 64, 96, 127, 128, 1000, 4000, 60000, 1000000, 10000000};
  const int64_t ks[] = {1024, 1531, 4096, 36864, 70000, 1000000, 4000000, 40000000};
  for (int64_t m : sides)
    for (int64_t n : sides)
      for (int64_t k : ks) {
        int64_t kps = 0;
        const int64_t s = stream_splits(m, n, k, &kps);
        if (s == 0) continue;
        ++streamed;
        const bool covers = kps > 0 && s * kps >= k && (s - 1) * kps < k;
        const bool room = s == 1 || size_t(s) * size_t(m) * size_t(n) * 8 <= kMaxWorkBytes;
        const bool small = s * m * n * 2 <= (m + n) * k;
        if (covers && room && small) continue;
        std::printf("%ld x %ld over %ld: %ld ranges of %ld, %.2f GB of partials\n", long(m),
                    long(n), long(k), long(s), long(kps), double(s) * m * n * 8 / 1e9);
        ++failures;
      }
  // The shapes the form is for still run on it.
  int64_t kps = 0;
  if (stream_splits(96, 64, 36864, &kps) == 0 || stream_splits(4095, 1, 1024, &kps) == 0) ++failures;
  std::printf("%d failures of %d streamed\n", failures, streamed);
  return failures != 0;
}
