// Products that run streamed by themselves (measured both ways, see stream_pays).
#include <cstdio>

#include "stream.h"

using namespace t1m::gb300;

int main() {
  int failures = 0;
  auto expect = [&](bool want, int fetch, int64_t m, int64_t n, int64_t k, int other) {
    int64_t kps = 0;
    const int s = stream_splits(m, n, k, &kps);
    const int64_t other_kps = (k / 16 + other) / other * 16;
    if (s > 0 && stream_pays(fetch, m, n, k, s, kps, other, other_kps) == want) return;
    std::printf("fetch %d, %ld x %ld over %ld (%d ranges): expected %d\n", fetch, long(m), long(n),
                long(k), s, int(want));
    ++failures;
  };
  for (int64_t k : {1024, 4096, 40000}) {
    expect(true, kStreamGathered, 500, 33, k, 19);
    expect(true, kStreamTma, 64, 64, k, 76);
    expect(true, kStreamTma, 96, 64, k, 76);
    expect(true, kStreamSectors, 64, 64, k, 75);
  }
  expect(true, kStreamTma, 64, 1000, 4096, 19);
  expect(true, kStreamTma, 96, 96, 40000, 38);
  expect(true, kStreamTma, 65, 1000, 40000, 10);
  expect(false, kStreamTma, 64, 1000, 40000, 19);
  expect(false, kStreamTma, 64, 256, 40000, 76);
  expect(false, kStreamTma, 64, 16000, 1024, 1);
  expect(false, kStreamTma, 8, 16000, 1024, 1);
  expect(true, kStreamTma, 16000, 33, 1024, 1);
  expect(true, kStreamSectors, 95, 63, 6061, 75);
  expect(true, kStreamSectors, 95, 63, 33511, 75);
  expect(true, kStreamSectors, 97, 65, 6061, 75);
  expect(true, kStreamSectors, 70, 70, 13824, 75);
  expect(false, kStreamSectors, 97, 65, 16983, 75);
  expect(false, kStreamSectors, 500, 33, 40425, 19);
  std::printf("%d failures\n", failures);
  return failures != 0;
}
