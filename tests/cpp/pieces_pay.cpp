// Products that run over operand pieces by themselves (measured both ways, see
// pieces_pay), and that the answer does not depend on which side is M.
#include <cstdio>

#include "pieces.h"

using namespace t1m::gb300;

int main() {
  int failures = 0;
  auto expect = [&](bool want, bool real, bool tma, int64_t m, int64_t n, int64_t k) {
    for (int swap = 0; swap < 2; ++swap)
      if (pieces_pay(real, tma, swap ? n : m, swap ? m : n, k) != want) {
        std::printf("%s %ld x %ld x %ld, TMA %d: expected %d\n", real ? "real" : "complex", long(m),
                    long(n), long(k), int(tma), int(want));
        ++failures;
      }
  };
  for (int64_t n : {1, 4, 16, 64}) {
    expect(false, true, true, 4000, n, 4000);
    expect(false, true, true, 300, n, 20000);
  }
  expect(false, true, true, 4000, 128, 4000);
  expect(false, true, true, 300, 256, 20000);
  expect(false, true, true, 1000, 1024, 100);
  expect(false, true, true, 4000, 512, 1024);
  expect(false, true, true, 2000, 1024, 512);
  expect(true, true, true, 1000, 128, 512);
  expect(true, true, true, 2000, 768, 2000);
  expect(true, true, true, 4000, 768, 100);
  expect(true, true, true, 2048, 2048, 2048);
  expect(true, true, true, 1000, 1024, 4000);
  expect(true, true, false, 1999, 2503, 1531);
  expect(false, true, false, 4000, 4, 4000);
  expect(true, false, true, 2304, 2304, 2304);
  expect(true, false, false, 1024, 1024, 1024);
  expect(false, false, false, 96, 64, 36864);
  std::printf("%d failures\n", failures);
  return failures != 0;
}
