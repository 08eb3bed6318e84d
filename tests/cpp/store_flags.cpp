// Every 16-byte store that c_store_flags / c_store_flags_real allow is
// 16-byte aligned: in every K range's partials, every row, every whole group
// of columns, with the operands in either order.
#include <cstdio>
#include <utility>
#include <vector>

#include "store_flags.h"

using namespace t1m::gb300;

namespace {

int failures = 0;

// es: element bytes; wide: elements per 16-byte store.
void check(int64_t M, int64_t N, int splits, bool swapped, int64_t es, int64_t wide) {
  // Partials of a split product: dense, m fastest, one slice per K range.
  GemmArgs g{};
  g.C = reinterpret_cast<void*>(uintptr_t(1) << 20);
  g.M = M;
  g.N = N;
  g.uC_m = 1;
  g.uC_n = M;
  g.c_split_stride = splits > 1 ? M * N : 0;
  if (swapped) {
    std::swap(g.M, g.N);
    std::swap(g.uC_m, g.uC_n);
  }
  const std::vector<int64_t> none;
  const uint32_t f = es == 8 ? c_store_flags(g, none, none) : c_store_flags_real(g, none, none);
  if (!(f & kFlagCPairs)) return;
  for (int s = 0; s < splits; ++s)
    for (int64_t m = 0; m < g.M; ++m)
      for (int64_t n = 0; n + wide <= g.N; n += wide) {
        const int64_t at = s * g.c_split_stride + m * g.uC_m + n * g.uC_n;
        if ((reinterpret_cast<uintptr_t>(g.C) + at * es) % 16 == 0) continue;
        std::printf("misaligned: M %ld N %ld splits %d swapped %d element %ld bytes\n", long(M),
                    long(N), splits, int(swapped), long(es));
        ++failures;
        return;
      }
}

}  // namespace

int main() {
  const int64_t sides[] = {1, 2, 3, 4, 5, 7, 8, 16, 17, 18, 20, 33, 64, 101, 129, 4095, 4096};
  int pairs = 0;
  for (int64_t m : sides)
    for (int64_t n : sides)
      for (int splits : {1, 2, 3, 5})
        for (bool swapped : {false, true}) {
          check(m, n, splits, swapped, 8, 2);
          check(m, n, splits, swapped, 4, 4);
          ++pairs;
        }
  // The wide form is still taken where every range starts aligned.
  const std::vector<int64_t> none;
  GemmArgs g{};
  g.M = 1;
  g.N = 64;
  g.uC_m = 64;
  g.uC_n = 1;
  g.c_split_stride = 64;
  if (!(c_store_flags(g, none, none) & kFlagCPairs)) ++failures;
  if (!(c_store_flags_real(g, none, none) & kFlagCPairs)) ++failures;
  std::printf("%d failures of %d\n", failures, pairs);
  return failures != 0;
}
