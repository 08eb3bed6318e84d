// Which wide stores the epilogues of the tensor-core kernels may use (host code).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "internal.h"

namespace t1m {
namespace gb300 {

// Epilogue store flags of a problem (kFlagCPairs, kFlagCCol16) from C's row
// and column offsets: the uniform strides where the arguments carry them (a
// uniform bundle, the dense split-K workspace), else the plan's vectors.
inline uint32_t c_store_flags(const GemmArgs& g, const std::vector<int64_t>& rsC,
                              const std::vector<int64_t>& csC) {
  auto col = [&](int64_t n) { return g.uC_n >= 0 ? n * g.uC_n : csC[n]; };
  auto row = [&](int64_t m) { return g.uC_m >= 0 ? m * g.uC_m : rsC[m]; };
  uint32_t f = 0;
  bool col16 = true;
  if (g.uC_n >= 0) {
    col16 = g.uC_n == 1 || g.N <= 1;
  } else {
    for (int64_t b = 0; b < g.N && col16; b += 16)
      for (int64_t i = b + 1; i < std::min<int64_t>(g.N, b + 16); ++i)
        if (col(i) != col(b) + (i - b)) {
          col16 = false;
          break;
        }
  }
  if (col16) f |= kFlagCCol16;
  // Every K range's partials start c_split_stride elements on (0 unsplit).
  bool pairs = reinterpret_cast<uintptr_t>(g.C) % 16 == 0 && g.c_split_stride % 2 == 0;
  if (pairs) {
    if (g.uC_m >= 0) {
      pairs = g.uC_m % 2 == 0 || g.M <= 1;
    } else {
      for (int64_t m = 0; m < g.M && pairs; ++m) pairs = row(m) % 2 == 0;
    }
  }
  if (pairs) {
    if (g.uC_n >= 0) {
      pairs = g.uC_n == 1;
    } else {
      for (int64_t n = 0; n + 1 < g.N && pairs; n += 2)
        pairs = col(n) % 2 == 0 && col(n + 1) == col(n) + 1;
    }
  }
  if (pairs) f |= kFlagCPairs;
  return f;
}

// Real epilogue flags: kFlagCCol16 as for complex; kFlagCPairs for four
// consecutive columns contiguous with 16-byte aligned starts.
inline uint32_t c_store_flags_real(const GemmArgs& g, const std::vector<int64_t>& rsC,
                                   const std::vector<int64_t>& csC) {
  auto col = [&](int64_t n) { return g.uC_n >= 0 ? n * g.uC_n : csC[n]; };
  auto row = [&](int64_t m) { return g.uC_m >= 0 ? m * g.uC_m : rsC[m]; };
  uint32_t f = 0;
  bool col16 = true;
  if (g.uC_n >= 0) {
    col16 = g.uC_n == 1 || g.N <= 1;
  } else {
    for (int64_t b = 0; b < g.N && col16; b += 16)
      for (int64_t i = b + 1; i < std::min<int64_t>(g.N, b + 16); ++i)
        if (col(i) != col(b) + (i - b)) {
          col16 = false;
          break;
        }
  }
  if (col16) f |= kFlagCCol16;
  bool quads = reinterpret_cast<uintptr_t>(g.C) % 16 == 0 && g.c_split_stride % 4 == 0;
  if (quads) {
    if (g.uC_m >= 0) {
      quads = g.uC_m % 4 == 0 || g.M <= 1;
    } else {
      for (int64_t m = 0; m < g.M && quads; ++m) quads = row(m) % 4 == 0;
    }
  }
  if (quads) {
    if (g.uC_n >= 0) {
      quads = g.uC_n == 1;
    } else {
      for (int64_t n = 0; n + 3 < g.N && quads; n += 4)
        quads = col(n) % 4 == 0 && col(n + 1) == col(n) + 1 && col(n + 2) == col(n) + 2 &&
                col(n + 3) == col(n) + 3;
    }
  }
  if (quads) f |= kFlagCPairs;
  return f;
}

}  // namespace gb300
}  // namespace t1m
