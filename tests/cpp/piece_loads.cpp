// Every bulk copy of the products over operand pieces stays inside the pieces
// array of its operand, and inside the operand where that is a part of the
// array: the halves of the host-buffer pipeline's resident operand and the
// slabs of its streamed one, ragged against the tiles.
#include <algorithm>
#include <cstdio>

#include "pieces.h"

using namespace t1m::gb300;

namespace {

int failures = 0;
long checked = 0;

// Rows [lo, hi) of an operand of `rows` (complex or real), pieces in one array.
struct Part {
  int64_t rows, lo, hi;
};

void check(int pieces, bool real, Part a, Part b, int64_t K, int tile_n) {
  const int64_t f = real ? 1 : 2;
  PieceProblem p{};
  p.g.M = a.hi - a.lo;
  p.g.N = b.hi - b.lo;
  p.g.K = K;
  p.tile_n = tile_n;
  const int64_t array_a = piece_groups(f * a.rows), array_b = piece_groups(b.rows);
  piece_operands(real, &p, array_a, array_b);
  const int64_t base_a = piece_groups(f * a.lo), base_b = piece_groups(b.lo);
  const int64_t end_a = piece_groups(f * a.hi), end_b = piece_groups(b.hi);
  const int64_t per = real ? 256 : 128;
  const int64_t stages = piece_stages(f * K);
  // Group range [first, first + bytes) of every stage and piece of an array.
  auto inside = [&](int64_t at, uint32_t bytes, int64_t array, int64_t base, int64_t end) {
    if (bytes == 0) return true;
    const int64_t first = base + at / kPieceAtom, last = first + bytes / kPieceAtom;
    const bool own = first >= base && last <= end;
    const int64_t limit = stages * pieces * array;
    return own && ((stages - 1) * pieces + pieces - 1) * array + last <= limit;
  };
  for (int64_t tm = 0; tm * per < p.g.M; ++tm)
    for (int64_t n0 = 0; n0 < p.g.N; n0 += tile_n)
      for (uint32_t rank = 0; rank < 2; ++rank) {
        const PieceLoads l = piece_loads(pieces, real, p, tm, n0, rank, 0);
        ++checked;
        // All rows and columns of the tile that exist are loaded.
        const int64_t row0 = (2 * tm + rank) * kPieceCtaRows, col0 = n0 + rank * (tile_n / 2);
        const int64_t rows = std::min<int64_t>(kPieceCtaRows, f * p.g.M - row0);
        const int64_t cols = std::min<int64_t>(tile_n / 2, p.g.N - col0);
        const bool full = int64_t(l.abytes) / 64 >= rows && int64_t(l.bbytes) / 64 >= cols;
        if (full && inside(l.a, l.abytes, array_a, base_a, end_a) &&
            inside(l.b, l.bbytes, array_b, base_b, end_b))
          continue;
        if (++failures <= 20)
          std::printf("%s P %d: A [%ld, %ld) of %ld, B [%ld, %ld) of %ld, tile (%ld, %ld) rank %u\n",
                      real ? "real" : "complex", pieces, long(a.lo), long(a.hi), long(a.rows),
                      long(b.lo), long(b.hi), long(b.rows), long(tm), long(n0), rank);
      }
}

}  // namespace

int main() {
  for (bool real : {false, true})
    for (int pieces : {2, 3})
      for (int tile_n : {32, 96, 128, 192, 256})
        for (int64_t M : {129, 257, 1040, 2080, 2305, 4160})
          for (int64_t N : {128, 200, 1999, 2176}) {
            const int64_t K = 640;
            check(pieces, real, {M, 0, M}, {N, 0, N}, K, tile_n);
            const int64_t half = (M / 2 + 127) / 128 * 128, slab = (N / 4 + 127) / 128 * 128;
            if (half >= M) continue;
            for (int h = 0; h < 2; ++h)
              for (int64_t lo = 0; lo < N; lo += slab)
                check(pieces, real, {M, h * half, h ? M : half}, {N, lo, std::min(N, lo + slab)},
                      K, tile_n);
          }
  std::printf("%d failures of %ld\n", failures, checked);
  return failures != 0;
}
