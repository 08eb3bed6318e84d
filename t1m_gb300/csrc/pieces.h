// Operand pieces (pieces.cu): descriptors of the split pass and of the
// CTA-pair product, shared with the dispatch (tc.cu) and the grouped launches.
#pragma once

#include <cstdint>

#include "internal.h"

namespace t1m {
namespace gb300 {

// Layout of an operand's pieces.  An operand of R real rows (A: the two 1M
// rows of every complex row, or the rows of a real A; B: its columns) and Kr
// real k (2 K complex, K real) is stored as atoms of 8 rows x 32 k bf16 (512
// bytes): piece p of stage ks (k in [32 ks, 32 ks + 32)) and row group rg is
// atom (ks * P + p) * rg_count + rg.  Inside an atom, row r holds 64 bytes;
// its 16-byte chunk c lies at chunk c ^ ((r >> 1) & 3).  That is the MMA's
// 64-byte-swizzled K-major shared-memory layout, so a tile's rows of one
// stage and piece are ONE contiguous copy of 512 bytes per row group: no
// tensor maps (a grouped launch needs one descriptor per product, not three)
// and every access is whole lines.
constexpr int kPieceStageK = 32;   // real k per stage
constexpr int kPieceAtom = 512;    // bytes
inline int64_t piece_groups(int64_t rows) { return (rows + 7) / 8; }
inline int64_t piece_stages(int64_t kreal) { return (kreal + kPieceStageK - 1) / kPieceStageK; }
inline size_t piece_bytes(int pieces, int64_t rows, int64_t kreal) {
  return size_t(pieces) * size_t(piece_groups(rows)) * size_t(piece_stages(kreal)) * kPieceAtom;
}

// Split pass of one operand: element (r, k) at src + ro(r) + ko(k).
enum : int32_t {
  kSplitRows = 0,  // consecutive threads along the rows (unit-stride runs of rows)
  kSplitK = 1,     // along k
  kSplitStep = 2   // along k_hi, where k = k_lo + step * k_hi and the source is
                   // contiguous in k_hi (step a multiple of a stage)
};
struct PieceSplit {
  const void* src;
  const int64_t *ro, *ko;  // offsets, or uniform strides ur / uk where >= 0
  int64_t ur, uk;
  int64_t R, K;            // source rows, elements of K
  int64_t step;
  uint8_t* out;
  int64_t rg;              // row groups of `out` (may exceed this operand's own)
  int64_t block_begin;     // first block of this operand in the launch
  int32_t expand;          // complex A: the two 1M rows of every row
  int32_t conj;
  int32_t mode;
  // Runs beside the split launched just before it, whose blocks let it start
  // once everything ahead of both has finished: it waits at its end instead.
  int32_t beside;
  int32_t kper;            // two-stage k blocks of a thread block (piece_split_blocks)
  int32_t pad;
};

// One product over pieces.  g: C, its offsets and epilogue, M, N, K,
// k_per_split and c_split_stride in elements.
struct PieceProblem {
  GemmArgs g;
  const uint8_t* a;
  const uint8_t* b;
  // Row groups of the arrays `a` and `b` point into (the distance from piece
  // to piece) and of the operands themselves: an operand may be a part of its
  // array, and nothing past its own groups is read (piece_operands).
  int64_t rg_a, rg_b, gn_a, gn_b;
  int64_t tile_begin;      // first tile of this problem in the launch
  int32_t tiles_m, tiles_n, splits;
  int32_t tile_n;          // output columns of a tile, a multiple of 32 up to 256
  // The operands (and M and N, C's offsets) are exchanged: the product
  // pairs run in the order of the unexchanged form, x0y1 before x1y0 of its x
  // and y, so every output sums the same values in the same order.
  int32_t swapped;
  int32_t pad;
};

// Sets the row groups of a product's operands (from g's M and N); arrays of
// `array_a` / `array_b` groups, 0: of the operand's own.
inline void piece_operands(bool real, PieceProblem* p, int64_t array_a, int64_t array_b) {
  p->gn_a = piece_groups((real ? 1 : 2) * p->g.M);
  p->gn_b = piece_groups(p->g.N);
  p->rg_a = array_a > 0 ? array_a : p->gn_a;
  p->rg_b = array_b > 0 ? array_b : p->gn_b;
}

// What CTA `rank` of a pair loads for the tile of row tile tm and first
// column n0, per stage and piece: 128 real rows of the first operand and half
// of the tile's columns, as many of their row groups as exist (the rest of a
// stage keeps old bytes: rows and columns nobody writes to C).
constexpr int kPieceCtaRows = 128;
struct PieceLoads {
  int64_t a, b;             // byte offsets in the arrays at k = kb, piece 0
  uint32_t abytes, bbytes;
};
__host__ __device__ inline PieceLoads piece_loads(int pieces, bool real, const PieceProblem& p,
                                                  int64_t tm, int64_t n0, uint32_t rank,
                                                  int64_t kb) {
  const int64_t ks = (real ? 1 : 2) * kb / kPieceStageK;
  const int64_t ga = (2 * tm + rank) * (kPieceCtaRows / 8), gb = (n0 + rank * (p.tile_n / 2)) / 8;
  const int64_t la = p.gn_a - ga, lb = p.gn_b - gb, ta = kPieceCtaRows / 8, tb = p.tile_n / 16;
  const int64_t na = la < ta ? la : ta, nb = lb < tb ? lb : tb;
  PieceLoads l;
  l.a = (ks * pieces * p.rg_a + ga) * kPieceAtom;
  l.b = (ks * pieces * p.rg_b + gb) * kPieceAtom;
  l.abytes = na > 0 ? static_cast<uint32_t>(na) * kPieceAtom : 0u;
  l.bbytes = nb > 0 ? static_cast<uint32_t>(nb) * kPieceAtom : 0u;
  return l;
}

// One product of a grouped launch (complex64, BF16x6): the product and the
// split passes of its operands, without their workspace (piece_item_place).
struct PieceItem {
  PieceProblem p;
  PieceSplit op[2];        // the product's first operand (1M rows), its second
  size_t bytes[2];         // their pieces
};
void tc_piece_item(const GemmArgs& g, const HostPlan& plan, int splits, PieceItem* it);
// Put the item's pieces at ws (bytes[0] + bytes[1] bytes).
void piece_item_place(PieceItem* it, void* ws);

// Whether a product of the automatic form runs over pieces.  `tma`: both
// operands are plain views that the one-tile kernels load by TMA; otherwise
// those gather them element by element, and pieces pay from 128 products per
// element on (2 M N / (M + N)): abcd,ebfd->aecf at 1024^3 77 -> 56 us, float32
// 1999 x 2503 x 1531 1012 -> 119; abcd,dbea->ec (96 x 64, K = 36864) 70
// without, 86 over pieces.  Complex products that load by TMA all do.
// float32 ones (one-tile / pieces, us a call queued among others over 260 MB of
// inputs): the pieces are three times the bytes of the operands, written and
// read, for a product that is a quarter of a complex one.
//   short K                     1000 x 1024 x 100 12.8 / 14.4, x 512 59 / 51;
//   few products per element    4000 x 4 x 4000 0.75 times as fast over pieces,
//                               1000 x 128 x 512 1.12, x 4000 0.86 times,
//                               1000 x 400 x 4000 1.10;
//   one wave of one-tile CTAs   4000 x 512 x 1024 0.92 times, 2000 x 768 x 1024
//   (76 to 152 tiles)           1.12, 2000 x 1024 x 256 0.86, x 4000 1.11;
//   more than one wave          4000 x 768 x 100 1.34, 2000 x 2000 x 2000 1.27.
// (After a flush of L2, code included, and alone, the pieces' extra launches
// cost up to 10 us more; calls of a program in a row do not see that.)
inline bool pieces_pay(bool real, bool tma, int64_t M, int64_t N, int64_t K) {
  if (!tma) return M * N >= 64 * (M + N);
  if (!real) return true;
  // One-tile CTAs, with the K ranges that the precision rule asks for.
  const int64_t tiles = ((M + 127) / 128) * ((N + 127) / 128) * ((K + 8191) / 8192);
  if (tiles > 152) return K >= 96;
  if (tiles >= 76) return K >= 1024 && M * N >= 500 * (M + N);
  return K >= 300 && (M * N >= 220 * (M + N) || (M * N >= 50 * (M + N) && K <= 1536));
}

// Thread blocks of the split pass of one operand; sets its kper.  `batch`: one
// of several operands in a launch.
int64_t piece_split_blocks(bool real, PieceSplit* s, bool batch = false);
// Split `n` operands in one launch (none of them kSplitStep when n > 1 or
// dev is given): `ops` by value (n <= 2) or the device array `dev`.
cudaError_t launch_piece_split(int pieces, bool real, const PieceSplit* ops, int n,
                               const PieceSplit* dev, int64_t blocks, cudaStream_t stream);
// Tile width of a product alone on the GPU, of one in a batch that fills it
// (up to 128 columns: their epilogue overlaps the next tile), and its tile
// counts (from g and splits).
int piece_tile_n_batch(int64_t N);
int piece_tile_n(bool real, int64_t M, int64_t N, int64_t K, int splits);
void piece_set_tiles(bool real, PieceProblem* p, int tile_n, int splits);
inline int64_t piece_tiles(const PieceProblem& p) {
  return int64_t(p.tiles_m) * p.tiles_n * p.splits;
}
// One launch over `total_tiles` tiles of `single`, or of the device array
// dev[0..nprob) (sorted by tile_begin); wide: every tile_n above 128 columns.
cudaError_t launch_piece_products(int pieces, bool real, bool wide, const PieceProblem* single,
                                  const PieceProblem* dev, int nprob, int64_t total_tiles,
                                  cudaStream_t stream, int* err_flag);

}  // namespace gb300
}  // namespace t1m
