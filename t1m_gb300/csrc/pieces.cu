// Operand pieces: products of complex64 / float32 operands split once into
// bf16 pieces, on CTA pairs whose MMAs read both operands from shared memory.
//
// split_pieces writes every operand element's P bf16 pieces (the split of
// tc_common.h, conjugation first) in the layout of pieces.h: for complex A the
// 1M rows [re, -im, ...] and [im, re, ...] of every row (t1m.h:309-325), for
// B the row [re, im, ...] of every column, real k = 2 k + part; for real
// operands the rows themselves.  It replaces the reference's per-block
// packing (t1m.h:309-337): once per operand instead of once per tile.
//
// tc1m_pieces then runs the real GEMM on clusters of two CTAs
// (tcgen05.mma.cta_group::2, M = 256 real rows per pair), persistent over the
// tiles of one product or of a batch.  Per accumulator the MMAs run in the
// order of tc.cu's pair form (the main product x0 y0 into a chunk
// accumulator, restarted every 16 MMAs and folded into FP32 registers with
// round-to-nearest adds; the corrections x0y1, x1y0 [, x1y1, x0y2, x2y0] into
// one accumulator for the whole K range), so both give the same bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "internal.h"
#include "pc_epilogue.h"
#include "pieces.h"
#include "ptx.h"
#include "t1m_capi.h"
#include "tc_common.h"

namespace t1m {
namespace gb300 {
namespace {

// ------------------------------------------------------------- split pass ---

struct SplitPair {
  PieceSplit op[2];
  int n;
};

// Pieces of 8 consecutive real k (v, already conjugated) into one 16-byte
// chunk per piece.  `at`: byte offset of the chunk in piece 0, pieces
// `stride` bytes apart.
template <int P>
__device__ __forceinline__ void put_chunk(uint8_t* out, int64_t at, int64_t stride,
                                          const float (&v)[8]) {
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) split_bf16<P>(v[2 * j], v[2 * j + 1], w[0][j], w[1][j], w[2][j]);
#pragma unroll
  for (int p = 0; p < P; ++p)
    *reinterpret_cast<uint4*>(out + at + p * stride) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// Byte offset of chunk c of real row rr in the piece-0 atom of stage ks.
template <int P>
__device__ __forceinline__ int64_t chunk_at(int64_t rg, int64_t ks, int64_t rr, int c) {
  const int rl = static_cast<int>(rr & 7);
  return (ks * P * rg + (rr >> 3)) * kPieceAtom + rl * 64 + ((c ^ ((rl >> 1) & 3)) << 4);
}

// Chunk c of source row r in stage ks from shared memory (`src`: its 4
// complex or 8 real values, consecutive k).
template <int P, bool kReal>
__device__ __forceinline__ void split_row_chunk(const PieceSplit& o, int64_t ks, int64_t r, int c,
                                                const float* src) {
  const int64_t stride = o.rg * kPieceAtom;
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = src[j];
  if constexpr (kReal) {
    put_chunk<P>(o.out, chunk_at<P>(o.rg, ks, r, c), stride, v);
  } else {
    if (o.conj) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[2 * j + 1] = -v[2 * j + 1];
    }
    if (!o.expand) {
      put_chunk<P>(o.out, chunk_at<P>(o.rg, ks, r, c), stride, v);
    } else {
      // The second 1M row's pairs [im, re] are the first's [re, -im] with the
      // halves exchanged and -im negated: the split is symmetric in the sign.
      uint32_t w[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        split_bf16<P>(v[2 * j], -v[2 * j + 1], w[0][j], w[1][j], w[2][j]);
      uint8_t* const at = o.out + chunk_at<P>(o.rg, ks, 2 * r, c);
      uint8_t* const at1 = o.out + chunk_at<P>(o.rg, ks, 2 * r + 1, c);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        *reinterpret_cast<uint4*>(at + p * stride) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) w[p][j] = __byte_perm(w[p][j], 0u, 0x1032) ^ 0x8000u;
        *reinterpret_cast<uint4*>(at1 + p * stride) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
      }
    }
  }
}

constexpr int kSplitRowsPer = 32;                                // source rows per block
template <bool kReal>
constexpr int split_k() { return kReal ? 64 : 32; }              // k per block: two stages

// Start of a split pass.  The kernels ahead have finished once a block is past
// its wait: then the next kernel may start (a second split reads and writes
// other memory than the first).  One that runs beside the split before it was
// launched by blocks of that split past their wait, so everything ahead of
// both has ended and written its results back; it takes them up by a fence of
// its own (its SM may hold older lines of its source), and waits at its end.
__device__ __forceinline__ void begin_split(bool beside) {
  if (beside)
    __threadfence();
  else
    begin_dependent();
  release_dependents();
}

// Blocks of 32 rows x kper times two stages: read into shared memory along
// the source's unit-stride direction, written as whole atoms (a warp writes
// the four chunks of eight rows).  k past K is written as zeros, rows past R
// are not written.  The next two stages are copied asynchronously while the
// current ones are split: with two stages a block, its own start (finding the
// operand, offsets) took longer than their data.  (Held in registers instead,
// they left room for two to six blocks per SM of eight and the pass slowed
// down by a third.)
// kMany false: one k block (kper 1), eight blocks per SM, for operands that
// leave no more than that to do.
template <int P, bool kReal, bool kMany>
__global__ void __launch_bounds__(256, kMany ? 6 : 8)
split_pieces(const SplitPair pair, const PieceSplit* dev, int n) {
  using T = typename std::conditional<kReal, float, float2>::type;
  constexpr int KB = split_k<kReal>();
  __shared__ T tile[kMany ? 2 : 1][kSplitRowsPer][KB + 1];
  __shared__ PieceSplit so;
  const bool beside = !dev && pair.op[0].beside;
  begin_split(beside);
  if (kMany && dev) {
    const int lo = block_find(n, blockIdx.x, [&](int i) { return dev[i].block_begin; });
    block_copy(&so, dev + lo);
    __syncthreads();
  }
  const PieceSplit& o =
      kMany && dev ? so : (pair.n > 1 && blockIdx.x >= pair.op[1].block_begin ? pair.op[1] : pair.op[0]);
  // Block counts of a launch fit 32 bits (launch_piece_split).
  const int bid = static_cast<int>(blockIdx.x - o.block_begin);
  const int kspan = kMany ? KB * o.kper : KB;
  const int kblocks = static_cast<int>((o.K + kspan - 1) / kspan);
  const int rb = bid / kblocks;
  const int64_t r0 = int64_t(rb) * kSplitRowsPer, kbeg = int64_t(bid - rb * kblocks) * kspan;
  const int64_t kend = min(o.K, kbeg + kspan);
  const T* __restrict__ src = static_cast<const T*>(o.src);
  const int t = threadIdx.x;
  constexpr int kPer = kSplitRowsPer * KB / 256;
  // 32 rows x 8 chunks: thread t takes chunk t & 3 of row (t >> 2) & 31 in
  // stage t >> 7 of the tile's two.
  const int c = t & 3, r = (t >> 2) & 31, st = t >> 7;
  constexpr int kStageE = kReal ? 32 : 16;  // elements per stage
  constexpr int kChunkE = kReal ? 8 : 4;
  auto put = [&](int64_t k0, int b) {
    const int64_t ks = k0 / kStageE + st;
    if (r0 + r >= o.R || ks * kStageE >= o.K) return;
    float v[8];
#pragma unroll
    for (int j = 0; j < kChunkE; ++j) {
      const T x = tile[b][r][st * kStageE + c * kChunkE + j];
      if constexpr (kReal) {
        v[j] = x;
      } else {
        v[2 * j] = x.x;
        v[2 * j + 1] = x.y;
      }
    }
    split_row_chunk<P, kReal>(o, ks, r0 + r, c, v);
  };
  if constexpr (kMany) {
    const bool by_rows = o.mode == kSplitRows;
    auto fetch = [&](int64_t k0, int b) {
      if (by_rows) {
        const int r = t & 31;
        const bool rin = r0 + r < o.R;
        const T* __restrict__ row = src + (rin ? offs(o.ro, o.ur, r0 + r) : 0);
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
          const int k = (t >> 5) + 8 * i;
          const bool in = rin && k0 + k < o.K;
          cp_async_elem<sizeof(T)>(&tile[b][r][k], in ? row + offs(o.ko, o.uk, k0 + k) : src, in);
        }
      } else {
        const int k = t & (KB - 1);
        const bool kin = k0 + k < o.K;
        const T* __restrict__ col = src + (kin ? offs(o.ko, o.uk, k0 + k) : 0);
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
          const int r = t / KB + (256 / KB) * i;
          const bool in = kin && r0 + r < o.R;
          cp_async_elem<sizeof(T)>(&tile[b][r][k], in ? col + offs(o.ro, o.ur, r0 + r) : src, in);
        }
      }
      cp_async_commit_group();
    };
    fetch(kbeg, 0);
    int b = 0;
    for (int64_t k0 = kbeg; k0 < kend; k0 += KB, b ^= 1) {
      if (k0 + KB < kend) {
        fetch(k0 + KB, b ^ 1);
        cp_async_wait_group<1>();
      } else {
        cp_async_wait_group<0>();
      }
      __syncthreads();
      put(k0, b);
      __syncthreads();  // this buffer is fetched into next
    }
  } else {
    if (o.mode == kSplitRows) {
      const int r = t & 31;
      const bool rin = r0 + r < o.R;
      const T* __restrict__ row = src + (rin ? offs(o.ro, o.ur, r0 + r) : 0);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int k = (t >> 5) + 8 * i;
        T v{};
        if (rin && kbeg + k < o.K) v = row[offs(o.ko, o.uk, kbeg + k)];
        tile[0][r][k] = v;
      }
    } else {
      const int k = t & (KB - 1);
      const bool kin = kbeg + k < o.K;
      const T* __restrict__ col = src + (kin ? offs(o.ko, o.uk, kbeg + k) : 0);
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int r = t / KB + (256 / KB) * i;
        T v{};
        if (kin && r0 + r < o.R) v = col[offs(o.ro, o.ur, r0 + r)];
        tile[0][r][k] = v;
      }
    }
    __syncthreads();
    put(kbeg, 0);
  }
  // This kernel's end stands for the other split's too.
  if (beside) begin_dependent();
}

// kSplitStep: the source is contiguous along k_hi (k = k_lo + step * k_hi).
// Blocks of 8 rows x one stage of k_lo x 32 k_hi: reads are runs of 32
// elements, writes whole atoms (one stage of every k_hi).
template <int P, bool kReal>
__global__ void __launch_bounds__(256)
split_pieces_step(const PieceSplit o) {
  using T = typename std::conditional<kReal, float, float2>::type;
  constexpr int KL = kReal ? 32 : 16, KH = 32, R = 8;
  // Rows padded by one element and k_hi planes by one more: neither the
  // stores along k_hi nor the chunk reads conflict.
  constexpr int kRow = KL + 1, kPlane = R * kRow + 1;
  __shared__ T tile[KH * kPlane];
  begin_split(o.beside);
  const int64_t nhi = o.K / o.step, nlo = o.step / KL;
  const int64_t hblocks = (nhi + KH - 1) / KH;
  int64_t b = blockIdx.x;
  const int64_t h0 = (b % hblocks) * KH;
  b /= hblocks;
  const int64_t l0 = (b % nlo) * KL, r0 = (b / nlo) * R;
  const T* __restrict__ src = static_cast<const T*>(o.src);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // Offsets are linear in the mode indices and `step` spans whole modes.
  const bool hin = h0 + lane < nhi;
  const int64_t oh = hin ? offs(o.ko, o.uk, o.step * (h0 + lane)) : 0;
  const bool rin = r0 + warp < o.R;
  const T* __restrict__ row = src + (rin ? offs(o.ro, o.ur, r0 + warp) : 0) + oh;
#pragma unroll 8
  for (int l = 0; l < KL; ++l) {
    T v{};
    if (hin && rin) v = row[offs(o.ko, o.uk, l0 + l)];
    tile[lane * kPlane + warp * kRow + l] = v;
  }
  __syncthreads();
  const int c = lane & 3, r = lane >> 2;
  constexpr int kChunkE = kReal ? 8 : 4;
#pragma unroll
  for (int i = 0; i < KH / 8; ++i) {
    const int h = warp + 8 * i;
    if (h0 + h >= nhi || r0 + r >= o.R) break;
    const T* s = tile + h * kPlane + r * kRow + c * kChunkE;
    float v[8];
#pragma unroll
    for (int j = 0; j < kChunkE; ++j) {
      if constexpr (kReal) {
        v[j] = s[j];
      } else {
        v[2 * j] = s[j].x;
        v[2 * j + 1] = s[j].y;
      }
    }
    split_row_chunk<P, kReal>(o, (l0 + o.step * (h0 + h)) / KL, r0 + r, c, v);
  }
  if (o.beside) begin_dependent();
}

// ---------------------------------------------------------------- product ---

constexpr int kPcThreads = 640;        // warp 0 MMA, 1 loads, 2 relay, 3 tiles, 4-19 epilogue
constexpr int kPcEpiBase = 128;
constexpr int kPcEpiWarps = 16;
constexpr uint32_t kPcTmemCols = 512;
constexpr int kPcBarriers = 512;
constexpr int kPcARows = kPieceCtaRows;  // real rows of A per CTA
constexpr int kPcABytes = kPcARows * 64;
constexpr int kPcFold = 8;             // stages per main chunk: 16 MMAs of K = 16

// One tile as the roles of a CTA see it, written to shared memory by the
// scheduling warp up to kPcWorks tiles ahead: finding a tile's problem and
// its fields takes about 1000 clocks of dependent loads and divisions, which
// each role used to pay per tile (K = 128: 12.9k clocks a tile for 6.9k of
// MMAs).
constexpr int kPcWorks = 4;

// kWide: tiles of 160 to 256 columns, one chunk and one correction
// accumulator of 256 columns; otherwise up to 128 columns and two of each.
// Ring stages: as many as 227 KB hold.
template <int P, bool kWide>
struct PcShape {
  static constexpr int kMaxN = kWide ? 256 : 128;
  static constexpr int kBufs = kWide ? 1 : 2;
  static constexpr int kBBytes = kMaxN / 2 * 64;            // one piece of this CTA's columns
  static constexpr int kStage = P * (kPcABytes + kBBytes);  // 48 / 36 KB for three pieces
  static constexpr int kStages = kWide ? (P == 3 ? 4 : 6) : (P == 3 ? 6 : 8);
  static constexpr int kUnits = kMaxN / 16 / (kPcEpiWarps / 4);  // 16-column units per thread
  static constexpr int kCols = 16 * kUnits;                      // columns per warpgroup
  static constexpr int kSmem = 1024 + kStages * kStage + kPcBarriers +
                               kPcWorks * static_cast<int>(sizeof(PcWork)) +
                               kPcEpiWarps * kCols * 8;
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
  static_assert(8 * (2 * kStages + 4 * kBufs + 2 * kPcWorks + 2) <= kPcBarriers, "barrier area");
  __device__ static constexpr uint32_t chunk_col(int b) { return 128u * b; }
  __device__ static constexpr uint32_t corr_col(int b) { return 256u + 128u * b; }
};

// Tile t of the launch for CTA `rank` of its pair.  Tiles of a problem are
// numbered split-major; within a split, groups of 8 pair tiles along M sweep
// N, so pairs running together share both operands in L2.
template <int P, bool kReal>
__device__ __forceinline__ void pc_fill(PcWork& w, const PieceProblem* single,
                                        const PieceProblem* group, int nprob, int64_t t,
                                        uint32_t rank, int& hint) {
  const PieceProblem* p = single;
  if (group) {
    int lo = hint;
    while (lo + 1 < nprob && group[lo + 1].tile_begin <= t) ++lo;
    hint = lo;
    p = group + lo;
  }
  const GemmArgs& g = p->g;
  // Tile counts of a launch fit 32 bits (launch_piece_products).
  const int lt = static_cast<int>(t - p->tile_begin);
  const int tiles_m = p->tiles_m, tiles_n = p->tiles_n, tn = p->tile_n;
  const int per_split = tiles_m * tiles_n;
  const int split = p->splits > 1 ? lt / per_split : 0, r = lt - split * per_split;
  constexpr int G = 8;
  const int grp = r / (G * tiles_n), in = r - grp * (G * tiles_n);
  const int first_m = grp * G;
  const int gsize = min(G, tiles_m - first_m);
  const int col = in / gsize;
  const int64_t tm = first_m + in - col * gsize;
  const int64_t n0 = int64_t(col) * tn;
  constexpr int64_t f = kReal ? 1 : 2;
  const int64_t kb = int64_t(split) * g.k_per_split;
  const int64_t ke = min(g.K, kb + g.k_per_split);
  const PieceLoads l = piece_loads(P, kReal, *p, tm, n0, rank, kb);
  w.a = p->a + l.a;
  w.b = p->b + l.b;
  w.pa = p->rg_a * kPieceAtom;
  w.pb = p->rg_b * kPieceAtom;
  w.abytes = l.abytes;
  w.bbytes = l.bbytes;
  w.C = static_cast<uint8_t*>(g.C) + split * g.c_split_stride * (kReal ? 4 : 8);
  w.rsC = g.rsC;
  w.csC = g.csC;
  w.uC_m = g.uC_m;
  w.uC_n = g.uC_n;
  w.row0 = (2 * tm + rank) * (kReal ? kPcARows : kPcARows / 2);
  w.M = g.M;
  w.n0 = n0;
  w.N = g.N;
  w.alpha[0] = static_cast<float>(g.alpha[0]);
  w.alpha[1] = static_cast<float>(g.alpha[1]);
  w.beta[0] = static_cast<float>(g.beta[0]);
  w.beta[1] = static_cast<float>(g.beta[1]);
  w.flags = g.flags;
  w.steps = static_cast<int>((f * (ke - kb) + 15) / 16);
  w.tn = tn;
  w.swapped = p->swapped;
}

// Persistent over the launch's tiles, one cluster of two CTAs per pair of
// SMs.  Warp 0 (even CTA, one lane) issues every MMA; warp 1 (one lane per
// CTA) loads the CTA's 128 rows of A and half of the tile's columns of B;
// warp 2 (odd CTA, one lane) relays the arrival of its stage to the MMA
// thread; warp 3 (one lane per CTA) finds the tiles; warps 4-19 fold chunks
// and write C (one TMEM lane per thread, the four warpgroups each a quarter of
// the columns).
//
// Overlap.  Loads run ahead over tile borders.  With tiles of up to 128
// columns both chunk and correction accumulators are doubled, so a tile's
// MMAs start while the previous tile is still being read and written.  Wide
// tiles fill TMEM with one set: a chunk is folded while the corrections of
// its last two stages run (their main products are issued first), and the
// next tile starts as soon as the accumulators are in registers, before C is
// written.
//
// Tile widths from 32 to 256 columns let the tiles of a product fill whole
// waves of the 76 pairs (piece_tile_n).  Measured at complex64 4096^3,
// BF16x6: 1.86 ms (one 128-column tile per pair, 64-k stages, MMAs issued
// from a lane-0 branch) -> 1.52 ms, 361 TFLOP/s of 8MNK.
template <int P, bool kReal, bool kWide>
__global__ void __launch_bounds__(kPcThreads, 1)
tc1m_pieces(const __grid_constant__ PieceProblem single, const PieceProblem* group, int nprob,
            int64_t total_tiles, int* err_flag) {
  using Sh = PcShape<P, kWide>;
  constexpr int S = Sh::kStages, kBufs = Sh::kBufs;
  constexpr int kUnits = Sh::kUnits, kCols = Sh::kCols;

  extern __shared__ __align__(16) uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const base_ptr = smem_raw + (base - ptx::smem_u32(smem_raw));
  const uint32_t bars = base + S * Sh::kStage;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (S + s); };
  auto chunk_full = [&](int b) { return bars + 8u * (2 * S + b); };
  auto chunk_empty = [&](int b) { return bars + 8u * (2 * S + kBufs + b); };
  auto corr_full = [&](int b) { return bars + 8u * (2 * S + 2 * kBufs + b); };
  auto corr_empty = [&](int b) { return bars + 8u * (2 * S + 3 * kBufs + b); };
  auto work_full = [&](int e) { return bars + 8u * (2 * S + 4 * kBufs + e); };
  auto work_empty = [&](int e) { return bars + 8u * (2 * S + 4 * kBufs + kPcWorks + e); };
  const uint32_t end_bar = bars + 8u * (2 * S + 4 * kBufs + 2 * kPcWorks);
  const uint32_t tmem_slot = end_bar + 8u;
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(base_ptr + (tmem_slot - base));
  PcWork* const works = reinterpret_cast<PcWork*>(base_ptr + S * Sh::kStage + kPcBarriers);
  int64_t* const col_offsets = reinterpret_cast<int64_t*>(works + kPcWorks);

  const int tid = threadIdx.x;
  // Broadcast from lane 0, so the compiler knows the roles are warp-uniform.
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t rank = __shfl_sync(0xffffffffu, ptx::cluster_ctarank(), 0);
  if (warp == 0) {
    ptx::tmem_alloc2(tmem_slot, kPcTmemCols);
    ptx::tmem_relinquish2();
  }
  if (tid == 32) {
    // A stage is full on the even CTA once its own copies and, through the
    // odd CTA's relay, the peer's have landed.
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar(s), rank == 0 ? 2 : 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < kBufs; ++b) {
      ptx::mbar_init(chunk_full(b), 1);
      ptx::mbar_init(chunk_empty(b), 2 * kPcEpiWarps);
      ptx::mbar_init(corr_full(b), 1);
      ptx::mbar_init(corr_empty(b), 2 * kPcEpiWarps);
    }
    // Readers of a tile: loads, epilogue warps, and the MMA warp (even CTA) or
    // the relay (odd CTA).
    for (int e = 0; e < kPcWorks; ++e) {
      ptx::mbar_init(work_full(e), 1);
      ptx::mbar_init(work_empty(e), 2 + kPcEpiWarps);
    }
    ptx::mbar_init(end_bar, 1);
    ptx::fence_mbar_init();
  }
  ptx::tc_fence_before();
  ptx::cluster_sync();
  ptx::tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot_ptr, 0);

  // Everything above may overlap the end of the split pass; the descriptors,
  // pieces and C below may have been written by earlier kernels.
  begin_dependent();
  // The next tile of this role: its entry, or null when there are no more
  // (or a wait ran out, which is recorded).
  struct Cursor {
    int e = 0;
    uint32_t phase = 0;
  };
  auto take = [&](const Cursor& c) -> const PcWork* {
    if (!ptx::mbar_wait(work_full(c.e), c.phase)) {
      record_error(err_flag, kErrWorkWait);
      return nullptr;
    }
    const PcWork* w = works + c.e;
    return w->steps > 0 ? w : nullptr;
  };
  // Hand the entry back (one arrival per role) and go on to the next.
  auto advance = [&](Cursor& c) {
    if (++c.e == kPcWorks) {
      c.e = 0;
      c.phase ^= 1u;
    }
  };
  if (warp == 3) {
    // --------------------------------------------------------- scheduling ---
    if (lane == 0) {
      const int64_t first = blockIdx.x >> 1, stride = gridDim.x >> 1;
      int hint = 0;
      Cursor c;
      for (int64_t t = first;; t += stride) {
        if (!ptx::mbar_wait(work_empty(c.e), c.phase ^ 1u)) {
          record_error(err_flag, kErrWorkWait);
          break;
        }
        PcWork& w = works[c.e];
        if (t < total_tiles)
          pc_fill<P, kReal>(w, &single, group, nprob, t, rank, hint);
        else
          w.steps = 0;
        ptx::mbar_arrive(work_full(c.e));
        advance(c);
        if (t >= total_tiles) break;
      }
    }
    __syncwarp();
  } else if (warp == 0) {
    // ---------------------------------------------------------- MMA issue ---
    // The whole warp runs this loop and one elected lane issues: with
    // warp-uniform control flow the descriptors stay in uniform registers.
    // Issued from a lane-0 branch an MMA cost its thread 75 clocks and a stage
    // 850 more, whatever the tile width (128-column tiles ran at half the
    // tensor rate).
    if (rank == 0) {
      const uint64_t desc0 = ptx::smem_desc_sw64(base);
      const bool issue = ptx::elect_one();
      int slot = 0, tile_cnt = 0, chunk = 0;
      uint32_t phase = 0;
      bool ok = true;
      // Products of one ring slot.  Piece p, K = 16 step kk: A at +p x 8 KB,
      // B after the A pieces, +32 bytes per step inside the 64-byte rows.
      auto mains = [&](int st, int nkk, uint32_t d, uint32_t idesc, bool first_of_chunk) {
        const uint64_t ds = desc0 + static_cast<uint32_t>((st * Sh::kStage) >> 4);
        if (issue) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk)
            if (kk < nkk)
              ptx::mma_f16_ss2(d, ds + ((32 * kk) >> 4), ds + ((P * kPcABytes + 32 * kk) >> 4),
                               idesc, (first_of_chunk && kk == 0) ? 0u : 1u);
        }
      };
      auto corrections = [&](int st, int nkk, uint32_t d, uint32_t idesc, bool first_of_tile,
                             bool swapped) {
        const uint64_t ds = desc0 + static_cast<uint32_t>((st * Sh::kStage) >> 4);
        // Product of pieces px of the x operand and py of y: x is A, or B
        // where the operands are exchanged.
        auto mma = [&](int px, int py, int kk, uint32_t acc) {
          const int pa = swapped ? py : px, pb = swapped ? px : py;
          ptx::mma_f16_ss2(d, ds + ((pa * kPcABytes + 32 * kk) >> 4),
                           ds + ((P * kPcABytes + pb * Sh::kBBytes + 32 * kk) >> 4), idesc, acc);
        };
        if (issue) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            if (kk < nkk) {
              mma(0, 1, kk, (first_of_tile && kk == 0) ? 0u : 1u);
              mma(1, 0, kk, 1u);
              if (P == 3) {
                mma(1, 1, kk, 1u);
                mma(0, 2, kk, 1u);
                mma(2, 0, kk, 1u);
              }
            }
          }
          ptx::mma_commit2(empty_bar(st));
        }
      };
      Cursor cur;
      while (ok) {
        const PcWork* w = take(cur);
        if (!w) break;
        const int steps = __shfl_sync(0xffffffffu, w->steps, 0);
        const int tn = __shfl_sync(0xffffffffu, w->tn, 0);
        const bool swapped = __shfl_sync(0xffffffffu, w->swapped, 0) != 0;
        if (issue) ptx::mbar_arrive(work_empty(cur.e));
        advance(cur);
        const uint32_t idesc = ptx::idesc_f32acc(1u /*BF16*/, 256u, static_cast<uint32_t>(tn));
        const int ns = (steps + 1) / 2;
        const int cb = tile_cnt % kBufs;
        const uint32_t d_corr = tmem + Sh::corr_col(cb);
        uint32_t d_main = 0;
        int buf = 0;
        for (int s = 0; s < ns;) {
          if (s % kPcFold == 0) {
            buf = chunk % kBufs;
            d_main = tmem + Sh::chunk_col(buf);
            if (chunk >= kBufs &&
                !ptx::mbar_wait(chunk_empty(buf), static_cast<uint32_t>((chunk / kBufs - 1) & 1))) {
              record_error(err_flag, kErrChunkWait);
              ok = false;
              break;
            }
          }
          // The last two stages of a chunk issue their main products
          // together, so its fold overlaps two stages of corrections.
          const bool two = s % kPcFold == kPcFold - 2 && s + 1 < ns;
          const int slot2 = slot + 1 == S ? 0 : slot + 1;
          const uint32_t phase2 = slot + 1 == S ? phase ^ 1u : phase;
          if (!ptx::mbar_wait(full_bar(slot), phase) ||
              (two && !ptx::mbar_wait(full_bar(slot2), phase2))) {
            record_error(err_flag, kErrFullWait);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const int nkk = steps - 2 * s >= 2 ? 2 : 1, nkk2 = steps - 2 * s >= 4 ? 2 : 1;
          mains(slot, nkk, d_main, idesc, s % kPcFold == 0);
          if (two) mains(slot2, nkk2, d_main, idesc, false);
          const int last = s + (two ? 1 : 0);
          if (last % kPcFold == kPcFold - 1 || last == ns - 1) {
            if (issue) ptx::mma_commit2(chunk_full(buf));
            ++chunk;
          }
          if (s == 0 && tile_cnt >= kBufs) {
            if (!ptx::mbar_wait(corr_empty(cb), static_cast<uint32_t>((tile_cnt / kBufs - 1) & 1))) {
              record_error(err_flag, kErrAccEmptyWait);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
          }
          corrections(slot, nkk, d_corr, idesc, s == 0, swapped);
          if (two) corrections(slot2, nkk2, d_corr, idesc, false, swapped);
          slot = two ? slot2 : slot;
          phase = two ? phase2 : phase;
          s += two ? 2 : 1;
          if (++slot == S) {
            slot = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (issue) ptx::mma_commit2(corr_full(cb));
        ++tile_cnt;
      }
      // No MMA may still write TMEM (or read shared memory) when the CTAs leave.
      if (issue) ptx::mma_commit2(end_bar);
      if (!ptx::mbar_wait(end_bar, 0)) record_error(err_flag, kErrAccWait);
    }
    __syncwarp();
  } else if (warp == 1) {
    // -------------------------------------------------------------- loads ---
    if (lane == 0) {
      int slot = 0;
      uint32_t phase = 0;
      Cursor cur;
      bool ok = true;
      while (ok) {
        const PcWork* w = take(cur);
        if (!w) break;
        const uint8_t *a = w->a, *b = w->b;
        const int64_t pa = w->pa, pb = w->pb;
        const uint32_t abytes = w->abytes, bbytes = w->bbytes;
        const int ns = (w->steps + 1) / 2;
        ptx::mbar_arrive(work_empty(cur.e));
        advance(cur);
        for (int s = 0; s < ns; ++s) {
          if (!ptx::mbar_wait(empty_bar(slot), phase ^ 1u)) {
            record_error(err_flag, kErrRawWait);
            ok = false;
            break;
          }
          const uint32_t dst = base + slot * Sh::kStage;
          ptx::mbar_arrive_expect_tx(full_bar(slot), P * (abytes + bbytes));
#pragma unroll
          for (int q = 0; q < P; ++q) {
            if (abytes) ptx::bulk_load(dst + q * kPcABytes, a, abytes, full_bar(slot));
            if (bbytes)
              ptx::bulk_load(dst + P * kPcABytes + q * Sh::kBBytes, b, bbytes, full_bar(slot));
            a += pa;
            b += pb;
          }
          if (++slot == S) {
            slot = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // -------------------------------------------------------------- relay ---
    if (lane == 0 && rank == 1) {
      int slot = 0;
      uint32_t phase = 0;
      Cursor cur;
      bool ok = true;
      while (ok) {
        const PcWork* w = take(cur);
        if (!w) break;
        const int ns = (w->steps + 1) / 2;
        ptx::mbar_arrive(work_empty(cur.e));
        advance(cur);
        for (int s = 0; s < ns; ++s) {
          if (!ptx::mbar_wait(full_bar(slot), phase)) {
            record_error(err_flag, kErrFullWait);
            ok = false;
            break;
          }
          ptx::mbar_arrive_cluster(ptx::mapa(full_bar(slot), 0));
          if (++slot == S) {
            slot = 0;
            phase ^= 1u;
          }
        }
      }
    }
    __syncwarp();
  } else if (tid >= kPcEpiBase) {
    // ------------------------------------------------- fold and epilogue ---
    const int pt = tid - kPcEpiBase;
    const int wg = pt >> 7;
    const int q = (pt >> 5) & 3;
    const int rho = 32 * q + lane;  // real row of this CTA's 128 = TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(32 * q) << 16;
    int64_t* const cols = col_offsets + (warp - 4) * kCols;
    int chunk = 0, tile_cnt = 0;
    Cursor cur;
    while (true) {
      const PcWork* w = take(cur);
      if (!w) break;
      const int tn = w->tn;
      // C's offsets of this lane's row and of the warpgroup's columns, while
      // the tile's products run.
      const int64_t row = w->row0 + (kReal ? rho : rho >> 1);
      const bool row_ok = row < w->M;
      const int64_t row_off = row_ok ? offs(w->rsC, w->uC_m, row) : 0;
#pragma unroll
      for (int j = 0; j < kCols / 32; ++j) {
        const int64_t n = w->n0 + kCols * wg + 32 * j + lane;
        cols[32 * j + lane] = n < w->N ? offs(w->csC, w->uC_n, n) : 0;
      }
      __syncwarp();
      float master[kUnits][16];
#pragma unroll
      for (int u = 0; u < kUnits; ++u)
#pragma unroll
        for (int j = 0; j < 16; ++j) master[u][j] = 0.f;
      // Unit u holds columns [unit_col(u), + 16) of the tile: each warpgroup
      // takes kCols adjacent columns.
      auto unit_col = [&](int u) { return kCols * wg + 16 * u; };
      auto fold = [&](uint32_t col) {
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          if (unit_col(u) < tn) {
            uint32_t r[16];
            ptx::tmem_ld16_sync(tmem + lane_base + col + unit_col(u), r);
#pragma unroll
            for (int j = 0; j < 16; ++j) master[u][j] += __uint_as_float(r[j]);
          }
        }
      };
      auto release = [&](uint32_t bar) {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa(bar, 0));
      };
      const int nchunks = (w->steps + 2 * kPcFold - 1) / (2 * kPcFold);
      bool ok = true;
      for (int c = 0; c < nchunks; ++c, ++chunk) {
        const int buf = static_cast<int>(chunk % kBufs);
        if (!ptx::mbar_wait(chunk_full(buf), static_cast<uint32_t>((chunk / kBufs) & 1))) {
          record_error(err_flag, kErrChunkWait);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        fold(Sh::chunk_col(buf));
        release(chunk_empty(buf));
      }
      if (!ok) break;
      const int cb = static_cast<int>(tile_cnt % kBufs);
      if (!ptx::mbar_wait(corr_full(cb), static_cast<uint32_t>((tile_cnt / kBufs) & 1))) {
        record_error(err_flag, kErrAccWait);
        break;
      }
      ptx::tc_fence_after();
      fold(Sh::corr_col(cb));
      release(corr_empty(cb));
      if constexpr (kReal) {
        if (row_ok) {
          float* Cr = static_cast<float*>(w->C) + row_off;
#pragma unroll
          for (int u = 0; u < kUnits; ++u)
            if (unit_col(u) < tn)
              pc_store16_real(*w, cols + 16 * u, Cr, w->n0 + unit_col(u), master[u]);
        }
      } else {
        float2* Cr = static_cast<float2*>(w->C) + row_off;
#pragma unroll
        for (int u = 0; u < kUnits; ++u)
          if (unit_col(u) < tn)
            pc_store16(*w, cols + 16 * u, Cr, row_ok, w->n0 + unit_col(u), rho & 1, master[u]);
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(work_empty(cur.e));
      advance(cur);
      ++tile_cnt;
    }
  }

  ptx::tc_fence_before();
  __syncwarp();
  ptx::cluster_sync();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc2(tmem, kPcTmemCols);
  }
}

template <int P, bool kReal, bool kWide>
cudaError_t launch_products(const PieceProblem* single, const PieceProblem* dev, int nprob,
                            int64_t total_tiles, cudaStream_t stream, int* err_flag) {
  constexpr int kSmem = PcShape<P, kWide>::kSmem;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(tc1m_pieces<P, kReal, kWide>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  });
  if (attr != cudaSuccess) return attr;
  PieceProblem none;
  if (!single) {
    std::memset(static_cast<void*>(&none), 0, sizeof(none));
    single = &none;
  }
  constexpr int64_t kPairs = 76;  // pairs of SMs
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * std::min<int64_t>(total_tiles, kPairs)));
  cfg.blockDim = dim3(kPcThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 2;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = stream && stream != cudaStreamLegacy && stream != cudaStreamPerThread ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, tc1m_pieces<P, kReal, kWide>, *single, dev, nprob, total_tiles,
                            err_flag);
}

template <int P, bool kReal>
cudaError_t launch_products_w(bool wide, const PieceProblem* single, const PieceProblem* dev,
                              int nprob, int64_t tiles, cudaStream_t stream, int* err_flag) {
  return wide ? launch_products<P, kReal, true>(single, dev, nprob, tiles, stream, err_flag)
              : launch_products<P, kReal, false>(single, dev, nprob, tiles, stream, err_flag);
}

template <int P, bool kReal>
cudaError_t launch_split_t(const PieceSplit* ops, int n, const PieceSplit* dev, int64_t blocks,
                           cudaStream_t stream) {
  if (!dev && n == 1 && ops[0].mode == kSplitStep) {
    return launch_dependent(split_pieces_step<P, kReal>, dim3(static_cast<unsigned>(blocks)),
                            dim3(256), 0, stream, ops[0]);
  }
  SplitPair pair;
  std::memset(static_cast<void*>(&pair), 0, sizeof(pair));
  if (!dev) {
    if (n > 2) return cudaErrorInvalidValue;
    for (int i = 0; i < n; ++i) pair.op[i] = ops[i];
    pair.n = n;
  }
  bool many = dev;
  for (int i = 0; i < n && !dev; ++i) many = many || ops[i].kper > 1;
  return launch_dependent(many ? split_pieces<P, kReal, true> : split_pieces<P, kReal, false>,
                          dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream, pair, dev, n);
}

}  // namespace

int64_t piece_split_blocks(bool real, PieceSplit* s, bool batch) {
  s->kper = 1;
  if (s->mode == kSplitStep) {
    const int64_t nhi = s->K / s->step, nlo = s->step / (real ? 32 : 16);
    return (s->R + 7) / 8 * nlo * ((nhi + 31) / 32);
  }
  const int64_t kb = real ? split_k<true>() : split_k<false>();
  const int64_t rows = (s->R + kSplitRowsPer - 1) / kSplitRowsPer, kblocks = (s->K + kb - 1) / kb;
  // Up to four k blocks a thread block, while the GPU (152 SMs x 8 blocks)
  // keeps a round of them, counting four operands of a batch (4096^2 twice:
  // 163 us with one, 140 with four; 1024^2: 9.5 us with one, 12.3 on the form
  // for several).
  s->kper = static_cast<int32_t>(
      std::max<int64_t>(1, std::min<int64_t>(4, rows * kblocks / (batch ? 304 : 1216))));
  return rows * ((kblocks + s->kper - 1) / s->kper);
}

cudaError_t launch_piece_split(int pieces, bool real, const PieceSplit* ops, int n,
                               const PieceSplit* dev, int64_t blocks, cudaStream_t stream) {
  if (blocks <= 0) return cudaSuccess;
  if (blocks >= (int64_t(1) << 31)) return cudaErrorInvalidConfiguration;
  if (pieces == 2)
    return real ? launch_split_t<2, true>(ops, n, dev, blocks, stream)
                : launch_split_t<2, false>(ops, n, dev, blocks, stream);
  return real ? launch_split_t<3, true>(ops, n, dev, blocks, stream)
              : launch_split_t<3, false>(ops, n, dev, blocks, stream);
}

int piece_tile_n(bool real, int64_t M, int64_t N, int64_t K, int splits) {
  // Clocks of the busiest pair: its tiles times a tile's MMAs, plus a per-tile
  // cost that wide tiles do not hide (reading the accumulators) and one
  // epilogue.  An MMA of K = 16 measured 138, 105, 72 and 61 clocks at 256,
  // 192, 128 and 64 columns (complex64 4096^3; below 110 columns the reads of
  // A bound it), so widths differ mostly in how evenly their tiles fill the
  // 76 pairs: complex64 2304^3 takes 290 us at 192 columns (216 tiles), 322
  // at 128 (324) and 372 at 256 (162); 1024^3 38 us at 128, 66 at 256.
  const int64_t rows = real ? 256 : 128;
  const int64_t tm = (M + rows - 1) / rows;
  const double steps = double((real ? 1 : 2) * K) / 16 / std::max(1, splits);
  int best = 128;
  double best_cost = 1e300;
  for (int w = 256; w >= 32; w -= 32) {
    const int64_t tiles = tm * ((N + w - 1) / w) * splits;
    const int64_t waves = (tiles + 75) / 76;
    const double mma = steps * 6 * std::max(60.0, 0.55 * w);
    const double cost = double(waves) * (mma + (w > 128 ? 1500 : 300)) + 30.0 * w;
    if (cost < best_cost) {
      best_cost = cost;
      best = w;
    }
  }
  return best;
}

int piece_tile_n_batch(int64_t N) {
  int best = 128;
  double best_cost = 1e300;
  for (int w = 128; w >= 32; w -= 32) {
    const double cost = double((N + w - 1) / w) * std::max(60.0, 0.55 * w);
    if (cost < best_cost) {
      best_cost = cost;
      best = w;
    }
  }
  return best;
}

void piece_item_place(PieceItem* it, void* ws) {
  it->op[0].out = static_cast<uint8_t*>(ws);
  it->op[1].out = it->op[0].out + it->bytes[0];
  it->p.a = it->op[0].out;
  it->p.b = it->op[1].out;
}

void piece_set_tiles(bool real, PieceProblem* p, int tile_n, int splits) {
  const int64_t rows = real ? 256 : 128;
  p->tile_n = tile_n;
  p->tiles_m = static_cast<int32_t>((p->g.M + rows - 1) / rows);
  p->tiles_n = static_cast<int32_t>((p->g.N + tile_n - 1) / tile_n);
  p->splits = splits;
}

cudaError_t launch_piece_products(int pieces, bool real, bool wide, const PieceProblem* single,
                                  const PieceProblem* dev, int nprob, int64_t total_tiles,
                                  cudaStream_t stream, int* err_flag) {
  if (total_tiles <= 0) return cudaSuccess;
  if (total_tiles >= (int64_t(1) << 31)) return cudaErrorInvalidConfiguration;
  if (pieces == 2)
    return real ? launch_products_w<2, true>(wide, single, dev, nprob, total_tiles, stream, err_flag)
                : launch_products_w<2, false>(wide, single, dev, nprob, total_tiles, stream, err_flag);
  return real ? launch_products_w<3, true>(wide, single, dev, nprob, total_tiles, stream, err_flag)
              : launch_products_w<3, false>(wide, single, dev, nprob, total_tiles, stream, err_flag);
}

}  // namespace gb300
}  // namespace t1m
