// Products with a small output and a long contracted bundle (complex64,
// BF16x6): both operands are streamed once, straight from the tensors.
//
// Such a product (abcd,dbea->ec: 96 x 64 over K = 36864) reads far more than
// it computes or writes, and its operands need not be matrices: packing them
// first, or writing their pieces, moves their bytes three to six times.  Here
// every CTA takes one K range of one output tile (64 complex rows x up to 128
// columns) and gathers its elements through the scatter vectors into
// registers, one stage ahead; the converter warps split them into bf16 pieces
// (tc_common.h) and store them as the 1M rows of the first operand and the
// rows of the second in the MMA's 128-byte-swizzled shared-memory layout.  The
// partial products of the K ranges go to the split-K workspace and are summed
// in FP64 (splitk.cu).  It replaces the reference's packing and five-loop GEMM
// for these shapes (t1m.h:309-337, 508-554).
//
// A stage is 32 complex k.  Where each operand has its unit stride along
// another K mode, the K order interleaves them (HostPlan::stream_k: 4 x 8 or 8
// x 4), so a stage is whole 32-byte sectors of both.  K ranges hold at most 12
// stages (outputs of up to 64 columns: 28): three (seven) main chunk
// accumulators of 16 MMAs each and the corrections fill TMEM, and nothing is
// folded before the end (the precision of pieces.cu, whose chunks are as long).
// Which products run so: stream_pays (stream.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>

#include "device_common.h"
#include "internal.h"
#include "pc_epilogue.h"
#include "ptx.h"
#include "stream.h"
#include "t1m_capi.h"
#include "tc_common.h"

namespace t1m {
namespace gb300 {
namespace {

constexpr int kStRows = 64;         // complex rows of a tile: 128 1M rows
constexpr int kStCols = 128;        // columns of a tile
constexpr int kStK = 32;            // complex k per stage: one 128-byte row per piece
constexpr int kStMaxStages = 28;    // per K range (see st_max_stages)
constexpr int kStWarps = 16;        // converter and epilogue warps; warp 16 issues MMAs
constexpr int kStThreads = 32 * (kStWarps + 1);
constexpr int kStPiece = 128 * 128;               // one piece of either operand
constexpr int kStX = 3 * kStPiece;
constexpr int kStStage = 2 * kStX;                // 96 KB
constexpr int kStBarriers = 256;
constexpr int kStMaxK = kStMaxStages * kStK;
constexpr int kStSmem = 1024 + 2 * kStStage + kStBarriers + (kStRows + kStCols + 2 * kStMaxK) * 8 +
                        static_cast<int>(sizeof(PcWork)) + kStWarps * 32 * 8;
static_assert(kStSmem <= 227 * 1024, "shared memory budget");
// TMEM columns of an accumulator, and the stages whose chunk accumulators fit
// beside the corrections: 12 at 128 columns, 28 at 64 or less.
__host__ __device__ constexpr int st_acc_cols(int64_t cols) { return cols > 64 ? 128 : 64; }
__host__ __device__ constexpr int st_max_stages(int64_t cols) {
  return 4 * (512 / st_acc_cols(cols) - 1);
}
static_assert(st_max_stages(64) == kStMaxStages, "K offsets of a range");

struct StreamArgs {
  const float2* x;                // first operand (1M rows), second operand
  const float2* y;
  const int64_t *xr, *xk, *yr, *yk;   // row and K offsets, or uniform strides
  int64_t uxr, uxk, uyr, uyk;
  int64_t rows, cols, K;
  int32_t conj_x, conj_y;
  GemmArgs g;                     // C with rows and columns in this order
};

// A stage takes 32 to 64 bytes of a line, later stages the rest: the whole
// line comes from HBM at once.
__device__ __forceinline__ float2 st_load(const float2* p) {
  float2 v;
  asm volatile("ld.global.nc.L2::128B.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// Byte offset of 16-byte chunk c of row r in a piece (8-row atoms of 1024
// bytes, 128-byte rows, chunks XOR-permuted by the row).
__device__ __forceinline__ uint32_t st_chunk(int r, int c) {
  return static_cast<uint32_t>((r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}
__device__ __forceinline__ void st_word(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// Rows warp + 16 j of a piece start 2 (1M rows: 4) atoms apart with the same
// swizzle, so one address per thread and constants reach all of them.
constexpr uint32_t kStXStep = 4 * 1024, kStYStep = 2 * 1024;
__device__ __forceinline__ void st_quad(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}
// The word [im, re] of a pair's pieces from its word [re, -im].
__device__ __forceinline__ uint32_t st_second(uint32_t w) {
  return __byte_perm(w, 0u, 0x1032) ^ 0x8000u;
}

// kXRows / kYRows: the operand has unit stride along its rows (consecutive
// threads take consecutive rows, four k each); else consecutive lanes take
// the stage's 32 k of one row.
template <bool kXRows, bool kYRows>
__global__ void __launch_bounds__(kStThreads, 1)
stream_contract(const __grid_constant__ StreamArgs s, int tiles_n, int* err_flag) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const base_ptr = smem_raw + (base - ptx::smem_u32(smem_raw));
  const uint32_t bars = base + 2 * kStStage;
  auto full_bar = [&](int b) { return bars + 8u * b; };
  auto empty_bar = [&](int b) { return bars + 8u * (2 + b); };
  const uint32_t acc_bar = bars + 32u, tmem_slot = bars + 40u;
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(base_ptr + (tmem_slot - base));
  int64_t* const xoff = reinterpret_cast<int64_t*>(base_ptr + 2 * kStStage + kStBarriers);
  int64_t* const yoff = xoff + kStRows;
  int64_t* const xk = yoff + kStCols;   // K offsets of the whole range, -1 past it
  int64_t* const yk = xk + kStMaxK;
  int64_t* const col_offsets = yk + kStMaxK;
  PcWork* const work = reinterpret_cast<PcWork*>(col_offsets + kStWarps * 32);

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int64_t row0 = int64_t(blockIdx.x / tiles_n) * kStRows;
  const int64_t col0 = int64_t(blockIdx.x % tiles_n) * kStCols;
  const int64_t kb = int64_t(blockIdx.y) * s.g.k_per_split;
  const int64_t ke = min(s.K, kb + s.g.k_per_split);
  const int nst = static_cast<int>((ke - kb + kStK - 1) / kStK);
  const int ncols = static_cast<int>(min(int64_t(kStCols), s.cols - col0));
  const int nrows = static_cast<int>(min(int64_t(kStRows), s.rows - row0));
  const uint32_t acc_cols = st_acc_cols(s.cols);

  if (warp == kStWarps) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
    if (lane == 0) {
      for (int b = 0; b < 2; ++b) {
        ptx::mbar_init(full_bar(b), kStWarps);
        ptx::mbar_init(empty_bar(b), 1);
      }
      ptx::mbar_init(acc_bar, 1);
      ptx::fence_mbar_init();
      const GemmArgs& g = s.g;
      PcWork& w = *work;
      w.C = static_cast<float2*>(g.C) + int64_t(blockIdx.y) * g.c_split_stride;
      w.rsC = g.rsC;
      w.csC = g.csC;
      w.uC_m = g.uC_m;
      w.uC_n = g.uC_n;
      w.M = g.M;
      w.N = g.N;
      w.alpha[0] = static_cast<float>(g.alpha[0]);
      w.alpha[1] = static_cast<float>(g.alpha[1]);
      w.beta[0] = static_cast<float>(g.beta[0]);
      w.beta[1] = static_cast<float>(g.beta[1]);
      w.flags = g.flags;
    }
  }
  begin_dependent();
  // Every offset the range needs, once: looked up per stage, an offset's
  // latency preceded its elements' (33 us for abcd,dbea->ec against 21).
  for (int i = tid; i < nst * kStK; i += kStThreads) {
    const bool in = kb + i < ke;
    xk[i] = in ? offs(s.xk, s.uxk, kb + i) : -1;
    yk[i] = in ? offs(s.yk, s.uyk, kb + i) : -1;
  }
  if (tid < kStRows) {
    xoff[tid] = row0 + tid < s.rows ? offs(s.xr, s.uxr, row0 + tid) : -1;
  } else if (tid >= 128 && tid < 128 + kStCols) {
    const int j = tid - 128;
    yoff[j] = col0 + j < s.cols ? offs(s.yr, s.uyr, col0 + j) : -1;
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot_ptr, 0);

  if (warp == kStWarps) {
    // ---------------------------------------------------------- MMA issue ---
    const bool issue = ptx::elect_one();
    const uint64_t desc0 = ptx::smem_desc_sw128(base);
    const uint32_t idesc =
        ptx::idesc_f32acc(1u /*BF16*/, 128u, static_cast<uint32_t>((ncols + 15) / 16 * 16));
    const int steps = static_cast<int>((2 * (ke - kb) + 15) / 16);
    for (int st = 0; st < nst; ++st) {
      const int b = st & 1;
      if (!ptx::mbar_wait(full_bar(b), static_cast<uint32_t>((st >> 1) & 1))) {
        record_error(err_flag, kErrFullWait);
        break;
      }
      ptx::tc_fence_after();
      const uint64_t ds = desc0 + static_cast<uint32_t>((b * kStStage) >> 4);
      const uint32_t d_main = tmem + acc_cols * (st >> 2), d_corr = tmem + 512u - acc_cols;
      const int nkk = min(4, steps - 4 * st);
      auto mma = [&](uint32_t d, int px, int py, int kk, uint32_t acc) {
        ptx::mma_f16_ss(d, ds + ((px * kStPiece + 32 * kk) >> 4),
                        ds + ((kStX + py * kStPiece + 32 * kk) >> 4), idesc, acc);
      };
      if (issue) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (kk < nkk) mma(d_main, 0, 0, kk, ((st & 3) == 0 && kk == 0) ? 0u : 1u);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (kk < nkk) {
            mma(d_corr, 0, 1, kk, (st == 0 && kk == 0) ? 0u : 1u);
            mma(d_corr, 1, 0, kk, 1u);
            mma(d_corr, 1, 1, kk, 1u);
            mma(d_corr, 0, 2, kk, 1u);
            mma(d_corr, 2, 0, kk, 1u);
          }
        ptx::mma_commit(empty_bar(b));
      }
    }
    // No MMA may still write TMEM when it is freed.
    if (issue) ptx::mma_commit(acc_bar);
    if (!ptx::mbar_wait(acc_bar, 0)) record_error(err_flag, kErrAccWait);
    __syncwarp();
  } else {
    // --------------------------------------------------------- converters ---
    // Elements of this thread in a stage: four of x, eight of y.
    struct Elements {
      float2 x[4], y[8];
    };
    auto load = [&](Elements& e, int st) {
      const int kl = st * kStK;
      auto get = [](const float2* p, int64_t ro, int64_t ko) {
        return ro >= 0 && ko >= 0 ? st_load(p + ro + ko) : make_float2(0.f, 0.f);
      };
      if constexpr (kXRows) {
        const int64_t ro = xoff[tid & 63];
#pragma unroll
        for (int j = 0; j < 4; ++j) e.x[j] = get(s.x, ro, xk[kl + 4 * (tid >> 6) + j]);
      } else {
        const int64_t ko = xk[kl + lane];
#pragma unroll
        for (int j = 0; j < 4; ++j) e.x[j] = get(s.x, xoff[warp + kStWarps * j], ko);
      }
      if constexpr (kYRows) {
        const int64_t ro = yoff[tid & 127];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          e.y[j] = get(s.y, ro, yk[kl + 4 * ((tid >> 7) + 4 * (j >> 2)) + (j & 3)]);
      } else {
        const int64_t ko = yk[kl + lane];
#pragma unroll
        for (int j = 0; j < 8; ++j) e.y[j] = get(s.y, yoff[warp + kStWarps * j], ko);
      }
    };
    const uint32_t x_at = st_chunk(2 * warp, lane >> 2) + 4 * (lane & 3);
    const uint32_t x_at2 = st_chunk(2 * warp + 1, lane >> 2) + 4 * (lane & 3);
    const uint32_t y_at = st_chunk(warp, lane >> 2) + 4 * (lane & 3);
    const float sx = s.conj_x ? -1.f : 1.f, sy = s.conj_y ? -1.f : 1.f;
    auto put = [&](const Elements& e, int b) {
      const uint32_t xs = base + b * kStStage, ys = xs + kStX;
      if constexpr (kXRows) {
        uint32_t w[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          split_bf16<3>(e.x[j].x, -sx * e.x[j].y, w[0][j], w[1][j], w[2][j]);
        const int r = tid & 63, c = tid >> 6;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          st_quad(xs + p * kStPiece + st_chunk(2 * r, c), w[p]);
#pragma unroll
          for (int j = 0; j < 4; ++j) w[p][j] = st_second(w[p][j]);
          st_quad(xs + p * kStPiece + st_chunk(2 * r + 1, c), w[p]);
        }
      } else {
        const uint32_t x0 = xs + x_at, x1 = xs + x_at2;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (warp + kStWarps * j >= nrows) break;  // uniform over the warp
          uint32_t w[3];
          split_bf16<3>(e.x[j].x, -sx * e.x[j].y, w[0], w[1], w[2]);
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            st_word(x0 + (j * kStXStep + p * kStPiece), w[p]);
            st_word(x1 + (j * kStXStep + p * kStPiece), st_second(w[p]));
          }
        }
      }
      if constexpr (kYRows) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w[3][4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            split_bf16<3>(e.y[4 * h + j].x, sy * e.y[4 * h + j].y, w[0][j], w[1][j], w[2][j]);
          const int r = tid & 127, c = (tid >> 7) + 4 * h;
          if (r < ncols) {
#pragma unroll
            for (int p = 0; p < 3; ++p) st_quad(ys + p * kStPiece + st_chunk(r, c), w[p]);
          }
        }
      } else {
        const uint32_t y0 = ys + y_at;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (warp + kStWarps * j >= ncols) break;  // uniform over the warp
          uint32_t w[3];
          split_bf16<3>(e.y[j].x, sy * e.y[j].y, w[0], w[1], w[2]);
#pragma unroll
          for (int p = 0; p < 3; ++p) st_word(y0 + (j * kStYStep + p * kStPiece), w[p]);
        }
      }
    };
    // One stage of elements in flight per thread beside the one being split
    // (a second one gained nothing: the splitting, not the loads, bounds this).
    Elements e[2];
    if (nst > 0) load(e[0], 0);
    bool ok = true;
#pragma unroll 1
    for (int st0 = 0; st0 < nst && ok; st0 += 2) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int st = st0 + b;
        if (st >= nst) break;
        if (st + 1 < nst) load(e[b ^ 1], st + 1);
        if (st >= 2 && !ptx::mbar_wait(empty_bar(b), static_cast<uint32_t>(((st >> 1) - 1) & 1))) {
          record_error(err_flag, kErrEmptyWait);
          ok = false;
          break;
        }
        put(e[b], b);
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(full_bar(b));
      }
    }
    // ----------------------------------------------------------- epilogue ---
    const int q = warp & 3, wg = warp >> 2;
    const int rho = 32 * q + lane;  // 1M row = TMEM lane
    const int64_t row = row0 + (rho >> 1);
    const bool row_ok = row < work->M;
    const int64_t row_off = row_ok ? offs(work->rsC, work->uC_m, row) : 0;
    int64_t* const cols = col_offsets + warp * 32;
    const int64_t n = col0 + 32 * wg + lane;
    cols[lane] = n < work->N ? offs(work->csC, work->uC_n, n) : 0;
    __syncwarp();
    if (!ptx::mbar_wait(acc_bar, 0)) {
      record_error(err_flag, kErrAccWait);
      ok = false;
    }
    ptx::tc_fence_after();
    if (ok) {
      const int nchunks = (nst + 3) / 4;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c0 = 32 * wg + 16 * u;
        if (c0 >= ncols) break;  // uniform over the warp
        float acc[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = 0.f;
        for (int c = 0; c <= nchunks; ++c) {
          uint32_t r[16];
          ptx::tmem_ld16_sync(tmem + (static_cast<uint32_t>(32 * q) << 16) +
                                  (c == nchunks ? 512u - acc_cols : acc_cols * c) + c0, r);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[j] += __uint_as_float(r[j]);
        }
        pc_store16(*work, cols + 16 * u, static_cast<float2*>(work->C) + row_off, row_ok, col0 + c0,
                   rho & 1, acc);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == kStWarps) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

template <bool kXRows, bool kYRows>
cudaError_t launch(const StreamArgs& s, dim3 grid, int tiles_n, cudaStream_t stream, int* err_flag) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(stream_contract<kXRows, kYRows>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kStSmem);
  });
  if (attr != cudaSuccess) return attr;
  return launch_dependent(stream_contract<kXRows, kYRows>, grid, dim3(kStThreads), kStSmem, stream, s,
                          tiles_n, err_flag);
}

}  // namespace

int stream_splits(int64_t M, int64_t N, int64_t K, int64_t* k_per_split) {
  // Short sides and a long bundle: fewer than 128 products per element read
  // (2 M N / (M + N)); above that the pieces form reads its copies often
  // enough.
  if (M * N >= 64 * (M + N) || K < 1024) return 0;
  const int64_t rows = std::min(M, N), cols = std::max(M, N);
  const int64_t tiles = ((rows + kStRows - 1) / kStRows) * ((cols + kStCols - 1) / kStCols);
  const int64_t stages = (K + kStK - 1) / kStK;
  // K ranges of at least two stages, as long as whole waves of the 152 SMs
  // allow.
  const int64_t most = st_max_stages(cols);
  int64_t per = 2;
  for (int64_t waves = 1;; ++waves) {
    per = (stages * tiles + 152 * waves - 1) / (152 * waves);
    if (per <= most) break;
  }
  per = std::max<int64_t>(2, per);
  // The partial products, written and read back, stay below the operands, and
  // within the split-K workspace.
  auto splits_of = [&](int64_t p) { return (stages + p - 1) / p; };
  auto fits = [&](int64_t s) {
    return s * M * N * 2 <= (M + N) * K &&
           (s == 1 || size_t(s) * size_t(M) * size_t(N) * 8 <= kMaxWorkBytes);
  };
  while (per < most && !fits(splits_of(per))) ++per;
  const int64_t splits = splits_of(per);
  if (!fits(splits) || splits > 65535 || tiles > 0x7fffffffLL) return 0;
  *k_per_split = per * kStK;
  return static_cast<int>(splits);
}

bool stream_pays(int fetch, int64_t M, int64_t N, int64_t K, int splits, int64_t kps, int other,
                 int64_t other_kps) {
  if (fetch == kStreamGathered) return true;
  const int64_t rows = std::min(M, N), cols = std::max(M, N);
  const int64_t tiles = ((rows + kStRows - 1) / kStRows) * ((cols + kStCols - 1) / kStCols);
  if (fetch == kStreamSectors)
    return tiles == 1 || K <= 14000;
  if (M > 64 || tiles == 1 || tiles * ((K + kStK - 1) / kStK) <= 7 * 152) return true;
  auto busiest = [](int64_t ctas, int64_t k) { return double((ctas + 151) / 152 * k); };
  const int64_t other_tiles = (N + 127) / 128;  // 64 rows: one tile
  return busiest(tiles * splits, kps) * (1.1 + double(rows) / 90) <=
         busiest(other_tiles * other, other_kps);
}

cudaError_t launch_stream(const GemmArgs& g, const StreamLayout& lay, int splits,
                          cudaStream_t stream, int* err_flag) {
  StreamArgs s;
  std::memset(static_cast<void*>(&s), 0, sizeof(s));
  // The smaller side takes the 1M rows.
  const bool swap = g.N < g.M;
  s.g = g;
  if (swap) {
    std::swap(s.g.M, s.g.N);
    std::swap(s.g.rsC, s.g.csC);
    std::swap(s.g.uC_m, s.g.uC_n);
  }
  s.g.flags = (g.flags & ~(kFlagCPairs | kFlagCCol16)) | lay.store_flags;
  const float2* const A = static_cast<const float2*>(g.A);
  const float2* const B = static_cast<const float2*>(g.B);
  s.x = swap ? B : A;
  s.y = swap ? A : B;
  const int64_t *ak = g.csA, *bk = g.rsB;
  int64_t uak = g.uA_k, ubk = g.uB_k;
  if (lay.a_k && lay.b_k) {
    ak = lay.a_k;
    bk = lay.b_k;
    uak = ubk = -1;
  }
  s.xr = swap ? g.csB : g.rsA;
  s.uxr = swap ? g.uB_n : g.uA_m;
  s.xk = swap ? bk : ak;
  s.uxk = swap ? ubk : uak;
  s.yr = swap ? g.rsA : g.csB;
  s.uyr = swap ? g.uA_m : g.uB_n;
  s.yk = swap ? ak : bk;
  s.uyk = swap ? uak : ubk;
  s.rows = s.g.M;
  s.cols = s.g.N;
  s.K = g.K;
  const bool ca = g.flags & kFlagConjA, cb = g.flags & kFlagConjB;
  s.conj_x = swap ? cb : ca;
  s.conj_y = swap ? ca : cb;
  const bool xrows = swap ? lay.b_rows : lay.a_rows, yrows = swap ? lay.a_rows : lay.b_rows;
  const int64_t tiles_m = (s.rows + kStRows - 1) / kStRows, tiles_n = (s.cols + kStCols - 1) / kStCols;
  const dim3 grid(static_cast<unsigned>(tiles_m * tiles_n), static_cast<unsigned>(splits));
  const int tn = static_cast<int>(tiles_n);
  if (xrows)
    return yrows ? launch<true, true>(s, grid, tn, stream, err_flag)
                 : launch<true, false>(s, grid, tn, stream, err_flag);
  return yrows ? launch<false, true>(s, grid, tn, stream, err_flag)
               : launch<false, false>(s, grid, tn, stream, err_flag);
}

}  // namespace gb300
}  // namespace t1m
