// Device helpers shared by the tensor-core kernels (tc.cu, pieces.cu): error
// codes, offset lookup, the bf16 split and the scatter epilogues.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "device_common.h"
#include "internal.h"
#include "ptx.h"

namespace t1m {
namespace gb300 {
namespace {

enum : int {
  kErrFullWait = 1,
  kErrEmptyWait = 2,
  kErrAccWait = 3,
  kErrChunkWait = 4,
  kErrRawWait = 5,
  kErrAccEmptyWait = 6,
  kErrDepWait = 7,
  kErrWorkWait = 8
};

__device__ __forceinline__ void record_error(int* flag, int code) {
  // Host memory (t1m_context::d_err): a plain store, the first code seen wins.
  volatile int* const f = flag;
  if (f && *f == 0) {
    *f = code;
    __threadfence_system();
  }
}

// Split-product precision of the one-tile-per-CTA kernel.
//   TF32x3: x = hi + lo (TF32), products hi*hi + hi*lo + lo*hi (kind::tf32).
//   BF16x3: x = x0 + x1 (bf16, 8 significant bits each), products
//           x0*y0 + x0*y1 + x1*y0 (kind::f16): about 16 correct bits.
//   BF16x6: x = x0 + x1 + x2, products x0*y0 + x0*y1 + x1*y0 + x1*y1 +
//           x0*y2 + x2*y0: about 24 correct bits (FP32-class).
// The bf16 forms are the split-and-sum scheme of Henry, Tang and Heinecke,
// "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations" (ARITH 2019).
enum : int { kPrecTF32x3 = 0, kPrecBF16x3 = 1, kPrecBF16x6 = 2 };

// Split a pair of floats (consecutive K) into P packed bf16x2 words: piece 0
// is the round-to-nearest bf16 of the value, each further piece the bf16 of
// the remainder (x - x0 is exact in FP32).  Low half = x, high half = y.
template <int P>
__device__ __forceinline__ void split_bf16(float x, float y, uint32_t& w0, uint32_t& w1,
                                           uint32_t& w2) {
  w0 = ptx::cvt_bf16x2(x, y);
  const float rx = __fsub_rn(x, __uint_as_float(w0 << 16));
  const float ry = __fsub_rn(y, __uint_as_float(w0 & 0xFFFF0000u));
  w1 = ptx::cvt_bf16x2(rx, ry);
  if (P == 3) {
    const float sx = __fsub_rn(rx, __uint_as_float(w1 << 16));
    const float sy = __fsub_rn(ry, __uint_as_float(w1 & 0xFFFF0000u));
    w2 = ptx::cvt_bf16x2(sx, sy);
  }
}

// Epilogue of one converter thread: accumulator columns [col0, col0 + kCols)
// of real row 2 ci + part (part 0 holds the real parts of complex row ci,
// part 1 the imaginary parts).  Lane pairs swap halves with two shuffles per
// four columns so that each thread holds complete complex values: part 0
// writes columns 4q, 4q + 1 and part 1 columns 4q + 2, 4q + 3 of every group
// of four.  With kFlagCPairs the two values go out as one 16-byte access (a
// lane pair fills a 32-byte sector); with kFlagCCol16 one column offset is
// looked up per 16 columns.  C <- alpha*acc (+ beta*C, or + C when
// accumulating).
template <int kCols>
__device__ __forceinline__ void store_tile(const GemmArgs& g, float2* __restrict__ Cp,
                                           int64_t row, bool row_ok, int64_t n0, int col0,
                                           int part, const float (&master)[kCols],
                                           int64_t n_end = INT64_MAX) {
  const uint32_t flags = g.flags;
  const bool accumulate = flags & kFlagAccumulate;
  const bool beta_zero = flags & kFlagBetaZero;
  const bool pairs = flags & kFlagCPairs;
  const bool col16 = flags & kFlagCCol16;
  const float ar = (float)g.alpha[0], ai = (float)g.alpha[1];
  const float br = (float)g.beta[0], bi = (float)g.beta[1];
  const int64_t N = min(g.N, n_end);  // columns of this tile: [n0, N)
  const int64_t* __restrict__ csC = g.csC;
  const int64_t uC_n = g.uC_n;
  const int64_t rowC = row_ok ? offs(g.rsC, g.uC_m, row) : 0;
  float2* __restrict__ Cr = Cp + rowC;
  int64_t blk = 0;  // offset of the current 16-column block (kFlagCCol16)
#pragma unroll
  for (int q = 0; q < kCols / 4; ++q) {
    const float s0 = part ? master[4 * q] : master[4 * q + 2];
    const float s1 = part ? master[4 * q + 1] : master[4 * q + 3];
    const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1);
    const float r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
    const float re0 = part ? r0 : master[4 * q], im0 = part ? master[4 * q + 2] : r0;
    const float re1 = part ? r1 : master[4 * q + 1], im1 = part ? master[4 * q + 3] : r1;
    const int c = col0 + 4 * q + 2 * part;
    const int64_t n = n0 + c;
    if (col16 && (q & 3) == 0) {
      const int64_t nb = n0 + col0 + 16 * (q >> 2);
      blk = (row_ok && nb < N) ? offs(csC, uC_n, nb) : 0;
    }
    if (!row_ok || n >= N) continue;
    const int64_t on = col16 ? blk + (c - col0 - 16 * (q >> 2)) : offs(csC, uC_n, n);
    const bool second = n + 1 < N;
    const float t0r = ar * re0 - ai * im0, t0i = ar * im0 + ai * re0;
    const float t1r = ar * re1 - ai * im1, t1i = ar * im1 + ai * re1;
    if (pairs && second) {
      float4* p4 = reinterpret_cast<float4*>(Cr + on);
      if (accumulate) {
        const float4 o = *p4;
        *p4 = make_float4(o.x + t0r, o.y + t0i, o.z + t1r, o.w + t1i);
      } else if (beta_zero) {
        *p4 = make_float4(t0r, t0i, t1r, t1i);
      } else {
        const float4 o = *p4;
        *p4 = make_float4(t0r + (br * o.x - bi * o.y), t0i + (br * o.y + bi * o.x),
                          t1r + (br * o.z - bi * o.w), t1i + (br * o.w + bi * o.z));
      }
    } else {
      float2* p0 = Cr + on;
      float2* p1 = second ? Cr + (col16 ? on + 1 : offs(csC, uC_n, n + 1)) : p0;
      if (accumulate) {
        const float2 o = *p0;
        *p0 = make_float2(o.x + t0r, o.y + t0i);
        if (second) {
          const float2 o1 = *p1;
          *p1 = make_float2(o1.x + t1r, o1.y + t1i);
        }
      } else if (beta_zero) {
        *p0 = make_float2(t0r, t0i);
        if (second) *p1 = make_float2(t1r, t1i);
      } else {
        const float2 o = *p0;
        *p0 = make_float2(t0r + (br * o.x - bi * o.y), t0i + (br * o.y + bi * o.x));
        if (second) {
          const float2 o1 = *p1;
          *p1 = make_float2(t1r + (br * o1.x - bi * o1.y), t1i + (br * o1.y + bi * o1.x));
        }
      }
    }
  }
}

// Real epilogue: accumulator columns [col0, col0 + kCols) of real row `row`
// (one TMEM lane per row, no pairing).  For real problems kFlagCPairs means
// four consecutive columns contiguous and 16-byte aligned: one 16-byte store
// per four values.  kFlagCCol16 as in store_tile.
template <int kCols>
__device__ __forceinline__ void store_tile_real(const GemmArgs& g, float* __restrict__ Cp,
                                                int64_t row, bool row_ok, int64_t n0, int col0,
                                                const float (&master)[kCols]) {
  if (!row_ok) return;
  const uint32_t flags = g.flags;
  const bool accumulate = flags & kFlagAccumulate;
  const bool beta_zero = flags & kFlagBetaZero;
  const bool quads = flags & kFlagCPairs;
  const bool col16 = flags & kFlagCCol16;
  const float ar = (float)g.alpha[0], br = (float)g.beta[0];
  const int64_t N = g.N;
  const int64_t* __restrict__ csC = g.csC;
  const int64_t uC_n = g.uC_n;
  float* __restrict__ Cr = Cp + offs(g.rsC, g.uC_m, row);
  int64_t blk = 0;
#pragma unroll
  for (int q = 0; q < kCols / 4; ++q) {
    const int c = col0 + 4 * q;
    const int64_t n = n0 + c;
    if (col16 && (q & 3) == 0) {
      const int64_t nb = n0 + col0 + 16 * (q >> 2);
      blk = nb < N ? offs(csC, uC_n, nb) : 0;
    }
    if (n >= N) continue;
    const int64_t on = col16 ? blk + (c - col0 - 16 * (q >> 2)) : offs(csC, uC_n, n);
    float t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = ar * master[4 * q + i];
    if (quads && n + 3 < N) {
      float4* p4 = reinterpret_cast<float4*>(Cr + on);
      if (accumulate) {
        const float4 o = *p4;
        *p4 = make_float4(o.x + t[0], o.y + t[1], o.z + t[2], o.w + t[3]);
      } else if (beta_zero) {
        *p4 = make_float4(t[0], t[1], t[2], t[3]);
      } else {
        const float4 o = *p4;
        *p4 = make_float4(t[0] + br * o.x, t[1] + br * o.y, t[2] + br * o.z, t[3] + br * o.w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (n + i >= N) break;
        float* p = Cr + (col16 ? on + i : (i == 0 ? on : offs(csC, uC_n, n + i)));
        if (accumulate) *p += t[i];
        else if (beta_zero) *p = t[i];
        else *p = t[i] + br * *p;
      }
    }
  }
}

}  // namespace
}  // namespace gb300
}  // namespace t1m
