// Epilogue of the tensor-core kernels that keep whole tiles in registers
// (pieces.cu, stream.cu): 16 columns of one TMEM lane at a time.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace t1m {
namespace gb300 {
namespace {

// Tile of an output as an epilogue sees it (and, for pieces.cu, as its loads
// do): C and its offsets, the tile's first row and column, the epilogue.
struct PcWork {
  const uint8_t* a;     // this CTA's rows and columns in the first stage, piece 0
  const uint8_t* b;
  int64_t pa, pb;       // bytes from piece to piece
  void* C;              // of the tile's split
  const int64_t *rsC, *csC;
  int64_t uC_m, uC_n;
  int64_t row0, M, n0, N;
  float alpha[2], beta[2];
  uint32_t flags;
  uint32_t abytes, bbytes;  // per piece and stage (row groups that exist)
  int32_t steps;        // K = 16 MMA steps; 0: no more tiles
  int32_t tn;
  int32_t swapped;
};

// C <- alpha * acc (+ beta * C, or + C when accumulating) for the 16 columns
// [n0, n0 + 16) below N of complex row at Cr: lane pairs hold its real (part
// 0) and imaginary row.  As store_tile, but old values are read together
// before any is written, so accumulating products wait once per group
// instead of once per access.
// `cols`: the 16 columns' offsets, in shared memory.
__device__ __forceinline__ void pc_store16(const PcWork& w, const int64_t* cols,
                                           float2* __restrict__ Cr, bool row_ok, int64_t n0,
                                           int part, const float* acc) {
  const uint32_t flags = w.flags;
  const bool accumulate = flags & kFlagAccumulate, read = accumulate || !(flags & kFlagBetaZero);
  const bool col16 = flags & kFlagCCol16;
  const float ar = w.alpha[0], ai = w.alpha[1], br = w.beta[0], bi = w.beta[1];
  const int64_t N = w.N;
  if (n0 >= N) return;  // uniform over the warp
  float2 v[8];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float s0 = part ? acc[4 * q] : acc[4 * q + 2];
    const float s1 = part ? acc[4 * q + 1] : acc[4 * q + 3];
    const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1);
    const float r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
    const float re0 = part ? r0 : acc[4 * q], im0 = part ? acc[4 * q + 2] : r0;
    const float re1 = part ? r1 : acc[4 * q + 1], im1 = part ? acc[4 * q + 3] : r1;
    v[2 * q] = make_float2(ar * re0 - ai * im0, ar * im0 + ai * re0);
    v[2 * q + 1] = make_float2(ar * re1 - ai * im1, ar * im1 + ai * re1);
  }
  if (!row_ok) return;
  auto combine = [&](float2 t, float2 o) {
    return accumulate ? make_float2(o.x + t.x, o.y + t.y)
                      : make_float2(t.x + (br * o.x - bi * o.y), t.y + (br * o.y + bi * o.x));
  };
  // Value 2 q + e belongs to column n0 + 4 q + 2 part + e.
  if ((flags & kFlagCPairs) && col16 && n0 + 16 <= N) {
    float4* p = reinterpret_cast<float4*>(Cr + cols[0] + 2 * part);
    if (read) {
      float4 o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = p[2 * q];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[2 * q] = combine(v[2 * q], make_float2(o[q].x, o[q].y));
        v[2 * q + 1] = combine(v[2 * q + 1], make_float2(o[q].z, o[q].w));
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      p[2 * q] = make_float4(v[2 * q].x, v[2 * q].y, v[2 * q + 1].x, v[2 * q + 1].y);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // four values at a time
      float2* p[4];
      bool in[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = 8 * h + 4 * (i >> 1) + 2 * part + (i & 1);
        in[i] = n0 + c < N;
        p[i] = Cr + cols[c];
      }
      if (read) {
        float2 o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = in[i] ? *p[i] : make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * h + i] = combine(v[4 * h + i], o[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (in[i]) *p[i] = v[4 * h + i];
    }
  }
}

// The real form: columns [n0, n0 + 16) of one real row per lane.
__device__ __forceinline__ void pc_store16_real(const PcWork& w, const int64_t* cols,
                                                float* __restrict__ Cr, int64_t n0,
                                                const float* acc) {
  const uint32_t flags = w.flags;
  const bool accumulate = flags & kFlagAccumulate, read = accumulate || !(flags & kFlagBetaZero);
  const float ar = w.alpha[0], br = w.beta[0];
  const int64_t N = w.N;
  if (n0 >= N) return;
  auto combine = [&](float t, float o) { return accumulate ? o + t : t + br * o; };
  if ((flags & kFlagCPairs) && (flags & kFlagCCol16) && n0 + 16 <= N) {
    float4* p = reinterpret_cast<float4*>(Cr + cols[0]);
    float4 o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = read ? p[q] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 t = make_float4(ar * acc[4 * q], ar * acc[4 * q + 1], ar * acc[4 * q + 2],
                             ar * acc[4 * q + 3]);
      if (read)
        t = make_float4(combine(t.x, o[q].x), combine(t.y, o[q].y), combine(t.z, o[q].z),
                        combine(t.w, o[q].w));
      p[q] = t;
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // eight values at a time
      float* p[8];
      bool in[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        in[i] = n0 + 8 * h + i < N;
        p[i] = Cr + cols[8 * h + i];
      }
      float o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = read && in[i] ? *p[i] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float t = ar * acc[8 * h + i];
        if (in[i]) *p[i] = read ? combine(t, o[i]) : t;
      }
    }
  }
}

}  // namespace
}  // namespace gb300
}  // namespace t1m
