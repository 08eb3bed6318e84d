// Element helpers of the SIMT kernels (simt.cu, small_tile.cu): complex and real
// arithmetic by element type, offset lookup and asynchronous element copies.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "device_common.h"

namespace t1m {
namespace gb300 {
namespace {

template <class T> struct Scalar;
template <> struct Scalar<float> {
  using real = float;
  static constexpr bool cplx = false;
};
template <> struct Scalar<double> {
  using real = double;
  static constexpr bool cplx = false;
};
template <> struct Scalar<float2> {
  using real = float;
  static constexpr bool cplx = true;
};
template <> struct Scalar<double2> {
  using real = double;
  static constexpr bool cplx = true;
};

template <class T> __device__ __forceinline__ T zero();
template <> __device__ __forceinline__ float zero<float>() { return 0.f; }
template <> __device__ __forceinline__ double zero<double>() { return 0.0; }
template <> __device__ __forceinline__ float2 zero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ double2 zero<double2>() { return make_double2(0.0, 0.0); }

__device__ __forceinline__ float conj_if(float v, bool) { return v; }
__device__ __forceinline__ double conj_if(double v, bool) { return v; }
__device__ __forceinline__ float2 conj_if(float2 v, bool c) { if (c) v.y = -v.y; return v; }
__device__ __forceinline__ double2 conj_if(double2 v, bool c) { if (c) v.y = -v.y; return v; }

// acc += a * b
__device__ __forceinline__ void mac(float& acc, float a, float b) { acc = fmaf(a, b, acc); }
__device__ __forceinline__ void mac(double& acc, double a, double b) { acc = fma(a, b, acc); }
__device__ __forceinline__ void mac(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(-a.y, b.y, acc.x);
  acc.y = fmaf(a.y, b.x, acc.y);
  acc.y = fmaf(a.x, b.y, acc.y);
}
__device__ __forceinline__ void mac(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.y, b.x, acc.y);
  acc.y = fma(a.x, b.y, acc.y);
}

template <class T> __device__ __forceinline__ T scal(const double* s);
template <> __device__ __forceinline__ float scal<float>(const double* s) { return (float)s[0]; }
template <> __device__ __forceinline__ double scal<double>(const double* s) { return s[0]; }
template <> __device__ __forceinline__ float2 scal<float2>(const double* s) { return make_float2((float)s[0], (float)s[1]); }
template <> __device__ __forceinline__ double2 scal<double2>(const double* s) { return make_double2(s[0], s[1]); }

__device__ __forceinline__ float mul(float a, float b) { return a * b; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ float2 mul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

}  // namespace
}  // namespace gb300
}  // namespace t1m
