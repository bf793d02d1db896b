// Device helpers shared by the simpfem kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace simpfem {

// Explicitly rounded arithmetic: the vector updates mirror the reference's
// numpy/CuPy expressions operation by operation (one rounding per operator),
// so contraction into FMA is suppressed where the reference rounds twice.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

template <typename T>
__device__ __forceinline__ float to_f(T v) { return (float)v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ double to_d(T v) { return (double)v; }
template <>
__device__ __forceinline__ double to_d<__nv_bfloat16>(__nv_bfloat16 v) {
  return (double)__bfloat162float(v);
}

template <typename T>
__device__ __forceinline__ T from_d(double v) { return (T)v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_d<__nv_bfloat16>(double v) {
  return __float2bfloat16_rn((float)v);
}

__device__ __forceinline__ bool guard_off(const int* g) { return g != nullptr && *g == 0; }

// First smoothing step from a zero start on entry i with right-hand side r
// (run_smoother's step 0: x = (s dinv) r, or d = dinv r and x = s d).
template <typename T>
__device__ __forceinline__ void zero_start(const ZeroStart& z, int64_t i, T r) {
  if (z.mode == 1) {
    ((T*)z.x)[i] = mul_rn(mul_rn((T)z.s, ((const T*)z.dinv)[i]), r);
  } else if (z.mode == 2) {
    const T d = mul_rn(((const T*)z.dinv)[i], r);
    ((T*)z.d)[i] = d;
    ((T*)z.x)[i] = mul_rn((T)z.s, d);
  }
}

// v[0] + v[1] + ... + v[n - 1] (shared memory, 16-byte aligned, zeros from n to a
// multiple of sixteen) added one by one; sixteen values are loaded together, so the
// chain waits for additions only (a zero added at its end changes nothing).
__device__ __forceinline__ double ordered_sum(const double* v, int n) {
  double s = 0.0;
#pragma unroll 1
  for (int b = 0; b < n; b += 16) {
    double2 c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = reinterpret_cast<const double2*>(v + b)[q];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s += c[q].x;
      s += c[q].y;
    }
  }
  return s;
}

inline int div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

}  // namespace simpfem
