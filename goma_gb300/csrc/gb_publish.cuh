// Device helpers shared by the triangular sweeps and the vector kernels: the
// arithmetic type of a vector's elements, and solution values published one
// by one through a sentinel.
#pragma once
#include <cuda_runtime.h>

namespace gb {

// Arithmetic type of the vector kernels: FP64 data is combined in FP64, FP32
// data in FP32.  On GB300 FP64 arithmetic runs at 1/64 of the FP32 rate, so
// an FP32 kernel that widened its operands to FP64 would be bound by the
// FP64 pipe instead of HBM; the FP32 inner solve gets its accuracy from the
// FP64 refinement around it.
template <class T>
struct AccT {
  using type = double;
};
template <>
struct AccT<float> {
  using type = float;
};
template <class T>
using acc_t = typename AccT<T>::type;
__device__ __forceinline__ double fmx(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmx(float a, float b, float c) { return fmaf(a, b, c); }

// the "unpublished" sentinels: signalling NaNs (exponent all ones, quiet bit
// clear, non-zero payload)
static constexpr unsigned long long kUnpub64 = 0xFFF5DEAD5EEDF00DULL;
static constexpr unsigned kUnpub32 = 0xFFA5EED5u;
__device__ __forceinline__ bool unpublished(double v) {
  return (unsigned long long)__double_as_longlong(v) == kUnpub64;
}
__device__ __forceinline__ bool unpublished(float v) { return __float_as_uint(v) == kUnpub32; }
__device__ __forceinline__ void set_unpublished(double *p) {
  *p = __longlong_as_double((long long)kUnpub64);
}
__device__ __forceinline__ void set_unpublished(float *p) { *p = __uint_as_float(kUnpub32); }

__device__ __forceinline__ double ld_relaxed(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_relaxed(const float *p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(double *p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(float *p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

}  // namespace gb
