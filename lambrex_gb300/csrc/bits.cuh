// bits.cuh -- words of FP32 and FP64 values and the FP32 helpers shared by the
// paired-FP32 (df32.cuh) and the fixed-point (fx64.cuh) collision; on the host
// they are plain C++, so that the tests run the kernels' code off the GPU.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

namespace lbx {

__host__ __device__ __forceinline__ float f_bits(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  std::memcpy(&f, &b, 4);
  return f;
#endif
}
__host__ __device__ __forceinline__ uint32_t bits_f(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t b;
  std::memcpy(&b, &f, 4);
  return b;
#endif
}
__host__ __device__ __forceinline__ void d_words(double x, uint32_t* hi, uint32_t* lo) {
#ifdef __CUDA_ARCH__
  *hi = (uint32_t)__double2hiint(x);
  *lo = (uint32_t)__double2loint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  *hi = (uint32_t)(b >> 32);
  *lo = (uint32_t)b;
#endif
}
__host__ __device__ __forceinline__ double d_from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
__host__ __device__ __forceinline__ float u2f(uint32_t r) {
#ifdef __CUDA_ARCH__
  return __uint2float_rn(r);
#else
  return (float)r;
#endif
}

// to an integer toward zero, a value beyond the largest to that one (as the
// device's conversion does; C++ leaves it undefined)
__host__ __device__ __forceinline__ int f2i(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rz(x);
#else
  return x >= 0x1p31f ? 0x7fffffff : (int)x;
#endif
}

// approximate FP32 reciprocal (the hardware's; any error below 2^-16 will do)
__host__ __device__ __forceinline__ float rcp_approx(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
}  // namespace lbx
