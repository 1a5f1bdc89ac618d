// checked.cuh -- global-memory accessors with the bounds checks of the debug
// build.
//
// Every kernel reads and writes population stores and per-cell fields
// through ld_pop / st_pop / ld_cell / st_cell.  In the release library they
// are plain loads and stores.  Built with LBX_CHECKED
// (liblbx_cuda_checked.so) each access first tests its element index against
// the extent of the array it addresses -- NV * sq elements for a population
// store of box b, the cell count for a per-cell field -- and on a miss counts
// it in a device counter of the translation unit, remembers the first bad
// index and skips the access (loads return 0).  Nothing traps; the host reads
// and clears the counters with lbx_debug_bounds().
#pragma once
#include <cuda_runtime.h>

#include "d3q15.cuh"

namespace lbx {

#ifdef LBX_CHECKED
// [0] = number of out-of-range accesses, [1] = first bad index (as written)
static __device__ unsigned long long g_oob[2];

__host__ __device__ __forceinline__ bool idx_ok(long long i, long long n) {
  if (i >= 0 && i < n) return true;
#ifdef __CUDA_ARCH__
  if (atomicAdd(&g_oob[0], 1ull) == 0ull) g_oob[1] = (unsigned long long)i;
#endif
  return false;
}

// Each translation unit that includes this header registers a reader of its
// own counters; lbx_debug_bounds() sums them.
using OobReader = int (*)(unsigned long long* count, long long* first, bool reset);
int register_oob_reader(OobReader r);

static int read_unit_oob(unsigned long long* count, long long* first, bool reset) {
  unsigned long long h[2] = {0ull, 0ull};
  if (cudaMemcpyFromSymbol(h, g_oob, sizeof h) != cudaSuccess) return -1;
  *count = h[0];
  *first = (long long)h[1];
  if (reset) {
    const unsigned long long z[2] = {0ull, 0ull};
    if (cudaMemcpyToSymbol(g_oob, z, sizeof z) != cudaSuccess) return -1;
  }
  return 0;
}
static const int g_oob_unit_registered = register_oob_reader(&read_unit_oob);
#else
__host__ __device__ __forceinline__ constexpr bool idx_ok(long long, long long) { return true; }
#endif

// read-only cached load on the device (a plain load in a host build)
template <typename T>
__host__ __device__ __forceinline__ T ld_ro(const T* p) {
#ifdef __CUDA_ARCH__
  return __ldg(p);
#else
  return *p;
#endif
}
// plain load of what an earlier kernel wrote: not through the read-only cache
// and not moved ahead of chain_begin() (launch.cuh); on the host a plain load,
// as the tests run the per-cell code off the GPU
__host__ __device__ __forceinline__ double ld_plain(const double* p) {
#ifdef __CUDA_ARCH__
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
#else
  return *p;
#endif
}
__host__ __device__ __forceinline__ float ld_plain(const float* p) {
#ifdef __CUDA_ARCH__
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
#else
  return *p;
#endif
}

// population store of box b: element index i = q * sq + cell (I: the
// index type of the caller, 64-bit or, for the batch engine's small boxes,
// 32-bit)
template <typename T, typename I>
__host__ __device__ __forceinline__ T ld_pop(const T* __restrict__ p, I i, const Box3& b) {
  return idx_ok((long long)i, NV * b.sq) ? ld_plain(p + i) : T(0);
}
// the same through the read-only cache, for kernels that are not chained: a
// compiler may move these ahead of the kernel's stores
template <typename T, typename I>
__host__ __device__ __forceinline__ T ld_pop_ro(const T* __restrict__ p, I i, const Box3& b) {
  return idx_ok((long long)i, NV * b.sq) ? ld_ro(p + i) : T(0);
}
// load of an entry the same kernel may also write (no read-only cache)
template <typename T, typename I>
__host__ __device__ __forceinline__ T ld_pop_rw(const T* p, I i, const Box3& b) {
  return idx_ok((long long)i, NV * b.sq) ? p[i] : T(0);
}
template <typename T, typename I>
__host__ __device__ __forceinline__ void st_pop(T* __restrict__ p, I i, const Box3& b, T v) {
  if (idx_ok((long long)i, NV * b.sq)) p[i] = v;
}

__host__ __device__ __forceinline__ unsigned ld_plain(const unsigned* p) {
#ifdef __CUDA_ARCH__
  unsigned v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
#else
  return *p;
#endif
}

// two neighbours of a row from an even element on, in one access
__host__ __device__ __forceinline__ void ld_plain2(const double* p, double* v) {
#ifdef __CUDA_ARCH__
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
#else
  v[0] = p[0], v[1] = p[1];
#endif
}
__host__ __device__ __forceinline__ void ld_plain2(const float* p, float* v) {
#ifdef __CUDA_ARCH__
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p));
#else
  v[0] = p[0], v[1] = p[1];
#endif
}
template <typename T, typename I>
__host__ __device__ __forceinline__ void ld_pop2(const T* __restrict__ p, I i, const Box3& b, T* v) {
  v[0] = v[1] = T(0);
  if (idx_ok((long long)i, NV * b.sq) && idx_ok((long long)i + 1, NV * b.sq)) ld_plain2(p + i, v);
}
__host__ __device__ __forceinline__ void st_plain2(double* p, double v) {
#ifdef __CUDA_ARCH__
  *reinterpret_cast<double2*>(p) = make_double2(v, v);
#else
  p[0] = p[1] = v;
#endif
}
__host__ __device__ __forceinline__ void st_plain2(float* p, float v) {
#ifdef __CUDA_ARCH__
  *reinterpret_cast<float2*>(p) = make_float2(v, v);
#else
  p[0] = p[1] = v;
#endif
}
// v into both
template <typename T, typename I>
__host__ __device__ __forceinline__ void st_pop2(T* __restrict__ p, I i, const Box3& b, T v) {
  if (idx_ok((long long)i, NV * b.sq) && idx_ok((long long)i + 1, NV * b.sq)) st_plain2(p + i, v);
}

// per-cell field of n elements (density, velocity components, partial sums)
template <typename T>
__host__ __device__ __forceinline__ T ld_cell(const T* __restrict__ p, long long i, long long n) {
  return idx_ok(i, n) ? ld_ro(p + i) : T(0);
}
template <typename T>
__host__ __device__ __forceinline__ void st_cell(T* __restrict__ p, long long i, long long n, T v) {
  if (idx_ok(i, n)) p[i] = v;
}

}  // namespace lbx
