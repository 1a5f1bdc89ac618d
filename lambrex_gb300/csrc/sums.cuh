// sums.cuh -- sums of many FP64 values over a block in 128-bit integers.
//
// GB300's FP64 pipe takes 17 clocks of an SM for one FP64 instruction of a
// warp, so a tree of compensated FP64 additions over a block's 256 threads
// (40 merges of 8 instructions per warp) costs more than reading the cells
// that are summed.  The values of a block are brought to one exponent instead
// and added as integers: exactly, on the integer pipe, in any order.
#pragma once
#include "fx64.cuh"

namespace lbx {

using i128 = __int128;
using u128 = unsigned __int128;

// Neumaier-compensated pair (s, e): value = s + e.
struct Comp {
  double s, e;
};

#ifdef __CUDACC__
__device__ __forceinline__ void comp_add(Comp& a, double v) {
  const double t = a.s + v;
  if (fabs(a.s) >= fabs(v))
    a.e += (a.s - t) + v;
  else
    a.e += (v - t) + a.s;
  a.s = t;
}

// exponent field of x, 1 for zeros and subnormals (2047: infinity or NaN)
__device__ __forceinline__ uint32_t sum_exponent(double x) {
  const uint32_t e = ((uint32_t)__double2hiint(x) >> 20) & 2047u;
  return e ? e : 1u;
}
// x in units of 2^-100 of the power of two of exponent field E >= x's own
// (|value| below 2^101; what lies below one unit is cut)
__device__ __forceinline__ i128 sum_units(double x, uint32_t E) {
  const uint32_t hi = (uint32_t)__double2hiint(x);
  const uint32_t f = (hi >> 20) & 2047u;
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | (f ? 0x100000u : 0u)) << 32) |
                     (uint32_t)__double2loint(x);
  const int s = 48 - (int)(E - (f ? f : 1u));
  u128 v = 0;
  if (s >= 0)
    v = (u128)m << s;
  else if (s > -64)
    v = m >> -s;
  return (int)hi < 0 ? -(i128)v : (i128)v;
}
// v units of 2^unit as a pair, exact to 106 bits
__device__ __forceinline__ Comp sum_pair(i128 v, int unit) {
  const bool neg = v < 0;
  const u128 m = neg ? -(u128)v : (u128)v;
  if (m == 0) return Comp{0.0, 0.0};
  const uint64_t mh = (uint64_t)(m >> 64);
  const int lead = mh ? 127 - __clzll((long long)mh) : 63 - __clzll((long long)(uint64_t)m);
  const int cut = lead > 52 ? lead - 52 : 0;
  const uint64_t top = (uint64_t)(m >> cut);
  u128 rest = m - ((u128)top << cut);
  const int cut2 = cut > 53 ? cut - 53 : 0;  // the rest to 53 bits too
  rest >>= cut2;
  const double s = ldexp((double)(long long)top, unit + cut);
  const double e = ldexp((double)(long long)(uint64_t)rest, unit + cut2);
  return neg ? Comp{-s, -e} : Comp{s, e};
}

__device__ __forceinline__ i128 shfl_down_i128(i128 v, int o) {
  const uint64_t lo = __shfl_down_sync(0xffffffffu, (uint64_t)(u128)v, o);
  const uint64_t hi = __shfl_down_sync(0xffffffffu, (uint64_t)((u128)v >> 64), o);
  return (i128)(((u128)hi << 64) | lo);
}

// Sums of each thread's four integers over the block (at most 8 warps, all
// threads call it, block-uniform); the sum k is returned in thread 8 k of the
// first warp.
struct Sum4Shared {
  i128 v[4][8];
  uint32_t e[4][8];
};
__device__ __forceinline__ i128 block_sum4(const i128* v, Sum4Shared& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    i128 t = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += shfl_down_i128(t, o);
    if (lane == 0) sh.v[k][warp] = t;
  }
  __syncthreads();
  i128 t = 0;
  if (warp == 0) {
    if ((lane & 7) < nw) t = sh.v[lane >> 3][lane & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += shfl_down_i128(t, o);
  }
  return t;
}

// Sums of each thread's four pairs over the block; the sum k is returned in
// thread 8 k of the first warp.  NaN where a value is infinite or NaN.
__device__ __forceinline__ Comp block_sum4(const Comp* c, Sum4Shared& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t E[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    E[k] = __reduce_max_sync(0xffffffffu, fx_umax(sum_exponent(c[k].s), sum_exponent(c[k].e)));
    if (lane == 0) sh.e[k][warp] = E[k];
  }
  __syncthreads();
  i128 v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    E[k] = __reduce_max_sync(0xffffffffu, sh.e[k][lane < nw ? lane : 0]);
    v[k] = sum_units(c[k].s, E[k]) + sum_units(c[k].e, E[k]);
  }
  const i128 t = block_sum4(v, sh);
  const int k = lane >> 3;
  const uint32_t Ek = k == 0 ? E[0] : k == 1 ? E[1] : k == 2 ? E[2] : E[3];
  if (Ek == 2047u) return Comp{nan(""), 0.0};
  return sum_pair(t, (int)Ek - 1023 - 100);
}
#endif

}  // namespace lbx
