// kernels_step.cu -- single-box kernels: fused periodic step, equilibrium,
// hydrodynamic fields, FP64 import/export and compensated reductions.
#include <algorithm>

#include "cells.cuh"
#include "launch.cuh"
#include "sums.cuh"

namespace lbx {

namespace {

// Launch shape of the FP64 steps: they want instructions in flight as much as
// bytes (1,090 a cell at 128 integer lanes), so blocks of 128 threads are held
// to 64 registers, eight to an SM.  251x190x133: 253 us a step, against 290 in
// blocks of 256 at 78 registers and 264 and 301 held to 56 and 48 (spills).
constexpr int kF64Threads = 128, kF64Blocks = 8;
constexpr int kPushThreads = 128;
#define LBX_STEP_BOUNDS(T)                              \
  __launch_bounds__(sizeof(T) == 8 ? kF64Threads : 256, \
                    sizeof(T) == 8 ? kF64Blocks : 1)

// Fused collide + push-stream over a periodic valid region
// (src/AmrSim.cpp:25-135; include/component.h:22-29 written as a push:
// f_new(x + c_q, q) = C(f)(x, q) is the same map as the reference's pull
// f_new(x, q) = C(f)(x - c_q, q)).
template <typename T, bool COVER, bool PAIRED, typename I, typename C = uint32_t>
__global__ void LBX_STEP_BOUNDS(T)
    k_step_periodic(const T* __restrict__ fin, T* __restrict__ fout, Box3 b, IBox cov, T om_s,
                    T om_b, T rho0, DfRates r) {
  chain_begin();
  int x, y, z;
  if (!cell_xyz<C>(b, x, y, z)) return;
  cell_step_periodic<T, COVER, PAIRED, I>(fin, fout, b, cov, x, y, z, om_s, om_b, rho0, r);
}

// pull-form step P -> C(S(P)) (see cells.cuh); I = int when every element
// index of the store fits in 31 bits (up to 15 x 2^27 elements: 512^3)
template <typename T, bool PAIRED, typename I>
__global__ void LBX_STEP_BOUNDS(T) k_step_pull(const T* __restrict__ fin, T* __restrict__ fout,
                                                   Box3 b, T om_s, T om_b, T rho0, DfRates r) {
  chain_begin();
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  cell_step_pull<T, PAIRED, I>(fin, fout, b, x, y, z, om_s, om_b, rho0, r);
}

// the pull-form step with CalcHydroVars fused in (cell_step_pull_hydro)
template <typename T, bool PAIRED, typename I>
__global__ void LBX_STEP_BOUNDS(T) k_step_pull_hydro(const T* __restrict__ fin,
                                                         T* __restrict__ fout, Box3 b, T om_s,
                                                         T om_b, T rho0, DfRates r, double rho0_d,
                                                         double* __restrict__ rho,
                                                         double* __restrict__ u) {
  chain_begin();
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  cell_step_pull_hydro<T, PAIRED, I>(fin, fout, b, x, y, z, om_s, om_b, rho0, r, rho0_d, rho, u);
}

// Q -> R = S(Q) (SIGN = +1, leaving the pull form) or R -> Q = S^-1(R)
// (SIGN = -1, entering it): a pure shift of each population
template <typename T, int SIGN>
__global__ void k_shift(const T* __restrict__ fin, T* __restrict__ fout, Box3 b) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  T v[NV];
  gather_periodic<T, SIGN>(fin, b, x, y, z, v);
  const long long c = b.at(x, y, z);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_pop(fout, q * b.sq + c, b, v[q]);
}

template <typename T, typename C>
__global__ void k_equilibrium(const double* __restrict__ rho, const double* __restrict__ u,
                              T* __restrict__ f, Box3 b, double rho0) {
  int x, y, z;
  if (!cell_xyz<C>(b, x, y, z)) return;
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  const long long v = ((long long)z * b.n[1] + y) * b.n[0] + x;
  const double r = ld_cell(rho, v, n), ux = ld_cell(u, v, 3 * n), uy = ld_cell(u, n + v, 3 * n),
               uz = ld_cell(u, 2 * n + v, 3 * n);
  const long long c = b.at(x, y, z);
  if constexpr (sizeof(T) == 4) {
    float g[NV];
    equilibrium_shifted(r, ux, uy, uz, rho0, g);
#pragma unroll
    for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + c, b, g[q]);
  } else {
    double e[NV];
    equilibrium_f64(r, ux, uy, uz, e);
#pragma unroll
    for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + c, b, (T)(e[q] - W(q) * rho0));
  }
}

// equilibrium of rho = 1 + amplitude on the plane coord[axis] == index, u = 0
template <typename T>
__global__ void k_init_pulse(T* __restrict__ f, Box3 b, int axis, int index, double amplitude,
                             double rho0) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  const int c[3] = {x, y, z};
  const double rho = 1.0 + (c[axis] == index ? amplitude : 0.0);
  const long long s = b.at(x, y, z);
  if constexpr (sizeof(T) == 4) {
    float g[NV];
    equilibrium_shifted(rho, 0.0, 0.0, 0.0, rho0, g);
#pragma unroll
    for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + s, b, g[q]);
  } else {
    double e[NV];
    equilibrium_f64(rho, 0.0, 0.0, 0.0, e);
#pragma unroll
    for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + s, b, (T)(e[q] - W(q) * rho0));
  }
}

template <typename T, bool GATHER, typename C = uint32_t>
__global__ void k_hydro(const T* __restrict__ f, Box3 b, double rho0, double* __restrict__ rho,
                        double* __restrict__ u) {
  chain_begin();
  int x, y, z;
  if (!cell_xyz<C>(b, x, y, z)) return;
  cell_hydro<T, GATHER>(f, b, rho0, rho, u, x, y, z);
}

template <typename T, bool GATHER>
__global__ void k_copy_out(const T* __restrict__ f, Box3 b, double rho0, double* __restrict__ out) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  const long long v = ((long long)z * b.n[1] + y) * b.n[0] + x;
  const long long c = b.at(x, y, z);
  T p[NV];
  if (GATHER) {
    gather_periodic<T>(f, b, x, y, z, p);
  } else {
#pragma unroll
    for (int q = 0; q < NV; ++q) p[q] = ld_pop_ro(f, q * b.sq + c, b);
  }
#pragma unroll
  for (int q = 0; q < NV; ++q) st_cell(out, q * n + v, NV * n, (double)p[q] + W(q) * rho0);
}

template <typename T>
__global__ void k_copy_in(const double* __restrict__ in, T* __restrict__ f, Box3 b, double rho0) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  const long long v = ((long long)z * b.n[1] + y) * b.n[0] + x;
  const long long c = b.at(x, y, z);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + c, b, (T)(ld_cell(in, q * n + v, NV * n) - W(q) * rho0));
}

// valid region of a store <-> packed FAB order in the storage type (raw, no
// shift applied): checkpoints keep the exact stored values
template <typename T>
__global__ void k_pack(const T* __restrict__ f, Box3 b, T* __restrict__ out) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  const long long v = ((long long)z * b.n[1] + y) * b.n[0] + x;
  const long long c = b.at(x, y, z);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_cell(out, q * n + v, NV * n, ld_pop_ro(f, q * b.sq + c, b));
}
template <typename T>
__global__ void k_unpack(const T* __restrict__ in, T* __restrict__ f, Box3 b) {
  int x, y, z;
  if (!cell_xyz(b, x, y, z)) return;
  const long long n = (long long)b.n[0] * b.n[1] * b.n[2];
  const long long v = ((long long)z * b.n[1] + y) * b.n[0] + x;
  const long long c = b.at(x, y, z);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_pop(f, q * b.sq + c, b, ld_cell(in, q * n + v, NV * n));
}

// Mass and momentum sums.  What bounds them is the bytes of the store as long
// as the FP64 pipe is kept out of it (sums.cuh): with FP64 additions per
// population 161x128x95 FP64 took 348 us and its second pass 24.6 us, against
// 35 us for the store's 235 MB.
//
// FP64 store: a cell's populations are brought to one exponent, that of the
// block's first cell, summed exactly in 64-bit integers (fx64.cuh) and added
// to the thread's 128-bit sums.  Cells of another scale (largest population
// more than a factor of two away), or with a negative one, are summed with
// FP64 instructions, compensated; a block that met any adds both sums.
template <bool FLAT>
__device__ __forceinline__ bool reduce_cell(const Box3& b, const IBox& skip, unsigned v,
                                            long long* c) {
  if (FLAT) {  // no ghost cells, nothing left out: the store in order
    *c = v;
    return true;
  }
  const unsigned n0 = (unsigned)b.n[0], n1 = (unsigned)b.n[1], r = v / n0;
  const int x = (int)(v - r * n0), y = (int)(r % n1), z = (int)(r / n1);
  *c = b.at(x, y, z);
  return !skip.contains(x, y, z);
}

template <bool FLAT>
__device__ __forceinline__ void reduce_cells(const double* __restrict__ f, const Box3& b,
                                             const IBox& skip, unsigned n, double rho0,
                                             Sum4Shared& sh, double* __restrict__ out8) {
  uint32_t E;  // of the block's first cell (b.at(0, 0, 0) + its place, ghost or left out or not)
  {
    uint32_t h[NV], l[NV];
    long long c;
    reduce_cell<FLAT>(b, skip, min(blockIdx.x * blockDim.x, n - 1u), &c);
#pragma unroll
    for (int q = 0; q < NV; ++q) d_words(ld_pop(f, q * b.sq + c, b), &h[q], &l[q]);
    const uint32_t top = fx_top(h);
    E = fx_top_ok(top) ? top >> 20 : 1020u;
  }
  const uint32_t base = fx_base(E);
  i128 t[4] = {0, 0, 0, 0};
  Comp acc[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  bool odd = false;
  for (unsigned v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    long long c;
    if (!reduce_cell<FLAT>(b, skip, v, &c)) continue;
    double p[NV];
    uint32_t h[NV], l[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      p[q] = ld_pop(f, q * b.sq + c, b);
      d_words(p[q], &h[q], &l[q]);
    }
    const uint32_t top = fx_top(h);
    // exponent E - 1, E or E + 1: units of E hold the sums (below 2^63)
    if (fx_top_ok(top) & ((top >> 20) + 1u - E < 3u)) {
      int64_t g[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) g[q] = fx_unit(h[q], l[q], base);
      const FxSums m = fx_sums(g);
      t[0] += m.rho;
      t[1] += m.jx;
      t[2] += m.jy;
      t[3] += m.jz;
    } else {
      odd = true;
      double m = rho0, j[3] = {0, 0, 0};
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        m += p[q];
        if (CX(q)) j[0] += CX(q) * p[q];
        if (CY(q)) j[1] += CY(q) * p[q];
        if (CZ(q)) j[2] += CZ(q) * p[q];
      }
      comp_add(acc[0], m);
#pragma unroll
      for (int a = 0; a < 3; ++a) comp_add(acc[1 + a], j[a]);
    }
  }
  const bool any = __syncthreads_or(odd);
  Comp s = sum_pair(block_sum4(t, sh), (int)E - 1023 - 57);
  if (any) {
    __syncthreads();
    const Comp o = block_sum4(acc, sh);
    comp_add(s, o.s);
    s.e += o.e;
  }
  if (threadIdx.x < 32 && (threadIdx.x & 7) == 0) {
    out8[2 * (threadIdx.x >> 3)] = s.s;
    out8[2 * (threadIdx.x >> 3) + 1] = s.e;
  }
}

// FP32 store: the shifted populations are small; each cell's sums in FP32
// (rounding ~1e-9 of the fluctuations), a thread's cells summed with two
// levels of FP32 compensation (error of order 2^-72; one FP64 addition and
// one conversion per value took 34 clocks of an SM per warp, four of them
// more than the 15 loads), the threads' sums exactly; the mass is rho0 per
// cell plus the fluctuations.
struct Comp3 {
  float s, c, cc;
};
__device__ __forceinline__ void comp_add(Comp3& a, float v) {
  const dfl t = two_sum(a.s, v);
  const dfl w = two_sum(a.c, t.lo);
  a.s = t.hi;
  a.c = w.hi;
  a.cc = add_f(a.cc, w.lo);
}
__device__ __forceinline__ Comp comp_of(const Comp3& a) {
  return Comp{(double)a.s, (double)a.c + (double)a.cc};
}
template <bool FLAT>
__device__ __forceinline__ void reduce_cells(const float* __restrict__ f, const Box3& b,
                                             const IBox& skip, unsigned n, double rho0,
                                             Sum4Shared& sh, double* __restrict__ out8) {
  Comp3 t[4] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  unsigned cells = 0;
  for (unsigned v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    long long c;
    if (!reduce_cell<FLAT>(b, skip, v, &c)) continue;
    float s = 0.f, sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const float fq = ld_pop(f, q * b.sq + c, b);
      s += fq;
      if (CX(q)) sx += CX(q) * fq;
      if (CY(q)) sy += CY(q) * fq;
      if (CZ(q)) sz += CZ(q) * fq;
    }
    comp_add(t[0], s);
    comp_add(t[1], sx);
    comp_add(t[2], sy);
    comp_add(t[3], sz);
    ++cells;
  }
  Comp acc[4] = {comp_of(t[0]), comp_of(t[1]), comp_of(t[2]), comp_of(t[3])};
  comp_add(acc[0], rho0 * (double)cells);
  const Comp s = block_sum4(acc, sh);
  if (threadIdx.x < 32 && (threadIdx.x & 7) == 0) {
    out8[2 * (threadIdx.x >> 3)] = s.s;
    out8[2 * (threadIdx.x >> 3) + 1] = s.e;
  }
}

template <typename T, bool FLAT>
__global__ void __launch_bounds__(kReduceThreads) k_reduce(const T* __restrict__ f, Box3 b,
                                                           IBox skip, double rho0,
                                                           double* __restrict__ partials) {
  chain_begin();
  if (!idx_ok(blockIdx.x, kReduceBlocks)) return;  // partials hold kReduceBlocks blocks
  __shared__ Sum4Shared sh;
  // cell counts of every caller are below 2^31 (checked on the host), so the
  // index arithmetic stays in 32 bits
  const unsigned n = (unsigned)((long long)b.n[0] * b.n[1] * b.n[2]);
  reduce_cells<FLAT>(f, b, skip, n, rho0, sh, partials + 8 * blockIdx.x);
}

// the blocks' pairs: one block, a chain of latencies (24.6 us as compensated
// FP64 additions)
__global__ void __launch_bounds__(kReduceThreads) k_reduce_final(const double* __restrict__ partials,
                                                                int nblocks,
                                                                double* __restrict__ out4) {
  __shared__ Sum4Shared sh;
  static_assert(kReduceBlocks <= 2 * kReduceThreads, "two pairs a thread");
  const int i = threadIdx.x, j = i + kReduceThreads;
  Comp acc[4], more[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    acc[k] = i < nblocks ? Comp{partials[8 * i + 2 * k], partials[8 * i + 2 * k + 1]} : Comp{0, 0};
    more[k] = j < nblocks ? Comp{partials[8 * j + 2 * k], partials[8 * j + 2 * k + 1]} : Comp{0, 0};
  }
  Comp s = block_sum4(acc, sh);
  if (nblocks > kReduceThreads) {
    __syncthreads();
    const Comp o = block_sum4(more, sh);
    comp_add(s, o.s);
    s.e += o.e;
  }
  if (threadIdx.x < 32 && (threadIdx.x & 7) == 0) out4[threadIdx.x >> 3] = s.s + s.e;
}

// sum of n doubles (the mean density that shifts an FP32 store): values
// within a factor of two of the block's first in 128-bit integers, others
// compensated in FP64; the order of the blocks is fixed and each block's sum
// exact, so the sum is the same on every run
__global__ void __launch_bounds__(kReduceThreads) k_sum(const double* __restrict__ x, size_t n,
                                                       double* __restrict__ partials) {
  if (!idx_ok(blockIdx.x, kReduceBlocks)) return;
  __shared__ Sum4Shared sh;
  const size_t first = blockIdx.x * (size_t)blockDim.x, step = (size_t)gridDim.x * blockDim.x;
  uint32_t h, l;
  d_words(ld_cell(x, (long long)(first < n ? first : n - 1), (long long)n), &h, &l);
  const uint32_t E = fx_top_ok(h) ? h >> 20 : 1023u, base = fx_base(E);
  i128 t[4] = {0, 0, 0, 0};
  Comp acc[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  bool odd = false;
  constexpr int kAhead = 4;  // loads in flight per thread
  for (size_t i = first + threadIdx.x; i < n; i += kAhead * step) {
    double v[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      v[k] = i + k * step < n ? ld_cell(x, (long long)(i + k * step), (long long)n) : 0.0;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      d_words(v[k], &h, &l);
      if (fx_top_ok(h) & ((h >> 20) + 1u - E < 3u)) {
        t[0] += fx_unit(h, l, base);
      } else if (h | l) {
        odd = true;
        comp_add(acc[0], v[k]);
      }
    }
  }
  const bool any = __syncthreads_or(odd);
  Comp s = sum_pair(block_sum4(t, sh), (int)E - 1023 - 57);
  if (any) {
    __syncthreads();
    const Comp o = block_sum4(acc, sh);
    comp_add(s, o.s);
    s.e += o.e;
  }
  if (threadIdx.x < 32 && (threadIdx.x & 7) == 0) {
    partials[8 * blockIdx.x + 2 * (threadIdx.x >> 3)] = s.s;
    partials[8 * blockIdx.x + 2 * (threadIdx.x >> 3) + 1] = s.e;
  }
}

__global__ void k_fill(double* __restrict__ p, size_t n, double v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    st_cell(p, (long long)i, (long long)n, v);
}

// C-order user vectors -> FAB order (InitDensity/InitVelocity,
// src/AmrSim.cpp:138-295): rho(i,j,k) = rho_c[(i*ny + j)*nz + k],
// u(i,j,k,n) = u_c[((i*ny + j)*nz + k)*3 + n].  For each j this is a
// transpose of the (i, k) plane: a block stages a 32 x 32 tile through
// shared memory, reading it with k contiguous (C order; the three velocity
// components of a tile row are 96 contiguous values) and writing it with i
// contiguous (FAB order), so both sides are coalesced.  A null source leaves
// its field alone (a scalar initial value was filled separately).
constexpr int kTT = 32;  // tile edge
constexpr int kTR = 8;   // rows of threads (blockDim = kTT x kTR)
__global__ void __launch_bounds__(kTT * kTR)
    k_c_to_fab(const double* __restrict__ rho_c, const double* __restrict__ u_c,
               double* __restrict__ rho, double* __restrict__ u, int nx, int ny, int nz) {
  __shared__ double tr[kTT][kTT + 1];     // [i][k]
  __shared__ double tu[3][kTT][kTT + 1];  // [component][i][k]
  const int k0 = blockIdx.x * kTT, i0 = blockIdx.y * kTT, j = blockIdx.z;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const long long n = (long long)nx * ny * nz;
  const int kn = min(kTT, nz - k0), in = min(kTT, nx - i0);
  for (int r = ty; r < in; r += kTR) {
    const long long row = ((long long)(i0 + r) * ny + j) * nz + k0;  // C index of (i, j, k0)
    if (rho_c && tx < kn) tr[r][tx] = ld_cell(rho_c, row + tx, n);
    if (u_c)
      for (int e = tx; e < 3 * kn; e += kTT) tu[e % 3][r][e / 3] = ld_cell(u_c, 3 * row + e, 3 * n);
  }
  __syncthreads();
  for (int r = ty; r < kn; r += kTR) {
    if (tx >= in) continue;
    const long long v = ((long long)(k0 + r) * ny + j) * nx + i0 + tx;  // FAB index of (i, j, k)
    if (rho_c) st_cell(rho, v, n, tr[tx][r]);
    if (u_c) {
      st_cell(u, v, 3 * n, tu[0][tx][r]);
      st_cell(u, n + v, 3 * n, tu[1][tx][r]);
      st_cell(u, 2 * n + v, 3 * n, tu[2][tx][r]);
    }
  }
}


}  // namespace

cudaError_t launch_c_to_fab(const double* rho_c, const double* u_c, double* rho, double* u,
                            int nx, int ny, int nz, cudaStream_t st) {
  const dim3 grid((unsigned)((nz + kTT - 1) / kTT), (unsigned)((nx + kTT - 1) / kTT), (unsigned)ny);
  k_c_to_fab<<<grid, dim3(kTT, kTR, 1), 0, st>>>(rho_c, u_c, rho, u, nx, ny, nz);
  return cudaGetLastError();
}

// blocks of a sum over n values: three to each of the 152 SMs, fewer where a
// thread would have no value
static int reduce_grid(long long n) {
  const long long blocks = (n + kReduceThreads - 1) / kReduceThreads;
  return (int)std::min<long long>(std::max<long long>(blocks, 1), 152 * 3);
}

cudaError_t launch_sum(const double* x, size_t n, double* partials, double* out4, cudaStream_t st) {
  const int grid = reduce_grid((long long)n);
  k_sum<<<grid, kReduceThreads, 0, st>>>(x, n, partials);
  k_reduce_final<<<1, kReduceThreads, 0, st>>>(partials, grid, out4);
  return cudaGetLastError();
}

cudaError_t launch_fill(double* p, size_t n, double v, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const size_t blocks = (n + 255) / 256;
  k_fill<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, st>>>(p, n, v);
  return cudaGetLastError();
}

template <typename T, bool COVER, bool PAIRED>
static void step_periodic(const T* fin, T* fout, const Box3& b, const IBox& covered, double om_s,
                          double om_b, double rho0, const DfRates& r, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, kPushThreads);
  if (index32(b))
    chained(k_step_periodic<T, COVER, PAIRED, int>, rl.grid, rl.block, st, fin, fout, b, covered, (T)om_s, (T)om_b, (T)rho0, r);
  else if (COVER || cells32(b))  // a covered box is a simulation's
    chained(k_step_periodic<T, COVER, PAIRED, long long>, rl.grid, rl.block, st, fin, fout, b, covered, (T)om_s, (T)om_b, (T)rho0, r);
  else
    chained(k_step_periodic<T, false, PAIRED, long long, uint64_t>, rl.grid, rl.block, st, fin, fout, b, covered, (T)om_s, (T)om_b, (T)rho0, r);
}

template <typename T>
cudaError_t launch_step_periodic(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                                 double om_b, double rho0, cudaStream_t st, bool paired,
                                 bool refined) {
  const bool cov = covered.hi[0] >= covered.lo[0] && covered.hi[1] >= covered.lo[1] &&
                   covered.hi[2] >= covered.lo[2];
  const DfRates r = refined ? quiet(rates_of<T>(om_s, om_b)) : rates_of<T>(om_s, om_b);
  if constexpr (sizeof(T) == 8) {
    if (refined ? paired : collides_in_pairs(paired, r)) {
      if (cov)
        step_periodic<T, true, true>(fin, fout, b, covered, om_s, om_b, 0.0, r, st);
      else
        step_periodic<T, false, true>(fin, fout, b, covered, om_s, om_b, 0.0, r, st);
      return cudaGetLastError();
    }
  }
  if (cov)
    step_periodic<T, true, false>(fin, fout, b, covered, om_s, om_b, rho0, r, st);
  else
    step_periodic<T, false, false>(fin, fout, b, covered, om_s, om_b, rho0, r, st);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_equilibrium(const double* rho, const double* u, T* f, const Box3& b,
                               double rho0, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  if (cells32(b))
    k_equilibrium<T, uint32_t><<<rl.grid, rl.block, 0, st>>>(rho, u, f, b, rho0);
  else
    k_equilibrium<T, uint64_t><<<rl.grid, rl.block, 0, st>>>(rho, u, f, b, rho0);
  return cudaGetLastError();
}

// one row of x per (blockIdx.y, blockIdx.z), a block's threads along it;
// each warp folds its tagged cells' box and count before one atomic each
__global__ void k_tag_density(const double* __restrict__ rho, int nx, int ny, int nz, double ref,
                              double threshold, int* __restrict__ box6,
                              unsigned long long* __restrict__ count) {
  const int y = blockIdx.y, z = blockIdx.z;
  const int lane = threadIdx.x & 31;
  int lo[3] = {nx, ny, nz}, hi[3] = {-1, -1, -1};
  unsigned k = 0;
  for (int x0 = blockIdx.x * blockDim.x; x0 < nx; x0 += gridDim.x * blockDim.x) {
    const int x = x0 + threadIdx.x;
    if (x < nx && fabs(rho[((long long)z * ny + y) * nx + x] - ref) > threshold) {
      lo[0] = min(lo[0], x);
      hi[0] = max(hi[0], x);
      lo[1] = hi[1] = y;
      lo[2] = hi[2] = z;
      ++k;
    }
  }
  const unsigned all = 0xffffffffu;
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(all, lo[d]);
    hi[d] = __reduce_max_sync(all, hi[d]);
  }
  k = __reduce_add_sync(all, k);
  if (lane == 0 && k) {
    for (int d = 0; d < 3; ++d) {
      atomicMin(box6 + d, lo[d]);
      atomicMax(box6 + 3 + d, hi[d]);
    }
    atomicAdd(count, (unsigned long long)k);
  }
}

cudaError_t launch_tag_density(const double* rho, const int* n, double ref, double threshold,
                               int* box6, unsigned long long* count, cudaStream_t st) {
  const int threads = 256;
  const dim3 grid((unsigned)std::min((n[0] + threads - 1) / threads, 8), (unsigned)n[1],
                  (unsigned)n[2]);
  k_tag_density<<<grid, threads, 0, st>>>(rho, n[0], n[1], n[2], ref, threshold, box6, count);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_hydro(const T* f, const Box3& b, double rho0, double* rho, double* u,
                         cudaStream_t st, bool gather) {
  const CellLaunch rl = cell_launch(b, 128);
  if (gather)
    chained(k_hydro<T, true>, rl.grid, rl.block, st, f, b, rho0, rho, u);
  else if (cells32(b))
    chained(k_hydro<T, false>, rl.grid, rl.block, st, f, b, rho0, rho, u);
  else
    chained(k_hydro<T, false, uint64_t>, rl.grid, rl.block, st, f, b, rho0, rho, u);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_copy_out(const T* f, const Box3& b, double rho0, double* out, cudaStream_t st,
                            bool gather) {
  const CellLaunch rl = cell_launch(b, 128);
  if (gather)
    k_copy_out<T, true><<<rl.grid, rl.block, 0, st>>>(f, b, rho0, out);
  else
    k_copy_out<T, false><<<rl.grid, rl.block, 0, st>>>(f, b, rho0, out);
  return cudaGetLastError();
}

// FP32: blocks of 128 threads while both stores fit in the 129 MB of L2, where
// the step is bound by latency (80^3: 6.70 us against 6.97 in blocks of 256), of
// 256 where it is bound by HBM (512^3: 2,313 us against 2,349)
template <typename T>
static int pull_threads(const Box3& b) {
  if (sizeof(T) == 8) return kF64Threads;
  return 2ll * NV * (long long)sizeof(T) * b.sq <= 129000000ll ? 128 : 256;
}

template <typename T, typename I>
cudaError_t launch_step_pull_i(const T* fin, T* fout, const Box3& b, double om_s, double om_b,
                               double rho0, bool paired, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, pull_threads<T>(b));
  if constexpr (sizeof(T) == 8) {
    if (collides_in_pairs(paired, df_rates(om_s, om_b))) {
      chained(k_step_pull<double, true, I>, rl.grid, rl.block, st, fin, fout, b, om_s, om_b, 0.0,
                                                                 df_rates(om_s, om_b));
      return cudaGetLastError();
    }
  }
  chained(k_step_pull<T, false, I>, rl.grid, rl.block, st, fin, fout, b, (T)om_s, (T)om_b, (T)rho0,
                                                          rates_of<T>(om_s, om_b));
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_step_pull(const T* fin, T* fout, const Box3& b, double om_s, double om_b,
                             double rho0, bool paired, cudaStream_t st) {
  // 64-bit element indices only where a store needs them: they cost a fifth of
  // the FP32 step's instructions (80^3: 8.33 us a step against 6.97, 512^3: 2,401
  // against 2,313) and more of the FP64 one's registers
  if (index32(b))
    return launch_step_pull_i<T, int>(fin, fout, b, om_s, om_b, rho0, paired, st);
  return launch_step_pull_i<T, long long>(fin, fout, b, om_s, om_b, rho0, paired, st);
}

template <typename T, typename I>
cudaError_t launch_step_pull_hydro_i(const T* fin, T* fout, const Box3& b, double om_s,
                                     double om_b, double rho0, bool paired, double* rho,
                                     double* u, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, pull_threads<T>(b));
  if constexpr (sizeof(T) == 8) {
    if (collides_in_pairs(paired, df_rates(om_s, om_b))) {
      chained(k_step_pull_hydro<double, true, I>, rl.grid, rl.block, st, fin, fout, b, om_s, om_b, 0.0, df_rates(om_s, om_b), rho0, rho, u);
      return cudaGetLastError();
    }
  }
  chained(k_step_pull_hydro<T, false, I>, rl.grid, rl.block, st, fin, fout, b, (T)om_s, (T)om_b,
                                                               (T)rho0, rates_of<T>(om_s, om_b), rho0, rho, u);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_step_pull_hydro(const T* fin, T* fout, const Box3& b, double om_s, double om_b,
                                   double rho0, bool paired, double* rho, double* u,
                                   cudaStream_t st) {
  if (index32(b))
    return launch_step_pull_hydro_i<T, int>(fin, fout, b, om_s, om_b, rho0, paired, rho, u, st);
  return launch_step_pull_hydro_i<T, long long>(fin, fout, b, om_s, om_b, rho0, paired, rho, u, st);
}

template <typename T>
cudaError_t launch_init_pulse(T* f, const Box3& b, int axis, int index, double amplitude,
                              double rho0, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_init_pulse<T><<<rl.grid, rl.block, 0, st>>>(f, b, axis, index, amplitude, rho0);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_unstream(const T* fin, T* fout, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_shift<T, -1><<<rl.grid, rl.block, 0, st>>>(fin, fout, b);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_stream_gather(const T* fin, T* fout, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_shift<T, 1><<<rl.grid, rl.block, 0, st>>>(fin, fout, b);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_copy_in(const double* in, T* f, const Box3& b, double rho0, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_copy_in<T><<<rl.grid, rl.block, 0, st>>>(in, f, b, rho0);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_pack(const T* f, const Box3& b, T* out, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_pack<T><<<rl.grid, rl.block, 0, st>>>(f, b, out);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_unpack(const T* in, T* f, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = cell_launch(b, 128);
  k_unpack<T><<<rl.grid, rl.block, 0, st>>>(in, f, b);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_reduce(const T* f, const Box3& b, IBox skip, double rho0, double* partials,
                          double* out4, cudaStream_t st) {
  const int grid = reduce_grid((long long)b.n[0] * b.n[1] * b.n[2]);
  const bool none = skip.hi[0] < skip.lo[0] || skip.hi[1] < skip.lo[1] || skip.hi[2] < skip.lo[2];
  if (b.g == 0 && none)
    chained(k_reduce<T, true>, grid, kReduceThreads, st, f, b, skip, rho0, partials);
  else
    chained(k_reduce<T, false>, grid, kReduceThreads, st, f, b, skip, rho0, partials);
  k_reduce_final<<<1, kReduceThreads, 0, st>>>(partials, grid, out4);
  return cudaGetLastError();
}

#define LBX_INST(T)                                                                             \
  template cudaError_t launch_step_periodic<T>(const T*, T*, const Box3&, IBox, double, double, \
                                               double, cudaStream_t, bool, bool);               \
  template cudaError_t launch_equilibrium<T>(const double*, const double*, T*, const Box3&,     \
                                             double, cudaStream_t);                             \
  template cudaError_t launch_hydro<T>(const T*, const Box3&, double, double*, double*,         \
                                       cudaStream_t, bool);                                     \
  template cudaError_t launch_copy_out<T>(const T*, const Box3&, double, double*, cudaStream_t, \
                                          bool);                                                \
  template cudaError_t launch_step_pull_hydro<T>(const T*, T*, const Box3&, double, double,    \
                                                 double, bool, double*, double*, cudaStream_t);  \
  template cudaError_t launch_step_pull<T>(const T*, T*, const Box3&, double, double, double,  \
                                           bool, cudaStream_t);                                 \
  template cudaError_t launch_unstream<T>(const T*, T*, const Box3&, cudaStream_t);             \
  template cudaError_t launch_init_pulse<T>(T*, const Box3&, int, int, double, double,          \
                                            cudaStream_t);                                      \
  template cudaError_t launch_stream_gather<T>(const T*, T*, const Box3&, cudaStream_t);        \
  template cudaError_t launch_copy_in<T>(const double*, T*, const Box3&, double, cudaStream_t);  \
  template cudaError_t launch_reduce<T>(const T*, const Box3&, IBox, double, double*, double*,  \
                                        cudaStream_t);                                          \
  template cudaError_t launch_pack<T>(const T*, const Box3&, T*, cudaStream_t);                 \
  template cudaError_t launch_unpack<T>(const T*, T*, const Box3&, cudaStream_t);
LBX_INST(double)
LBX_INST(float)
#undef LBX_INST

}  // namespace lbx
