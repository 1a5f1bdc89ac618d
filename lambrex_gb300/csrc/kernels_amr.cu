// kernels_amr.cu -- coarse/fine coupling kernels.
//
// Three schemes share these files.  The reference-faithful one restates the
// Rohde cycle of src/AmrSim.cpp:430-631 as separate FP64 passes over
// ghost-cell boxes (fill patch, collide, stream, zero invalid, sum from fine).
// The conservative one is the library's volumetric scheme: the coarse
// post-collision populations that head into the patch are exploded onto the
// fine ghost shell (constant over the coarse step, so no time interpolation
// is needed), the fine level sub-cycles twice, and every population that left
// the patch is coalesced back with volume weight 1/8; total mass is conserved
// to round-off.  The rescaled one keeps the covered coarse cells active,
// refills the fine ghost shell before every sub-step from the parents
// interpolated in time, with the non-equilibrium part rescaled between the
// levels, and restricts the covered cells after the two sub-steps.
#include <algorithm>

#include "cells.cuh"
#include "launch.cuh"
#include "faithful.cuh"

namespace lbx {

namespace {

// storage coordinates of a grown box: (sx, sy, sz) in [0, n + 2g).  Storage
// rows (n + 4 cells) are never a multiple of a warp, so each x-y plane is
// flattened over blocks of `threads` (grid.x) and z is grid.y (grown_launch);
// one multiplicative division per thread recovers (sx, sy).
struct GIdx {
  int x, y, z;
};
__device__ __forceinline__ bool grown_index(const Box3& b, GIdx& s) {
  const int SX = b.n[0] + 2 * b.g;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= SX * (b.n[1] + 2 * b.g)) return false;
  s.y = (int)divide((uint32_t)t, b.srow);
  s.x = t - s.y * SX;
  s.z = blockIdx.y;
  return true;
}
inline CellLaunch grown_launch(const Box3& b, int threads) {
  const int plane = (b.n[0] + 2 * b.g) * (b.n[1] + 2 * b.g);
  return CellLaunch{dim3((unsigned)((plane + threads - 1) / threads), (unsigned)(b.n[2] + 2 * b.g), 1),
                   dim3((unsigned)threads, 1, 1)};
}
// ------------------------------------------------------------------ conservative

template <typename T, bool PAIRED, typename I>
__global__ void k_explode(const T* __restrict__ coarse, T* __restrict__ fine, Coupling c, T om_s,
                          T om_b, T rho0, DfRates r) {
  chain_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  int s[3];
  if (t >= ghost_cells_of(c.fb) || !ghost_coords(c.fb, t, s)) return;
  cell_explode<T, PAIRED, I>(coarse, fine, c, s[0], s[1], s[2], om_s, om_b, rho0, r);
}

// FP64: eight blocks an SM (64 registers): a rescaled two-level coarse step of
// 104x88x72 took 158 us, against 162, 164 and 169 with six, five and four.  FP32:
// the compiler's own choice, 48 registers (conservative 64^3 21.4 us against 22.2
// at the 56 that it takes when told of one block; 128^3 154.8 against 154.0)
template <typename T, bool COVER, bool PAIRED, typename I>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 8 : 0)
    k_step_patch(const T* __restrict__ fin, T* __restrict__ fout, Box3 b, IBox cov, T om_s, T om_b,
                 T rho0, DfRates r, const unsigned* moving) {
  chain_begin();
  if (sizeof(T) == 8 && moving && ld_plain(moving)) r.fx.quiet = 0;
  GIdx s;
  if (!grown_index(b, s)) return;
  cell_step_patch<T, COVER, PAIRED, I>(fin, fout, b, cov, s.x, s.y, s.z, om_s, om_b, rho0, r);
}

template <typename T, typename I>
__global__ void k_coalesce(const T* __restrict__ fine, T* __restrict__ coarse, Coupling c, T rho0) {
  chain_begin();
  // (ring cell, population), neighbouring ring cells of one population per
  // warp: their children and coarse entries lie side by side
  const int cell = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
  int r[3];
  if (cell >= ring_cells_of(c) || !ring_coords(c, cell, r)) return;
  cell_coalesce_q<T, I>(fine, coarse, c, r[0], r[1], r[2], q, rho0);
}

// one thread a covered cell and population, neighbouring cells of one per warp
// (a thread a cell took 13.5 to 14.2 us whatever the size, its loads in turn;
// 9,216 / 32,768 / 49,152 covered cells, FP32, out of L2: 4.3 / 6.6 / 8.0)
template <typename T, typename I>
__global__ void k_restrict(const T* __restrict__ fine, T* __restrict__ coarse, Coupling c) {
  const int ex = c.fb.n[0] / 2, ey = c.fb.n[1] / 2, ez = c.fb.n[2] / 2;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)ex * ey * ez) return;
  const int rx = (int)(t % ex), ry = (int)((t / ex) % ey), rz = (int)(t / ((long long)ex * ey));
  cell_restrict_q<T, I>(fine, coarse, c, rx, ry, rz, blockIdx.y);
}

template <typename T, bool PAIRED, typename I>
__global__ void k_explode_resc(const T* __restrict__ cprev, const T* __restrict__ cnow,
                               T* __restrict__ fine, Coupling c, T om_s, T om_b, T rho0, T wp, T wn,
                               DfRates r, const unsigned* moving) {
  chain_begin();
  if (sizeof(T) == 8 && moving && ld_plain(moving)) r.fx.quiet = 0;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (sizeof(T) == 8) {
    Ring g;
    if (t >= ring_cells_of(c) || !ring_coords(c, t, g.r)) return;
    ring_explode_resc<T, PAIRED, I>(cprev, cnow, fine, c, g, om_s, om_b, rho0, wp, wn, r);
  } else {
    int s[3];
    if (t >= ghost_cells_of(c.fb) || !ghost_coords(c.fb, t, s)) return;
    cell_explode_resc<T, PAIRED, I>(cprev, cnow, fine, c, s[0], s[1], s[2], om_s, om_b, rho0, wp, wn, r);
  }
}

// The step of a periodic level and the explosion of the state it starts from in
// one launch: they read the same store and write different ones.  The explosion
// alone is a chain of latencies (4 us for the 2 MB of a 32^3 patch, at 15 % of
// the warp slots); as the first blocks of the step's launch it is done before
// the step is.  64^3 conservative FP32: 25.4 -> 22.9 us a coarse step.
template <typename T, bool COVER, bool PAIRED, typename I, bool RESC>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 8 : RESC ? 1 : 0)
    k_step_explode(const T* __restrict__ fin, T* __restrict__ fout, Box3 b, IBox cov, T om_s, T om_b,
                   T rho0, DfRates r, T* __restrict__ fine, Coupling c, T es, T eb, DfRates re,
                   unsigned first, const unsigned* moving) {
  chain_begin();
  if (RESC && sizeof(T) == 8 && moving && ld_plain(moving)) r.fx.quiet = re.fx.quiet = 0;
  if (blockIdx.x < first) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int s[3];
    if (t >= ghost_cells_of(c.fb) || !ghost_coords(c.fb, t, s)) return;
    if (RESC)  // the state before the step alone
      cell_explode_resc<T, PAIRED, I, true>(fin, fin, fine, c, s[0], s[1], s[2], es, eb, rho0, T(1), T(0), re);
    else
      cell_explode<T, PAIRED, I>(fin, fine, c, s[0], s[1], s[2], om_s, om_b, rho0, r);
    return;
  }
  int x, y, z;
  if (!cell_xyz(b, x, y, z, first)) return;
  cell_step_periodic<T, COVER, PAIRED, I>(fin, fout, b, cov, x, y, z, om_s, om_b, rho0, r);
}

// Whether anything moves on a level, of the cells at every fourth place: sets
// *moving, which the last kernel of the step before cleared.  While a patch is at
// rest, its cells and the coarse ones take the FP64 instructions (collide_f64);
// once a wave is in it, what is rounding alone no longer shows, and the fluid at
// rest elsewhere is collided in fixed point like the rest (a pulse's first 20 steps
// in 104x88x72, rescaled: 5.5 to 8.3 ms without the look, 3.4 to 4.4 with it, 3.2
// and 3.3 later on).  So the look chooses between two roundings of cells at rest:
// last bits depend on it, and a wave that it misses leaves them at the error of the
// FP64 instructions.
__global__ void __launch_bounds__(128) k_moving(const double* __restrict__ f, Box3 b, unsigned* moving) {
  chain_begin();
  const int nx = (b.n[0] + 3) / 4, ny = (b.n[1] + 3) / 4, nz = (b.n[2] + 3) / 4;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  bool moves = false;
  if (t < nx * ny * nz) {
    const long long c = b.at(4 * (t % nx), 4 * (t / nx % ny), 4 * (t / (nx * ny)));
    double p[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) p[q] = ld_pop(f, q * b.sq + c, b);
    moves = !at_rest(p);
  }
  if (__syncthreads_or(moves) && threadIdx.x == 0) *moving = 1;
}

template <typename T, bool PAIRED, typename I>
__global__ void k_restrict_resc(const T* __restrict__ fine, T* __restrict__ coarse, Coupling c,
                                T om_s, T om_b, T rho0, DfRates r, unsigned* moving) {
  chain_begin();
  if (moving && blockIdx.x == 0 && threadIdx.x == 0) *moving = 0;  // until the next look
  const int ex = c.fb.n[0] / 2, ey = c.fb.n[1] / 2, ez = c.fb.n[2] / 2;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)ex * ey * ez) return;
  const int rx = (int)(t % ex), ry = (int)((t / ex) % ey), rz = (int)(t / ((long long)ex * ey));
  cell_restrict_resc<T, PAIRED, I>(fine, coarse, c, rx, ry, rz, om_s, om_b, rho0, r);
}

// The same for few cells: one thread a cell takes its fifteen means one after
// the other, each a round of loads.  Here four warps take a quarter of the
// populations of 32 cells each, and the first of them collides the means.
// Where the line lies: us a coarse step, one thread a cell against this, FP64
// with 1,728 / 13,824 / 32,768 / 64,000 / 82,368 / 190,000 covered cells 33.9 / 48.2
// / 76.7 / 115.0 / 136.9 / 277.7 against 29.1 / 45.6 / 74.0 / 113.5 / 141.5 / 280.8
// (36.1 / 51.1 / 78.8 / 117.2 / 141.6 / 281.9 before the loads ran ahead); FP32 with
// 32,768 / 82,368 / 128,128 / 262,144 28.9 / 66.2 / 95.2 / 187.3 against 26.9 / 63.7 /
// 94.4 / 189.7.  From there on a thread a cell fills the chip, and this form's
// blocks hold three idle warps while the first collides.
constexpr int kMeanCells = 32, kMeanWarps = 4;
constexpr long long kFewCells = 1 << 16;
template <typename T, bool PAIRED, typename I>
__global__ void __launch_bounds__(kMeanCells* kMeanWarps, sizeof(T) == 8 ? 0 : 8)
    k_restrict_resc_few(const T* __restrict__ fine, T* __restrict__ coarse, Coupling c, T om_s,
                        T om_b, T rho0, DfRates r, unsigned* moving) {
  __shared__ T mean[NV][kMeanCells];
  chain_begin();
  if (moving && blockIdx.x == 0 && threadIdx.x == 0) *moving = 0;
  const int ex = c.fb.n[0] / 2, ey = c.fb.n[1] / 2, ez = c.fb.n[2] / 2;
  const int lane = threadIdx.x % kMeanCells, part = threadIdx.x / kMeanCells;
  const int t = blockIdx.x * kMeanCells + lane;
  const bool in = t < ex * ey * ez;
  const int rx = t % ex, ry = (t / ex) % ey, rz = t / (ex * ey);
#pragma unroll
  for (int k = 0; k < NV; k += kMeanWarps)
    if (in && k + part < NV) {
      T v[8];
      ld_covered<T, I>(fine, c, rx, ry, rz, k + part, v);
      mean[k + part][lane] = mean8(v);
    }
  __syncthreads();
  if (part != 0 || !in) return;
  T f[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) f[q] = mean[q][lane];
  const I cc = covered_index<I>(c, rx, ry, rz), csq = (I)c.cb.sq;
  collide_cell<T, PAIRED, true>(f, om_s, om_b, rho0, r);
#pragma unroll
  for (int q = 0; q < NV; ++q) st_pop(coarse, (I)q * csq + cc, c.cb, f[q]);
}

template <typename T>
__global__ void k_fill_from_coarse(const T* __restrict__ coarse, T* __restrict__ fine, Coupling c) {
  GIdx s;
  if (!grown_index(c.fb, s)) return;
  cell_fill_from_coarse<T>(coarse, fine, c, s.x, s.y, s.z);
}

// ------------------------------------------------------------------ faithful (FP64)

__global__ void k_f_fill_single(const double* __restrict__ src, double* __restrict__ dst, Box3 b) {
  GIdx s;
  if (!grown_index(b, s)) return;
  f_cell_fill_single(src, dst, b, s.x, s.y, s.z);
}

__global__ void k_f_fill_two(const double* __restrict__ fnow, double* __restrict__ dst,
                             const double* __restrict__ cnow, Coupling c, int fdx, int fdy,
                             int fdz) {
  GIdx s;
  if (!grown_index(c.fb, s)) return;
  f_cell_fill_two(fnow, dst, cnow, c, fdx, fdy, fdz, s.x, s.y, s.z);
}

__global__ void k_f_zero_ring0(double* __restrict__ f, Box3 b) {
  GIdx s;
  if (!grown_index(b, s)) return;
  f_cell_zero_ring0(f, b, s.x, s.y, s.z);
}

// ROWS: a block's threads stand along rows of x, padded to warps, not along the
// cells in storage order.  For the paired collision of small boxes with rows
// longer than a warp: cells that the pairs cannot hold (empty populations behind
// the covered cells' edge) lie at the same places of many rows, a warp with any of
// them takes the FP64 instructions too, and there are too few warps to hide it.
// us, rows | storage order: 48x40x32 12.2 | 15.9, 40^3 13.9 | 14.9, 48^3 18.1 | 18.1,
// 20x60x60 21.9 | 17.4, 100x90x70 48.8 | 43.9, 130^3 144 | 126.
template <bool PAIRED, bool ROWS = false>
__global__ void k_f_collide(double* __restrict__ f, Box3 b, IBox cov, double om_s, double om_b,
                            DfRates r) {
  int x, y, z;
  if (ROWS) {
    x = blockIdx.x * blockDim.x + threadIdx.x;
    y = blockIdx.y * blockDim.y + threadIdx.y;
    z = blockIdx.z;
    if (x >= b.n[0] || y >= b.n[1]) return;
  } else if (!cell_xyz(b, x, y, z)) {
    return;
  }
  f_cell_collide<PAIRED>(f, b, cov, x, y, z, om_s, om_b, r);
}

__global__ void k_f_stream(const double* __restrict__ src, double* __restrict__ dst, Box3 b) {
  GIdx s;
  if (!grown_index(b, s)) return;
  f_cell_stream(src, dst, b, s.x, s.y, s.z);
}

__global__ void k_f_fill_boundary(double* __restrict__ f, Box3 b) {
  GIdx s;
  if (!grown_index(b, s)) return;
  f_cell_fill_boundary(f, b, s.x, s.y, s.z);
}

__global__ void k_f_zero_invalid(double* __restrict__ f, Box3 b) {
  GIdx s;
  if (!grown_index(b, s)) return;
  f_cell_zero_invalid(f, b, s.x, s.y, s.z);
}

__global__ void k_f_sum_from_fine(const double* __restrict__ fnow, double* __restrict__ cnext,
                                  Coupling c) {
  // coarse cells of coarsen(fine valid) grown by one
  const int ex = c.fb.n[0] / 2 + 2, ey = c.fb.n[1] / 2 + 2, ez = c.fb.n[2] / 2 + 2;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)ex * ey * ez) return;
  const int rx = (int)(t % ex), ry = (int)((t / ex) % ey), rz = (int)(t / ((long long)ex * ey));
  f_cell_sum_from_fine(fnow, cnext, c, rx, ry, rz);
}

inline unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }
// cells of coarsen(patch) grown by one (interior and ring)
inline long long grown_coarse_cells(const Box3& fb) {
  return (long long)(fb.n[0] / 2 + 2) * (fb.n[1] / 2 + 2) * (fb.n[2] / 2 + 2);
}

}  // namespace

// threads of a block over ring cells: one warp, to reach every SM
constexpr int kRingThreads = 32;
// f(index type) with int where every element index of the boxes fits in 31
// bits: the kernels here are bound by instructions and latency, and 64-bit
// element offsets took a third of the instructions of a patch step
template <typename F>
static void with_index(bool narrow, F f) {
  if (narrow)
    f(int{});
  else
    f((long long)0);
}

template <typename T>
cudaError_t launch_explode(const T* coarse, T* fine, const Coupling& c, double om_s, double om_b,
                           double rho0, cudaStream_t st, bool paired) {
  const unsigned grid = blocks_for(ghost_cells_of(c.fb), 128);
  const DfRates r = quiet(rates_of<T>(om_s, om_b));
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    using I = decltype(i);
    if (sizeof(T) == 8 && paired)
      chained(k_explode<T, sizeof(T) == 8, I>, grid, 128, st, coarse, fine, c, (T)om_s, (T)om_b, (T)rho0, r);
    else
      chained(k_explode<T, false, I>, grid, 128, st, coarse, fine, c, (T)om_s, (T)om_b, (T)rho0, r);
  });
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_step_patch(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                              double om_b, double rho0, cudaStream_t st, bool paired,
                              const unsigned* moving) {
  const bool cov = covered.hi[0] >= covered.lo[0] && covered.hi[1] >= covered.lo[1] &&
                   covered.hi[2] >= covered.lo[2];
  const CellLaunch rl = grown_launch(b, 128);
  const DfRates r = quiet(rates_of<T>(om_s, om_b));
  with_index(index32(b), [&](auto i) {
    using I = decltype(i);
    constexpr bool P = sizeof(T) == 8;
    const T ts = (T)om_s, tb = (T)om_b, t0 = (T)rho0;
    if (P && paired && cov)
      chained(k_step_patch<T, true, P, I>, rl.grid, rl.block, st, fin, fout, b, covered, ts, tb, t0, r, moving);
    else if (P && paired)
      chained(k_step_patch<T, false, P, I>, rl.grid, rl.block, st, fin, fout, b, covered, ts, tb, t0, r, moving);
    else if (cov)
      chained(k_step_patch<T, true, false, I>, rl.grid, rl.block, st, fin, fout, b, covered, ts, tb, t0, r, moving);
    else
      chained(k_step_patch<T, false, false, I>, rl.grid, rl.block, st, fin, fout, b, covered, ts, tb, t0, r, moving);
  });
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_coalesce(const T* fine, T* coarse, const Coupling& c, double rho0,
                            cudaStream_t st) {
  const dim3 grid(blocks_for(ring_cells_of(c), 128), NV);
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    chained(k_coalesce<T, decltype(i)>, grid, 128, st, fine, coarse, c, (T)rho0);
  });
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_restrict(const T* fine, T* coarse, const Coupling& c, cudaStream_t st) {
  const long long n = (long long)(c.fb.n[0] / 2) * (c.fb.n[1] / 2) * (c.fb.n[2] / 2);
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    k_restrict<T, decltype(i)><<<dim3(blocks_for(n, 128), NV), 128, 0, st>>>(fine, coarse, c);
  });
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_explode_resc(const T* cprev, const T* cnow, T* fine, const Coupling& c,
                                double om_s, double om_b, double rho0, double wp, double wn,
                                cudaStream_t st, bool paired, const unsigned* moving) {
  const int threads = sizeof(T) == 8 ? kRingThreads : 128;
  const unsigned grid =
      blocks_for(sizeof(T) == 8 ? ring_cells_of(c) : ghost_cells_of(c.fb), threads);
  const DfRates r = quiet(rates_of<T>(om_s, om_b));
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    using I = decltype(i);
    if (sizeof(T) == 8 && paired)
      chained(k_explode_resc<T, sizeof(T) == 8, I>, grid, threads, st, cprev, cnow, fine, c, (T)om_s, (T)om_b, (T)rho0, (T)wp, (T)wn, r, moving);
    else
      chained(k_explode_resc<T, false, I>, grid, threads, st, cprev, cnow, fine, c, (T)om_s, (T)om_b,
                                                        (T)rho0, (T)wp, (T)wn, r, moving);
  });
  return cudaGetLastError();
}

template <typename T, bool COVER, bool PAIRED, bool RESC>
static void step_explode(const T* fin, T* fout, const Box3& b, const IBox& cov, double om_s,
                         double om_b, double rho0, T* fine, const Coupling& c, double es, double eb,
                         cudaStream_t st, const unsigned* moving) {
  const unsigned first = blocks_for(ghost_cells_of(c.fb), 128);
  const unsigned cells = blocks_for((long long)b.n[0] * b.n[1] * b.n[2], 128);
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    chained(k_step_explode<T, COVER, PAIRED, decltype(i), RESC>, first + cells, 128, st, fin, fout, b,
            cov, (T)om_s, (T)om_b, (T)rho0, quiet(rates_of<T>(om_s, om_b)), fine, c, (T)es, (T)eb,
            quiet(rates_of<T>(es, eb)), first, moving);
  });
}
template <typename T>
cudaError_t launch_step_explode(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                                double om_b, double rho0, T* fine, const Coupling& c, bool rescaled,
                                double es, double eb, cudaStream_t st, bool paired,
                                const unsigned* moving) {
  constexpr bool P = sizeof(T) == 8;
  if (rescaled && P && paired)
    step_explode<T, false, P, true>(fin, fout, b, covered, om_s, om_b, rho0, fine, c, es, eb, st, moving);
  else if (rescaled)
    step_explode<T, false, false, true>(fin, fout, b, covered, om_s, om_b, rho0, fine, c, es, eb, st, moving);
  else if (P && paired)
    step_explode<T, true, P, false>(fin, fout, b, covered, om_s, om_b, rho0, fine, c, es, eb, st, moving);
  else
    step_explode<T, true, false, false>(fin, fout, b, covered, om_s, om_b, rho0, fine, c, es, eb, st, moving);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_restrict_resc(const T* fine, T* coarse, const Coupling& c, double om_s,
                                 double om_b, double rho0, cudaStream_t st, bool paired,
                                 unsigned* moving) {
  const long long n = (long long)(c.fb.n[0] / 2) * (c.fb.n[1] / 2) * (c.fb.n[2] / 2);
  const DfRates r = quiet(rates_of<T>(om_s, om_b));
  const bool few = n < (sizeof(T) == 8 ? kFewCells : 2 * kFewCells);
  const unsigned grid = blocks_for(n, few ? kMeanCells : 128);
  with_index(index32(c.cb) && index32(c.fb), [&](auto i) {
    using I = decltype(i);
    auto go = [&](auto pairs) {
      constexpr bool P = decltype(pairs)::value;
      chained(few ? k_restrict_resc_few<T, P, I> : k_restrict_resc<T, P, I>, grid,
              few ? kMeanCells * kMeanWarps : 128, st, fine, coarse, c, (T)om_s, (T)om_b, (T)rho0, r,
              moving);
    };
    if (sizeof(T) == 8 && paired)
      go(std::integral_constant<bool, sizeof(T) == 8>());
    else
      go(std::false_type());
  });
  return cudaGetLastError();
}

cudaError_t launch_moving(const double* f, const Box3& b, unsigned* moving, cudaStream_t st) {
  const long long n = (long long)((b.n[0] + 3) / 4) * ((b.n[1] + 3) / 4) * ((b.n[2] + 3) / 4);
  chained(k_moving, blocks_for(n, 128), 128, st, f, b, moving);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_fill_from_coarse(const T* coarse, T* fine, const Coupling& c, cudaStream_t st) {
  const CellLaunch rl = grown_launch(c.fb, 128);
  k_fill_from_coarse<T><<<rl.grid, rl.block, 0, st>>>(coarse, fine, c);
  return cudaGetLastError();
}

#define LBX_INST(T)                                                                            \
  template cudaError_t launch_explode<T>(const T*, T*, const Coupling&, double, double, double, \
                                         cudaStream_t, bool);                                  \
  template cudaError_t launch_step_patch<T>(const T*, T*, const Box3&, IBox, double, double,   \
                                            double, cudaStream_t, bool, const unsigned*);      \
  template cudaError_t launch_step_explode<T>(const T*, T*, const Box3&, IBox, double, double, \
                                              double, T*, const Coupling&, bool, double,       \
                                              double, cudaStream_t, bool, const unsigned*);    \
  template cudaError_t launch_coalesce<T>(const T*, T*, const Coupling&, double, cudaStream_t); \
  template cudaError_t launch_restrict<T>(const T*, T*, const Coupling&, cudaStream_t);        \
  template cudaError_t launch_fill_from_coarse<T>(const T*, T*, const Coupling&, cudaStream_t); \
  template cudaError_t launch_explode_resc<T>(const T*, const T*, T*, const Coupling&, double,   \
                                              double, double, double, double, cudaStream_t,     \
                                              bool, const unsigned*);                           \
  template cudaError_t launch_restrict_resc<T>(const T*, T*, const Coupling&, double, double,   \
                                               double, cudaStream_t, bool, unsigned*);
LBX_INST(double)
LBX_INST(float)
#undef LBX_INST

cudaError_t launch_f_fill_single(const double* src, double* dst, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = grown_launch(b, 128);
  k_f_fill_single<<<rl.grid, rl.block, 0, st>>>(src, dst, b);
  return cudaGetLastError();
}
cudaError_t launch_f_fill_two(const double* fine_now, double* dst, const double* coarse_now,
                              const Coupling& c, const int* fdom, cudaStream_t st) {
  const CellLaunch rl = grown_launch(c.fb, 128);
  k_f_fill_two<<<rl.grid, rl.block, 0, st>>>(fine_now, dst, coarse_now, c, fdom[0],
                                                         fdom[1], fdom[2]);
  return cudaGetLastError();
}
cudaError_t launch_f_zero_ring0(double* f, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = grown_launch(b, 128);
  k_f_zero_ring0<<<rl.grid, rl.block, 0, st>>>(f, b);
  return cudaGetLastError();
}
cudaError_t launch_f_collide(double* f, const Box3& b, IBox covered, double om_s, double om_b,
                             cudaStream_t st, bool paired) {
  const DfRates r = quiet(df_rates(om_s, om_b));
  const long long cells = (long long)b.n[0] * b.n[1] * b.n[2];
  const CellLaunch rl = cell_launch(b, 128);
  if (paired && b.n[0] > 32 && cells < (1 << 16)) {  // so y and z are within a grid's limits
    const int bx = std::min((b.n[0] + 31) / 32 * 32, 128), by = 128 / bx;
    const dim3 grid((b.n[0] + bx - 1) / bx, (b.n[1] + by - 1) / by, b.n[2]);
    k_f_collide<true, true><<<grid, dim3(bx, by, 1), 0, st>>>(f, b, covered, om_s, om_b, r);
  } else if (paired) {
    k_f_collide<true><<<rl.grid, rl.block, 0, st>>>(f, b, covered, om_s, om_b, r);
  } else {
    k_f_collide<false><<<rl.grid, rl.block, 0, st>>>(f, b, covered, om_s, om_b, r);
  }
  return cudaGetLastError();
}
cudaError_t launch_f_stream(const double* src, double* dst, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = grown_launch(b, 128);
  k_f_stream<<<rl.grid, rl.block, 0, st>>>(src, dst, b);
  return cudaGetLastError();
}
cudaError_t launch_f_fill_boundary(double* f, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = grown_launch(b, 128);
  k_f_fill_boundary<<<rl.grid, rl.block, 0, st>>>(f, b);
  return cudaGetLastError();
}
cudaError_t launch_f_zero_invalid(double* f, const Box3& b, cudaStream_t st) {
  const CellLaunch rl = grown_launch(b, 128);
  k_f_zero_invalid<<<rl.grid, rl.block, 0, st>>>(f, b);
  return cudaGetLastError();
}
cudaError_t launch_f_sum_from_fine(const double* fine_now, double* coarse_next, const Coupling& c,
                                   cudaStream_t st) {
  k_f_sum_from_fine<<<blocks_for(grown_coarse_cells(c.fb), 128), 128, 0, st>>>(fine_now, coarse_next, c);
  return cudaGetLastError();
}

}  // namespace lbx
