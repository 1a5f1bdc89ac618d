// kernels.cuh -- launchers of the device kernels of liblbx_cuda.so.
// All launchers are asynchronous on `st` and return cudaGetLastError().
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "d3q15.cuh"

namespace lbx {

// An axis-aligned box of cells in storage-valid coordinates (0..n-1 of the
// valid region); empty when hi < lo in any direction.
struct IBox {
  int lo[3], hi[3];
  __host__ __device__ bool contains(int x, int y, int z) const {
    return x >= lo[0] && x <= hi[0] && y >= lo[1] && y <= hi[1] && z >= lo[2] && z <= hi[2];
  }
};
inline IBox empty_ibox() { return IBox{{0, 0, 0}, {-1, -1, -1}}; }

// Launch shape of a kernel over the valid cells of a box in storage order: one
// thread a cell, whatever the extents (rows padded to warps left 22 % of the
// lanes idle at 100 or 104 cells, 16 % at 161).  Neighbouring threads have
// neighbouring addresses across the ends of rows too, as the cells do.  A box
// that would not give every other SM a block gets smaller blocks (10x10x50 in
// blocks of 32: FP64 2.38 us a step against 2.46, FP32 1.60 against 1.79; with
// the line at 152 or 304 blocks 32^3 FP32 took 2.06 us instead of 1.85).
struct CellLaunch {
  dim3 grid, block;
};
inline CellLaunch cell_launch(const Box3& b, int threads) {
  const double n = (double)b.n[0] * b.n[1] * b.n[2];
  while (threads > 32 && n < 76.0 * threads) threads /= 2;
  const double blocks = std::ceil(n / threads);  // past a grid's limit: refused by the launch
  return CellLaunch{dim3(blocks < 4294967295.0 ? (unsigned)blocks : 4294967295u), dim3((unsigned)threads)};
}
// Whether the cells of a box are numbered in 32 bits.  The simulations and the
// batch engine refuse larger boxes; the steps, the equilibrium and the fields on
// device pointers take them.
inline bool cells32(const Box3& b) { return (double)b.n[0] * b.n[1] * b.n[2] < 2147483648.0; }
// (x, y, z) of valid cell c in storage order, false beyond the last one; 64-bit
// numbers (C) take the place of Box3's multipliers, which hold below 2^31
template <typename C>
__host__ __device__ __forceinline__ bool cell_coords(const Box3& b, C c, int& x, int& y, int& z) {
  if constexpr (sizeof(C) == 4) {
    z = (int)divide(c, b.plane);
    const uint32_t p = c - (uint32_t)z * (uint32_t)(b.n[0] * b.n[1]);
    y = (int)divide(p, b.row);
    x = (int)(p - (uint32_t)y * (uint32_t)b.n[0]);
    return z < b.n[2];
  } else {
    const C row = (C)b.n[0], plane = row * (C)b.n[1], q = c / plane, p = c - q * plane;
    if (q >= (C)b.n[2]) return false;
    z = (int)q;
    y = (int)(p / row);
    x = (int)(p - (C)y * row);
    return true;
  }
}
// whether every element index of a store fits in 31 bits (512^3 does)
inline bool index32(const Box3& b) { return (long long)NV * b.sq < (1ll << 31); }
#ifdef __CUDACC__
// (x, y, z) of this thread's cell under cell_launch (its first block being
// block `first` of the grid); false beyond the last one
template <typename C = uint32_t>
__device__ __forceinline__ bool cell_xyz(const Box3& b, int& x, int& y, int& z, unsigned first = 0) {
  return cell_coords<C>(b, (C)(blockIdx.x - first) * blockDim.x + threadIdx.x, x, y, z);
}
#endif

// ---- single box, fully periodic over its valid region -------------------
// One fused collide + push-stream step (now <- S(C(now))).  Cells inside
// `covered` are inactive: they emit zero populations (f = 0).
// paired: FP64 store with the collision carried in pairs of FP32 values
// (df32.cuh); ignored for the FP32 store.  refined: the level of a refined run
// (collide_f64 and collides_in_pairs say what differs).
template <typename T>
cudaError_t launch_step_periodic(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                                 double om_b, double rho0, cudaStream_t st, bool paired = false,
                                 bool refined = false);

// compensated sum of x[0..n) into out4[0] (out4[1..3] = 0); partials holds
// kReduceBlocks x 8 doubles
cudaError_t launch_sum(const double* x, size_t n, double* partials, double* out4, cudaStream_t st);
// p[0..n) = v
cudaError_t launch_fill(double* p, size_t n, double v, cudaStream_t st);

// C-order user vectors (rho_c, u_c) -> FAB-order rho, u (nz <= 65535*128,
// ny and nx <= 65535).
cudaError_t launch_c_to_fab(const double* rho_c, const double* u_c, double* rho, double* u,
                            int nx, int ny, int nz, cudaStream_t st);

// Equilibrium of rho = 1 + amplitude on the plane coord[axis] == index and
// u = 0 (a request of the serving loop), shifted by rho0.
template <typename T>
cudaError_t launch_init_pulse(T* f, const Box3& b, int axis, int index, double amplitude,
                              double rho0, cudaStream_t st);

// Equilibrium of the valid region from double rho[k][j][i], u[n][k][j][i].
template <typename T>
cudaError_t launch_equilibrium(const double* rho, const double* u, T* f, const Box3& b,
                               double rho0, cudaStream_t st);
// rho, u (double, FAB order) of the valid region; gather = the store holds
// post-collision populations of a periodic box (pull form) and the
// streamed state is read through the neighbours.
template <typename T>
cudaError_t launch_hydro(const T* f, const Box3& b, double rho0, double* rho, double* u,
                         cudaStream_t st, bool gather = false);
// Cells to refine by density (solution-driven tagging): over an FP64
// density field in FAB order of extents n[3], the cells with
// |rho - ref| > threshold; box6 (device, int[6]) receives the bounding box
// (lo x,y,z then hi x,y,z; to be initialised to n / -1) and count (device)
// how many.  Blocks of 256 threads over rows of x.
cudaError_t launch_tag_density(const double* rho, const int* n, double ref, double threshold,
                               int* box6, unsigned long long* count, cudaStream_t st);
// valid region <-> packed FAB order in the storage type (raw values)
template <typename T>
cudaError_t launch_pack(const T* f, const Box3& b, T* out, cudaStream_t st);
template <typename T>
cudaError_t launch_unpack(const T* in, T* f, const Box3& b, cudaStream_t st);
// valid region <-> FP64 FAB order
template <typename T>
cudaError_t launch_copy_out(const T* f, const Box3& b, double rho0, double* out, cudaStream_t st,
                            bool gather = false);

// ---- pull form of a periodic box: the store holds Q_n = C(R_{n-1}) -----
// one step Q -> C(S(Q)); paired selects the paired-FP32 collision (FP64 store)
template <typename T>
cudaError_t launch_step_pull(const T* fin, T* fout, const Box3& b, double om_s, double om_b,
                             double rho0, bool paired, cudaStream_t st);
// the same step with CalcHydroVars fused in: rho, u of the state the step
// gathers (what launch_hydro with gather gives) are written on the way
template <typename T>
cudaError_t launch_step_pull_hydro(const T* fin, T* fout, const Box3& b, double om_s, double om_b,
                                   double rho0, bool paired, double* rho, double* u,
                                   cudaStream_t st);
// R -> Q = S^-1(R) into fout (entering the form)
template <typename T>
cudaError_t launch_unstream(const T* fin, T* fout, const Box3& b, cudaStream_t st);
// Q -> S(Q) = R into fout (leaving the form)
template <typename T>
cudaError_t launch_stream_gather(const T* fin, T* fout, const Box3& b, cudaStream_t st);
template <typename T>
cudaError_t launch_copy_in(const double* in, T* f, const Box3& b, double rho0, cudaStream_t st);

// Compensated FP64 sums over the valid region minus `skip`:
// out4 = {sum f, sum cx f, sum cy f, sum cz f}.  `partials` must hold
// reduce_partials_doubles() doubles; the kernels write every entry they read.
constexpr int kReduceBlocks = 512;  // at most; the launches use three per SM
constexpr int kReduceThreads = 256;
inline size_t reduce_partials_doubles() { return (size_t)kReduceBlocks * 8; }
template <typename T>
cudaError_t launch_reduce(const T* f, const Box3& b, IBox skip, double rho0, double* partials,
                          double* out4, cudaStream_t st);

// ---- conservative two-level coupling ------------------------------------
// Geometry of a fine patch relative to its parent.  Global coordinates of
// level L are 0..N_L-1; storage-valid coordinate s maps to global lo + s.
struct Coupling {
  Box3 cb;        // coarse storage
  int clo[3];     // global coordinates of the coarse valid origin
  int cdom[3];    // coarse domain extents (periodic wrap of parent indices)
  int cper;       // 1 if the coarse level is the periodic level 0
  Box3 fb;        // fine storage (ghost width 2)
  int flo[3];     // global coordinates of the fine valid origin
};
// fine ghost shell <- coarse post-collision populations heading into the patch
// (paired: FP64 store, collision in paired FP32 as in launch_step_periodic)
template <typename T>
cudaError_t launch_explode(const T* coarse, T* fine, const Coupling& c, double om_s,
                           double om_b, double rho0, cudaStream_t st, bool paired = false);
// fused step of a patch level: valid cells collide (covered ones emit zero),
// ghost cells stream raw, populations leaving the storage are dropped.
template <typename T>
cudaError_t launch_step_patch(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                              double om_b, double rho0, cudaStream_t st, bool paired = false,
                              const unsigned* moving = nullptr);
// coarse ring cells += volume-weighted populations that left the patch
template <typename T>
cudaError_t launch_coalesce(const T* fine, T* coarse, const Coupling& c, double rho0,
                            cudaStream_t st);
// covered coarse cells <- mean of their eight children
template <typename T>
cudaError_t launch_restrict(const T* fine, T* coarse, const Coupling& c, cudaStream_t st);
// ---- rescaled coupling ------------------------------------------------------
// fine ghost shell <- parents collided at the explosion rates (om_s, om_b),
// wp x (coarse at the start of the coarse step) + wn x (coarse at its end)
template <typename T>
cudaError_t launch_explode_resc(const T* cprev, const T* cnow, T* fine, const Coupling& c,
                                double om_s, double om_b, double rho0, double wp, double wn,
                                cudaStream_t st, bool paired = false,
                                const unsigned* moving = nullptr);
// Both at once: the step of a periodic level (launch_step_periodic, refined) and
// the explosion onto the level above it of the state the step starts from
// (launch_explode, or with rescaled launch_explode_resc at wp = 1, wn = 0 and
// the rates es, eb)
template <typename T>
cudaError_t launch_step_explode(const T* fin, T* fout, const Box3& b, IBox covered, double om_s,
                                double om_b, double rho0, T* fine, const Coupling& c, bool rescaled,
                                double es, double eb, cudaStream_t st, bool paired = false,
                                const unsigned* moving = nullptr);
// covered coarse cells <- mean of their children collided at the restriction rates
template <typename T>
cudaError_t launch_restrict_resc(const T* fine, T* coarse, const Coupling& c, double om_s,
                                 double om_b, double rho0, cudaStream_t st, bool paired = false,
                                 unsigned* moving = nullptr);
// FP64: sets *moving where the valid cells of a finer level are not all at rest
// (a look at every fourth along each axis); the other launches read it, the
// restriction onto level 0 clears it for the next step
cudaError_t launch_moving(const double* f, const Box3& b, unsigned* moving, cudaStream_t st);
// level creation: fine grown box <- parent coarse cell (piecewise constant)
template <typename T>
cudaError_t launch_fill_from_coarse(const T* coarse, T* fine, const Coupling& c,
                                    cudaStream_t st);

// ---- reference-faithful Rohde cycle (FP64, ghost width 2 everywhere) ------
// FillPatchSingleLevel of the periodic level 0: every storage cell of dst
// <- the periodic image in src's valid region.
cudaError_t launch_f_fill_single(const double* src, double* dst, const Box3& b,
                                 cudaStream_t st);
// FillPatchTwoLevels + PCInterp: fine now where it (or a periodic image)
// exists, otherwise the parent cell of coarse now.  fdom = fine domain.
cudaError_t launch_f_fill_two(const double* fine_now, double* dst, const double* coarse_now,
                              const Coupling& c, const int* fdom, cudaStream_t st);
cudaError_t launch_f_zero_ring0(double* f, const Box3& b, cudaStream_t st);
cudaError_t launch_f_collide(double* f, const Box3& b, IBox covered, double om_s, double om_b,
                             cudaStream_t st, bool paired = false);
// pull stream over valid + 1 ring into a zeroed buffer
cudaError_t launch_f_stream(const double* src, double* dst, const Box3& b, cudaStream_t st);
cudaError_t launch_f_fill_boundary(double* f, const Box3& b, cudaStream_t st);
cudaError_t launch_f_zero_invalid(double* f, const Box3& b, cudaStream_t st);
// coarse next += mean of 2^3 fine blocks over the coarsened fine box grown by
// one, through every periodic image (sum_fine_to_coarse, FabArrayBase::ADD)
cudaError_t launch_f_sum_from_fine(const double* fine_now, double* coarse_next,
                                   const Coupling& c, cudaStream_t st);

}  // namespace lbx
