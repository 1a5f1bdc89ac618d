// fx64.cuh -- the FP64 collision of d3q15.cuh (collide<double>) in 64-bit
// fixed point on the integer pipe.
//
// GB300 issues about 1.9 FP64 instructions per clock per SM against 64
// integer ones, so the collision's 128 FP64 instructions take 67 clocks of an
// SM per cell where the 240 bytes of the step take 10.  Here a cell's
// populations are brought to one exponent (block fixed point: the largest has
// its leading bit at bit 57), every sum is an exact 64-bit integer addition,
// every product keeps the upper 64 bits of 128, and each result is rounded to
// FP64 once, to nearest even.
//
// Accuracy.  One unit is 2^-59 of rho or less; populations down to a 32nd of
// the largest convert exactly, smaller ones are cut at one unit.  The
// roundings inside are of one unit each, below half an ulp of every output
// (2^-57 rho for the axes, 2^-60 rho for the diagonals, which are formed at
// eight times their value), so a collision's error is that of rounding its
// results: over 2e5 random cells the largest error against the collision in
// 113-bit arithmetic is 0.70, 0.67 and 1.7 ulp of the rest, axis and diagonal
// populations (rms 0.29, 0.29, 0.35), against 6.0, 4.1 and 12 (rms 1.08, 0.96,
// 1.65) with FP64 instructions; a cell's mass changes by 1.3e-17 rms, against
// 1.1e-16.
//
// Measured on one GB300: 192^3, 40 steps with the readout, 13.2 ms against
// 63.1 ms with FP64 instructions (12.3 since the step is held to 64 registers);
// 10x10x50, 100 steps, 0.56 ms against 1.19 ms (0.28 in chained launches; a
// warp's FP64 instructions alone took 1.1 us of each step).
//
// Range.  Cells that the fixed point cannot hold (a negative, infinite or NaN
// population, a largest one outside 2^-950..2^1000, |u_a| above 1/4, density
// out of proportion to the largest population, rates outside (-1, 3)) are
// left to collide<double>; an empty population (+0) is fine.
#pragma once
#include <cmath>
#include <cstdint>

#include "bits.cuh"
#include "d3q15.cuh"

namespace lbx {

// A factor c as two signed 32-bit digits of round(c 2^63) or round(c 2^64):
// hi 2^32 + lo with lo in [-2^31, 2^31).
struct FxDigits {
  int hi, lo;
};

// (omega - 1) / 2 of the two rates in units of 2^-63; ok = 0: the rates are
// outside the range of the fixed-point collision (or were not given); quiet:
// cells at rest are left to the FP64 instructions (collide_f64)
struct FxRates {
  FxDigits s, b;
  int ok, quiet;
};

inline FxDigits fx_digits_host(int64_t v) {
  const int lo = (int)(uint32_t)(uint64_t)v;
  return FxDigits{(int)((v - lo) / (int64_t(1) << 32)), lo};
}
inline FxRates fx_rates(double om_s, double om_b) {
  FxRates r{{0, 0}, {0, 0}, 0, 0};
  const double om[2] = {om_s, om_b};
  FxDigits d[2];
  for (int k = 0; k < 2; ++k) {
    if (!(om[k] > -0.99 && om[k] < 2.99)) return r;
    // (om - 1) 2^62, with om - 2 (exact there) from om = 2 on
    const bool high = om[k] >= 2.0;
    const int64_t t = std::llrint(std::ldexp(high ? om[k] - 2.0 : om[k], 62));
    d[k] = fx_digits_host(high ? t + (int64_t(1) << 62) : t - (int64_t(1) << 62));
  }
  r.s = d[0];
  r.b = d[1];
  r.ok = 1;
  return r;
}

__host__ __device__ __forceinline__ uint64_t fx_shr(uint64_t v, uint32_t s) {  // 0 from s = 64 on
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
#else
  return s > 63 ? 0 : v >> s;
#endif
}
// position of the leading one bit of a nonzero word
__host__ __device__ __forceinline__ uint32_t fx_lead(uint32_t v) {
#ifdef __CUDA_ARCH__
  uint32_t p;
  asm("bfind.u32 %0, %1;" : "=r"(p) : "r"(v));
  return p;
#else
  return 31u - (uint32_t)__builtin_clz(v);
#endif
}
__host__ __device__ __forceinline__ uint32_t fx_umax(uint32_t a, uint32_t b) { return a > b ? a : b; }
__host__ __device__ __forceinline__ int fx_min(int a, int b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ int64_t fx_from_words(uint32_t hi, uint32_t lo) {
  return (int64_t)(((uint64_t)hi << 32) | lo);
}
// twice v, as an addition (no signed shift)
__host__ __device__ __forceinline__ int64_t fx_dbl(int64_t v) { return v + v; }

__host__ __device__ __forceinline__ FxDigits fx_digits(int64_t v) {
  return FxDigits{(int)(uint32_t)((uint64_t)(v + 0x80000000ll) >> 32), (int)(uint32_t)(uint64_t)v};
}
// a b / 2^64 rounded, for |a| < 2^62 and |b| < 2^63: with signed low digits
// the product of the two low ones is at most a quarter of a unit, of either
// sign, and is left out
__host__ __device__ __forceinline__ int64_t fx_mul(FxDigits a, FxDigits b) {
  int64_t c = (int64_t)a.hi * b.lo + 0x80000000ll;
  c += (int64_t)a.lo * b.hi;
  return (int64_t)a.hi * b.hi + (c >> 32);
}
__host__ __device__ __forceinline__ int64_t fx_mul(int64_t a, FxDigits b) {
  return fx_mul(fx_digits(a), b);
}

// 2^121 / rho for rho in [2^58, 2^61): an FP32 reciprocal of the upper word
// (relative error below 2^-21) and one step of the series
// 1/rho = x0 (1 + e + e^2 + ...), e = 1 - rho x0 (Newton's iteration with its
// second-order term), all in integers; relative error below 2^-56
__host__ __device__ __forceinline__ int64_t fx_inverse(int64_t rho) {
  const uint32_t rh = (uint32_t)((uint64_t)rho >> 32), rl = (uint32_t)rho;
  const uint32_t x0 = (uint32_t)f2i(rcp_approx(u2f(rh)) * 0x1p57f);  // 2^89 / rho, to 2^31 - 1
  const int64_t y = (int64_t)(((uint64_t)x0 * rl >> 32) + (uint64_t)x0 * rh);  // rho x0 / 2^32
  const int64_t e = (int64_t(1) << 57) - y;                                    // |e| < 2^36
  const int eh = (int)(e >> 6);
  const int64_t c = e + (((int64_t)eh * eh) >> 45);
  const int64_t k = c * 128;
  const int64_t d = (int64_t)(int)x0 * (int)(k >> 32) + (int64_t)((uint64_t)x0 * (uint32_t)k >> 32);
  return (int64_t)((uint64_t)x0 << 32) + d;
}

// v units, leading bit of v at 2^p, as FP64: `ex` is the exponent field of
// 2^32 units less 1 (the field of a value with leading bit 32 + p is ex + p + 1)
__host__ __device__ __forceinline__ double fx_to_f64(int64_t v, int ex) {  // v >= 2^32
  const uint32_t h = (uint32_t)((uint64_t)v >> 32);
  const uint32_t p = fx_lead(h);
  uint64_t t = (uint64_t)v << (30u - p);  // leading bit at 62
  t += 0x1ffu + (((uint32_t)t >> 10) & 1u);  // to nearest even at bit 10
  t >>= 10;
  return d_from_words((uint32_t)(t >> 32) + ((uint32_t)(ex + (int)p) << 20), (uint32_t)t);
}
// the same with the conversion instruction, which the FP64 pipe executes: two of
// a cell's fifteen keep that pipe, idle otherwise, and the integer pipe both busy
// (192^3: 276.4 -> 273.6 us a step, rescaled 104x88x72 138.6 -> 136.3; four: 270.2
// and 134.9, but 10x10x50 2.37 -> 2.44; all fifteen: 302 and 137.7)
__host__ __device__ __forceinline__ double fx_to_f64_fp64(int64_t v, int ex) {
#ifdef __CUDA_ARCH__
  const double d = __ll2double_rn(v);
  return __hiloint2double(__double2hiint(d) + ((ex - 1054) << 20), __double2loint(d));
#else
  return fx_to_f64(v, ex);
#endif
}
// the same for every v (zero, negative, small)
__host__ __device__ __forceinline__ double fx_to_f64_any(int64_t v, int ex) {
  const uint64_t m = v < 0 ? 0ull - (uint64_t)v : (uint64_t)v;
  if (m == 0) return 0.0;
  double r;
  if (m >> 32) {
    r = fx_to_f64((int64_t)m, ex);
  } else {  // 32 bits fit the significand: exact
    const uint32_t p = fx_lead((uint32_t)m);
    const uint64_t t = m << (52u - p);
    r = d_from_words((uint32_t)(t >> 32) + ((uint32_t)(ex - 32 + (int)p) << 20), (uint32_t)t);
  }
  return v < 0 ? -r : r;
}

// Populations of one cell in units of 2^-57 of the power of two of exponent
// field E: population = (2^52 | significand) 2^(e - E + 5) units, e its
// exponent field.  The largest has its leading bit at 57 (58 where it is one
// power above E); a sign bit, an infinity or a NaN has to be excluded by the
// caller.
__host__ __device__ __forceinline__ int64_t fx_unit(uint32_t h, uint32_t l, uint32_t base) {
  const uint64_t m = ((uint64_t)((h << 11) | (l >> 21) | 0x80000000u) << 32) | (l << 11);
  return (int64_t)fx_shr(m, (base - h) >> 20);
}
__host__ __device__ __forceinline__ uint32_t fx_base(uint32_t E) { return ((E + 6u) << 20) | 0xfffffu; }
// largest high word of a cell: a sign bit, an infinity or a NaN makes it large
__host__ __device__ __forceinline__ uint32_t fx_top(const uint32_t* h) {
  uint32_t top = h[0];
#pragma unroll
  for (int q = 1; q < NV; ++q) top = fx_umax(top, h[q]);
  return top;
}
__host__ __device__ __forceinline__ bool fx_top_ok(uint32_t top) {
  return top - (73u << 20) < (1950u << 20);
}

// sums of one cell's populations g (units): pair sums and differences and
// what the collision and the hydrodynamic fields form from them
struct FxSums {
  int64_t s1, s3, s5, D, A, rho, jx, jy, jz, Q1, Q2, Q3, Q4;
};
__host__ __device__ __forceinline__ FxSums fx_sums(const int64_t* g) {
  FxSums m;
  m.s1 = g[1] + g[2];
  m.s3 = g[3] + g[4];
  m.s5 = g[5] + g[6];
  const int64_t s7 = g[7] + g[14], d7 = g[7] - g[14];
  const int64_t s8 = g[8] + g[13], d8 = g[8] - g[13];
  const int64_t s9 = g[9] + g[12], d9 = g[9] - g[12];
  const int64_t sA = g[10] + g[11], dA = g[10] - g[11];
  m.Q1 = s7 + s8;
  m.Q2 = s9 + sA;
  m.Q3 = s7 - s8;
  m.Q4 = s9 - sA;
  m.D = m.Q1 + m.Q2;
  m.A = m.s1 + m.s3 + m.s5;
  m.rho = g[0] + m.A + m.D;
  const int64_t P1 = d7 + d8, P2 = d9 + dA, P3 = d7 - d8, P4 = d9 - dA;
  m.jx = (g[1] - g[2]) + P1 + P2;
  m.jy = (g[3] - g[4]) + P1 - P2;
  m.jz = (g[5] - g[6]) + P3 + P4;
  return m;
}

// |momenta| and |differences of the stresses| all below 2^15 units (2^-44 of
// the density): a fluid at rest but for the last bits
__host__ __device__ __forceinline__ bool fx_at_rest(const FxSums& m) {
  const int64_t v[8] = {m.jx, m.jy, m.jz, m.s1 - m.s3, m.s3 - m.s5, m.Q1 - m.Q2, m.Q3 + m.Q4, m.Q3 - m.Q4};
  uint64_t any = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) any |= (uint64_t)(v[k] + 0x8000) >> 16;
  return any == 0;
}

// In-place collision; returns false, f untouched, where the cell is left to
// collide<double>.
template <bool QUIET = false>
__host__ __device__ __forceinline__ bool collide_fx(double* f, const FxRates& r) {
  uint32_t h[NV], l[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) d_words(f[q], &h[q], &l[q]);
  const uint32_t top = fx_top(h);
  bool ok = (r.ok != 0) & fx_top_ok(top);
  const int E = (int)(top >> 20);
  const uint32_t base = fx_base(top >> 20);
  int64_t g[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) g[q] = fx_unit(h[q], l[q], base);
  const FxSums m = fx_sums(g);
  const int64_t s1 = m.s1, s3 = m.s3, s5 = m.s5, D = m.D, A = m.A, rho = m.rho;
  const int64_t jx = m.jx, jy = m.jy, jz = m.jz;
  const int64_t Q1 = m.Q1, Q2 = m.Q2, Q3 = m.Q3, Q4 = m.Q4;
  const int64_t sxy = Q1 - Q2, sxz = Q3 + Q4, syz = Q3 - Q4;
  const int64_t TrS = fx_dbl(D) - g[0];  // trace of the stress: 3 D + A - rho
  {
    // rho in [2^58.3, 2^60.5), |j_a| <= rho / 4 and D <= rho / 2 keep every
    // value below 2^63 at any rates in (-1, 3): the largest, a diagonal
    // output at eight times its value, stays below 4.9 rho
    const int rh = (int)(rho >> 32), q4 = rh >> 2;
    ok = ok & ((uint32_t)(rh - 0x05000000) < 0x11a09e66u);
    const int jh[3] = {(int)(jx >> 32), (int)(jy >> 32), (int)(jz >> 32)};
#pragma unroll
    for (int a = 0; a < 3; ++a) ok = ok & ((uint32_t)(jh[a] + q4) < (uint32_t)(2 * q4));
    ok = ok & ((int)(D >> 32) < 2 * q4);
  }
  if (QUIET) ok = ok & !(r.quiet != 0 && fx_at_rest(m));
  if (!ok) return false;

  // u_a in units of 2^-63: j_a 2^63 / rho
  const FxDigits inv = fx_digits(fx_inverse(rho));
  const FxDigits dx = fx_digits(jx), dy = fx_digits(jy), dz = fx_digits(jz);
  const FxDigits ux = fx_digits(fx_mul(dx, inv) * 64), uy = fx_digits(fx_mul(dy, inv) * 64),
                 uz = fx_digits(fx_mul(dz, inv) * 64);
  // halves of rho u_a u_b, and below halves of the moments m_ab
  const int64_t Nxx = fx_mul(dx, ux), Nyy = fx_mul(dy, uy), Nzz = fx_mul(dz, uz);
  const int64_t Nxy = fx_mul(dx, uy), Nxz = fx_mul(dx, uz), Nyz = fx_mul(dy, uz);
  const FxDigits third{0x55555555, 0x55555555}, fifteenth{0x11111111, 0x11111111};
  const FxDigits ninth{0x1c71c71c, 0x71c71c72};
  const int64_t ruu = Nxx + Nyy + Nzz;
  const int64_t c15 = fx_mul(ruu, fifteenth);
  // m = neq + (omega - 1)(neq - s): half of it is n + 2 [(omega - 1) / 2] [(2 n - s) / 2]
  const int64_t T3 =
      fx_mul(ruu + fx_dbl(fx_mul(fx_dbl(ruu) - TrS, r.b)), third);  // a third of the relaxed trace
  const int64_t A3 = fx_mul(A, third);
  const int64_t nx = Nxx - c15, ny = Nyy - c15, nz = Nzz - c15;
  const int64_t mxx = nx + T3 + fx_dbl(fx_mul(fx_dbl(nx) - s1 + A3, r.s));
  const int64_t myy = ny + T3 + fx_dbl(fx_mul(fx_dbl(ny) - s3 + A3, r.s));
  const int64_t mzz = nz + T3 + fx_dbl(fx_mul(fx_dbl(nz) - s5 + A3, r.s));
  const int64_t mxy = Nxy + fx_dbl(fx_mul(fx_dbl(Nxy) - sxy, r.s));
  const int64_t mxz = Nxz + fx_dbl(fx_mul(fx_dbl(Nxz) - sxz, r.s));
  const int64_t myz = Nyz + fx_dbl(fx_mul(fx_dbl(Nyz) - syz, r.s));
  // back-projection: rho/9 - T'/6 = (rho - 3 T'/2) / 9 on the axes, the rest
  // population twice that, the diagonals at eight times their value
  const int64_t Tp = mxx + myy + mzz;
  const int64_t ba = fx_mul(rho - Tp - fx_dbl(Tp), ninth);
  const int64_t ex = ba + mxx, ey = ba + myy, ez = ba + mzz;
  const int64_t kx = fx_mul(dx, third), ky = fx_mul(dy, third), kz = fx_mul(dz, third);
  g[0] = fx_dbl(ba);
  g[1] = ex + kx;
  g[2] = ex - kx;
  g[3] = ey + ky;
  g[4] = ey - ky;
  g[5] = ez + kz;
  g[6] = ez - kz;
  const int64_t bd = ba + Tp;  // rho/9 + T'/3
  const int64_t R1 = mxy + mxz, R2 = mxy - mxz;
  const int64_t e7 = bd + fx_dbl(R1 + myz), e8 = bd + fx_dbl(R2 - myz);
  const int64_t e9 = bd - fx_dbl(R2 + myz), eA = bd - fx_dbl(R1 - myz);
  const int64_t S1 = kx + ky, S2 = kx - ky;
  const int64_t o7 = S1 + kz, o8 = S1 - kz, o9 = S2 + kz, oA = S2 - kz;
  g[7] = e7 + o7;
  g[14] = e7 - o7;
  g[8] = e8 + o8;
  g[13] = e8 - o8;
  g[9] = e9 + o9;
  g[12] = e9 - o9;
  g[10] = eA + oA;
  g[11] = eA - oA;
  int low = (int)(g[0] >> 32);
#pragma unroll
  for (int q = 1; q < NV; ++q) low = fx_min(low, (int)(g[q] >> 32));
  // exponent fields: 2^57 units is E
  const int xa = E - 26, xd = E - 29;
  if (low > 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q)
      f[q] = q < 2 ? fx_to_f64_fp64(g[q], xa) : fx_to_f64(g[q], q < 7 ? xa : xd);
  } else {
#pragma unroll
    for (int q = 0; q < NV; ++q) f[q] = fx_to_f64_any(g[q], q < 7 ? xa : xd);
  }
  return true;
}

// Density and velocity of one cell's FP64 populations (src/AmrSim.cpp:957-971)
// from the exact sums: the density is rounded once, u_a = j_a / rho from j_a
// rounded once and the series' inverse (relative error below 2^-56), rounded.
// The FP64 form's 45 additions and its division take 40 clocks of an SM per
// cell, against 6 for its memory traffic.
// Cells left to the caller: as the collision, with the density alone in range.
__host__ __device__ __forceinline__ bool hydro_fx(const double* f, double* rho, double* u) {
  uint32_t h[NV], l[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) d_words(f[q], &h[q], &l[q]);
  const uint32_t top = fx_top(h), base = fx_base(top >> 20);
  int64_t g[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) g[q] = fx_unit(h[q], l[q], base);
  const FxSums m = fx_sums(g);
  // rho in [2^58, 2^61): the range of the inverse
  const bool ok = fx_top_ok(top) & ((uint32_t)(m.rho >> 32) - 0x04000000u < 0x1c000000u);
  if (!ok) return false;
  *rho = fx_to_f64(m.rho, (int)(top >> 20) - 26);
  const int one = 1054;  // exponent field of 2^32 less 1: whole units
  const double inv = fx_to_f64(fx_inverse(m.rho), one - 121);
  u[0] = fx_to_f64_any(m.jx, one) * inv;
  u[1] = fx_to_f64_any(m.jy, one) * inv;
  u[2] = fx_to_f64_any(m.jz, one) * inv;
  return true;
}

// Mean of eight populations (a coarse cell's children): summed exactly and
// rounded once where all are of ordinary size and not negative.  As FP64
// additions the 15 means take 2,000 clocks of an SM per warp, more than their
// loads.  Children within 2^9 units in the last place of each other (a fluid
// at rest, see collide_f64) keep the additions, equal ones are their mean.
__host__ __device__ __forceinline__ double mean8(const double* v) {
  uint32_t h[8], l[8], top = 0, far = 0, differ = 0;
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    d_words(v[m], &h[m], &l[m]);
    top = fx_umax(top, h[m]);
    differ |= (h[m] ^ h[0]) | (l[m] ^ l[0]);
    const uint64_t d = ((uint64_t)h[m] << 32 | l[m]) - ((uint64_t)h[0] << 32 | l[0]) + 512u;
    far |= (uint32_t)(d >> 32) | ((uint32_t)d >> 10);
  }
  if (differ == 0) return v[0];
  if (fx_top_ok(top) & (far != 0)) {
    const uint32_t base = fx_base(top >> 20);
    int64_t g = 0;
#pragma unroll
    for (int m = 0; m < 8; ++m) g += fx_unit(h[m], l[m], base);
    return fx_to_f64(g, (int)(top >> 20) - 29);  // an eighth of it
  }
  return 0.125 * (((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
}
__host__ __device__ __forceinline__ float mean8(const float* v) {
  return 0.125f * (((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
}

// a/2 + b/2 where the sum leaves the ordinary range; out of line, as its
// instructions in the way cost a rescaled 104x88x72 pass 0.5 %
#ifdef __CUDACC__
static __device__ __noinline__ double halves(double a, double b) { return 0.5 * a + 0.5 * b; }
#endif
// wp a + wn b: halves as one addition and the sum's exponent lowered (the
// bits of the general form), one FP64 instruction instead of two
template <typename T>
__host__ __device__ __forceinline__ T weighted(T wp, T a, T wn, T b) {
  if constexpr (sizeof(T) == 8) {
    if (wp == T(0.5) && wn == T(0.5)) {
      const double s = a + b;
      uint32_t h, l;
      d_words(s, &h, &l);
      const uint32_t e = (h >> 20) & 2047u;
#ifdef __CUDA_ARCH__
      return e - 2u < 2044u ? d_from_words(h - 0x100000u, l) : halves(a, b);
#else
      if (e - 2u < 2044u) return d_from_words(h - 0x100000u, l);
#endif
    }
  }
  return wp * a + wn * b;
}

// |u| below 1/4 in units of 2^-62
__host__ __device__ __forceinline__ int64_t fx_velocity(uint32_t h, uint32_t l) {
  const uint64_t m = ((uint64_t)((h << 11) | (l >> 21) | 0x80000000u) << 32) | (l << 11);
  const int64_t v = (int64_t)fx_shr(m, 1024u - ((h >> 20) & 2047u));
  return (int)h < 0 ? -v : v;
}

// The equilibrium of d3q15.cuh (src/AmrSim.cpp:873-927) in fixed point: the
// velocity polynomial of each population in units of 2^-60 (exact but for the
// six products' half units), times 4/9 of the density's significand, every
// weight being 4/9 times a power of two; one rounding to FP64 follows.  Its
// FP64 form's 90 instructions take 47 clocks of an SM per cell.  Left to the
// caller: densities that are not positive and ordinary, |u_a| of 1/4 and more.
__host__ __device__ __forceinline__ bool equilibrium_fx(double rho, double ux, double uy, double uz,
                                                        double* out) {
  uint32_t hr, lr, h[3], l[3];
  d_words(rho, &hr, &lr);
  d_words(ux, &h[0], &l[0]);
  d_words(uy, &h[1], &l[1]);
  d_words(uz, &h[2], &l[2]);
  bool ok = hr - (73u << 20) < (1950u << 20);
#pragma unroll
  for (int a = 0; a < 3; ++a) ok = ok & ((h[a] & 0x7fffffffu) < (1021u << 20));
  if (!ok) return false;
  const int64_t x = fx_velocity(h[0], l[0]), y = fx_velocity(h[1], l[1]), z = fx_velocity(h[2], l[2]);
  const FxDigits dx = fx_digits(x), dy = fx_digits(y), dz = fx_digits(z);
  const int64_t xx = fx_mul(dx, dx), yy = fx_mul(dy, dy), zz = fx_mul(dz, dz);
  const int64_t xy9 = fx_mul(dx, dy) * 9, xz9 = fx_mul(dx, dz) * 9, yz9 = fx_mul(dy, dz) * 9;
  const int64_t ax = (x * 3) >> 2, ay = (y * 3) >> 2, az = (z * 3) >> 2;  // 3 u_a
  const int64_t m2 = (xx + yy + zz) * 3;                                // 3 u^2
  const int64_t one = int64_t(1) << 60;
  const int64_t r0 = one - (m2 >> 1), d0 = one + m2;
  const int64_t bx = r0 + ((xx * 9) >> 1), by = r0 + ((yy * 9) >> 1), bz = r0 + ((zz * 9) >> 1);
  // 4/9 of the significand at 2^61
  const int64_t sig = (int64_t)(((uint64_t)((hr & 0xfffffu) | 0x100000u) << 41) | ((uint64_t)lr << 9));
  const FxDigits four_ninths{0x71c71c72, (int)0xc71c71c7u};  // 8/9 of 2^63
  const FxDigits w = fx_digits(fx_mul(sig, four_ninths));
  const int e = (int)(hr >> 20);
  out[0] = fx_to_f64(fx_mul(r0, w), e - 27);
  out[1] = fx_to_f64(fx_mul(bx + ax, w), e - 28);
  out[2] = fx_to_f64(fx_mul(bx - ax, w), e - 28);
  out[3] = fx_to_f64(fx_mul(by + ay, w), e - 28);
  out[4] = fx_to_f64(fx_mul(by - ay, w), e - 28);
  out[5] = fx_to_f64(fx_mul(bz + az, w), e - 28);
  out[6] = fx_to_f64(fx_mul(bz - az, w), e - 28);
  const int64_t e7 = d0 + xy9 + (xz9 + yz9), e8 = d0 + xy9 - (xz9 + yz9);
  const int64_t e9 = d0 - xy9 + (xz9 - yz9), eA = d0 - xy9 - (xz9 - yz9);
  const int64_t o7 = ax + ay + az, o8 = ax + ay - az, o9 = ax - ay + az, oA = ax - ay - az;
  out[7] = fx_to_f64(fx_mul(e7 + o7, w), e - 31);
  out[14] = fx_to_f64(fx_mul(e7 - o7, w), e - 31);
  out[8] = fx_to_f64(fx_mul(e8 + o8, w), e - 31);
  out[13] = fx_to_f64(fx_mul(e8 - o8, w), e - 31);
  out[9] = fx_to_f64(fx_mul(e9 + o9, w), e - 31);
  out[12] = fx_to_f64(fx_mul(e9 - o9, w), e - 31);
  out[10] = fx_to_f64(fx_mul(eA + oA, w), e - 31);
  out[11] = fx_to_f64(fx_mul(eA - oA, w), e - 31);
  return true;
}
// in fixed point, or in FP64 where that does not hold the cell
__host__ __device__ __forceinline__ void equilibrium_f64(double rho, double ux, double uy, double uz,
                                                         double* out) {
  if (!equilibrium_fx(rho, ux, uy, uz, out)) equilibrium(rho, ux, uy, uz, out);
}

// x 2^k for |k| < 16, without an FP64 instruction where x is of ordinary size
__host__ __device__ __forceinline__ double times_pow2(double x, int k) {
  uint32_t h, l;
  d_words(x, &h, &l);
  if (((h >> 20) & 2047u) - 16u < 2015u) return d_from_words(h + ((uint32_t)k << 20), l);
  return x * (k > 0 ? (double)(1 << k) : 1.0 / (double)(1 << -k));
}
// collide<double> of a cell whose six axis populations are equal and whose
// eight diagonal ones are: what is left of it, with the roundings that its
// operations have as the device's compiler contracts them, so that the bits are
// its own: 14 FP64 instructions instead of 128 (powers of two change only the
// exponents; 1/9, 2/9 and 1/72, and 1/3, 1/6 and 1/24 are such multiples)
__host__ __device__ __forceinline__ void collide_rest(double* f, double om_s, double om_b) {
#ifdef __CUDA_ARCH__
  const double A = __dmul_rn(6.0, f[1]);  // rounded, not part of an FMA
#else
  const double A = 6.0 * f[1];
#endif
  const double drho = fma(8.0, f[7], f[0] + A);
  const double d = fma(-1.0 / 3.0, A, times_pow2(f[1], 1));
  const double TrS = fma(24.0, f[7], A) - drho;
  const double m = fma(fma(om_b, -TrS, TrS), 1.0 / 3.0, fma(om_s, -d, d));
  const double Tp = 3.0 * m, t9 = (1.0 / 9.0) * drho;
  const double ba = fma(-1.0 / 6.0, Tp, t9);
  const double ex = fma(0.5, m, ba);
  const double bd = times_pow2(fma(1.0 / 3.0, Tp, t9), -3);
  f[0] = times_pow2(ba, 1);
#pragma unroll
  for (int q = 1; q < NV; ++q) f[q] = q < 7 ? ex : bd;
}
// such a cell, none of its populations negative and one of them at least 2^-1022:
// the general form divides by the density, an empty cell is NaN there
__host__ __device__ __forceinline__ bool is_rest(const double* f) {
  uint32_t h[NV], l[NV], d = 0;
#pragma unroll
  for (int q = 0; q < NV; ++q) d_words(f[q], &h[q], &l[q]);
#pragma unroll
  for (int q = 2; q < NV; ++q) {
    const int t = q < 7 ? 1 : 7;
    d |= (h[q] ^ h[t]) | (l[q] ^ l[t]);
  }
  return (d == 0) & ((h[0] | h[1] | h[7]) - 0x00100000u < 0x7fe00000u);
}

// whether a cell's populations are those of a fluid at rest (fx_at_rest)
__host__ __device__ __forceinline__ bool at_rest(const double* f) {
  uint32_t h[NV], l[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) d_words(f[q], &h[q], &l[q]);
  const uint32_t top = fx_top(h);
  if (!fx_top_ok(top)) return false;
  int64_t g[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) g[q] = fx_unit(h[q], l[q], fx_base(top >> 20));
  return fx_at_rest(fx_sums(g));
}

// The FP64 collision of one cell: in fixed point, or with FP64 instructions
// where the cell or the rates are outside its range.  A host build forms the
// digits of rates that were not given here; the kernels' launchers give them.
//
// QUIET, on the levels of a refined run: a cell at rest takes the FP64
// instructions too.  The levels collide at different rates, whose roundings of
// the one rest state differ in the last bit, so that a patch which no wave has
// reached holds velocities of a few 1e-17 that are rounding alone; they stay
// what they are with FP64 instructions.  An exactly uniform cell needs 14 of
// those (238 clocks of an SM per warp, less than the fixed point's 450).
template <bool QUIET = false>
__host__ __device__ __forceinline__ void collide_f64(double* f, double om_s, double om_b,
                                                     const FxRates& r) {
#ifdef __CUDA_ARCH__
  if (collide_fx<QUIET>(f, r)) return;
#else
  if (collide_fx<QUIET>(f, r.ok ? r : fx_rates(om_s, om_b))) return;
#endif
  if (QUIET && is_rest(f))
    collide_rest(f, om_s, om_b);
  else
    collide<double>(f, om_s, om_b, 0.0);
}

}  // namespace lbx
