// Shared device code for the fused finite-volume stage kernels (sm_100a).
//
// Device layout of a state buffer (one allocation per state, structure of
// arrays): element (var q, ghosted plane gz, ghosted row gy, ghosted column gx)
// lives at  q*var_stride + gz*plane + gy*pitch + (gx + padx).  One ghost layer
// per side, as in the reference (navier_stokes.py:33-39).  `padx` is chosen so
// that the first interior column (gx = 1) starts on a 16-byte boundary, which
// lets a TMA box start at an aligned x coordinate and lets warps store whole
// aligned 128-byte rows.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace fvm {

// ---------------------------------------------------------------- enums ----
enum Coord : int { COORD_CART = 0, COORD_CYL = 1, COORD_SPH = 2 };
enum Limiter : int { LIM_PC = 0, LIM_MINMOD = 1, LIM_MC = 2, LIM_VANLEER = 3 };
enum Riemann : int { RIEM_RUSANOV = 0, RIEM_HLL = 1 };
// Stage epilogue modes (time_integrators.py:42-221 stage combinations).
enum StageMode : int {
  MODE_RHS = 0,    // out = k (single residual, for parity checks)
  MODE_EULER = 1,  // out = Ucur + dt*k
  MODE_AXPY = 2,   // out = U0 + (ca*dt)*k
  MODE_SSP = 3,    // out = ca*U0 + cb*(Ucur + dt*k)
  MODE_FINAL = 4   // out = U0 + (dt/6)*(acc + k)
};
enum AccMode : int { ACC_NONE = 0, ACC_SET = 1, ACC_ADD = 2 };  // acc = k | acc = acc + w*k

// Status bits written by kernels (never a trap).
enum Status : unsigned {
  ST_NONFINITE = 1u, ST_DENSITY = 2u, ST_PRESSURE = 4u, ST_DT = 8u, ST_TMA_TIMEOUT = 16u
};

// ------------------------------------------------------- grid metadata ----
// Per-axis 1D metric tables, built on the host with the reference's own
// expressions (geometry.py:37-171) in float64 and cast once to Real.
template <typename Real>
struct Metric {
  const Real* dx1;    // nx1: face differences along x1
  const Real* dx2;    // nx2
  const Real* dx3;    // nx3
  const Real* r_c;    // nx1: x1 cell centres
  const Real* r_f;    // nx1+1: x1 faces
  const Real* r_f2;   // nx1+1: x1 faces squared
  const Real* a1;     // nx1: (rf+^2 - rf-^2)/2
  const Real* b1;     // nx1: (rf+^3 - rf-^3)/3
  const Real* inv_r;  // nx1: 1/x1
  const Real* two_inv_r;  // nx1: 2/x1
  const Real* c2;     // nx2: cos(th-) - cos(th+)
  const Real* sin_f2; // nx2+1: sin(theta faces)
  const Real* sin_c2; // nx2: sin(theta centres)
  const Real* cot_c2; // nx2: 1/tan(theta centres)
  const Real* inv_dx1;   // nx1: 1/dx1  (float32 fast path)
  const Real* inv_dx2;   // nx2
  const Real* inv_dx3;   // nx3
  const Real* inv_sin_c2;  // nx2: 1/sin(theta centres)
};

struct Layout {
  int nx, ny, nz;         // interior cells
  long long pitch;        // elements per x row (>= nx+2+padx)
  long long plane;        // pitch*(ny+2)
  long long var_stride;   // >= plane*(nz+2)
  int padx;               // front pad so that gx=1 is 16-byte aligned
  __host__ __device__ long long idx(int q, int gz, int gy, int gx) const {
    return (long long)q * var_stride + (long long)gz * plane + (long long)gy * pitch + gx + padx;
  }
};

// Cell metrics (interior cell i,j,k, 0-based).  Products keep the reference's
// left-to-right order so that the float64 build reproduces NumPy bitwise.
template <typename Real, int COORD>
struct Geo {
  static __device__ __forceinline__ Real L1(const Metric<Real>& m, int i, int, int) { return __ldg(m.dx1 + i); }
  static __device__ __forceinline__ Real L2(const Metric<Real>& m, int i, int j, int) {
    if constexpr (COORD == COORD_CART) return __ldg(m.dx2 + j);
    else return __ldg(m.r_c + i) * __ldg(m.dx2 + j);
  }
  static __device__ __forceinline__ Real L3(const Metric<Real>& m, int i, int j, int k) {
    if constexpr (COORD == COORD_SPH) return (__ldg(m.r_c + i) * __ldg(m.sin_c2 + j)) * __ldg(m.dx3 + k);
    else return __ldg(m.dx3 + k);
  }
  template <int D>
  static __device__ __forceinline__ Real L(const Metric<Real>& m, int i, int j, int k) {
    if constexpr (D == 0) return L1(m, i, j, k);
    else if constexpr (D == 1) return L2(m, i, j, k);
    else return L3(m, i, j, k);
  }
  static __device__ __forceinline__ Real V(const Metric<Real>& m, int i, int j, int k) {
    if constexpr (COORD == COORD_CART) return (__ldg(m.dx1 + i) * __ldg(m.dx2 + j)) * __ldg(m.dx3 + k);
    else if constexpr (COORD == COORD_CYL) return (__ldg(m.a1 + i) * __ldg(m.dx2 + j)) * __ldg(m.dx3 + k);
    else return (__ldg(m.b1 + i) * __ldg(m.c2 + j)) * __ldg(m.dx3 + k);
  }
  // Face areas: S1 at x1-face index fi (0..nx1), S2 at x2-face fj, S3 any k.
  static __device__ __forceinline__ Real S1(const Metric<Real>& m, int fi, int j, int k) {
    if constexpr (COORD == COORD_CART) return __ldg(m.dx2 + j) * __ldg(m.dx3 + k);
    else if constexpr (COORD == COORD_CYL) return (__ldg(m.r_f + fi) * __ldg(m.dx2 + j)) * __ldg(m.dx3 + k);
    else return (__ldg(m.r_f2 + fi) * __ldg(m.c2 + j)) * __ldg(m.dx3 + k);
  }
  static __device__ __forceinline__ Real S2(const Metric<Real>& m, int i, int fj, int k) {
    if constexpr (COORD == COORD_SPH) return (__ldg(m.a1 + i) * __ldg(m.sin_f2 + fj)) * __ldg(m.dx3 + k);
    else return __ldg(m.dx1 + i) * __ldg(m.dx3 + k);
  }
  static __device__ __forceinline__ Real S3(const Metric<Real>& m, int i, int j) {
    if constexpr (COORD == COORD_CART) return __ldg(m.dx1 + i) * __ldg(m.dx2 + j);
    else return __ldg(m.a1 + i) * __ldg(m.dx2 + j);
  }
};

// 1/L_D at a cell, from the inverse tables (float32 fast path only).
template <typename Real, int COORD, int D>
__device__ __forceinline__ Real inv_len(const Metric<Real>& m, int i, int j, int k) {
  if constexpr (D == 0) return __ldg(m.inv_dx1 + i);
  else if constexpr (D == 1) {
    if constexpr (COORD == COORD_CART) return __ldg(m.inv_dx2 + j);
    else return __ldg(m.inv_r + i) * __ldg(m.inv_dx2 + j);
  } else {
    if constexpr (COORD == COORD_SPH) return (__ldg(m.inv_r + i) * __ldg(m.inv_sin_c2 + j)) * __ldg(m.inv_dx3 + k);
    else return __ldg(m.inv_dx3 + k);
  }
}

// Lame data at a cell: h[3], dl[a][b] = d_a ln h_b, d123[a] = d_a ln(h1h2h3).
template <typename Real>
struct Lame {
  Real h[3];
  Real dl[3][3];
  Real d123[3];
};
template <typename Real, int COORD>
__device__ __forceinline__ void lame_at(const Metric<Real>& m, int i, int j, Lame<Real>& L) {
  for (int a = 0; a < 3; ++a) {
    L.h[a] = Real(1);
    L.d123[a] = Real(0);
    for (int b = 0; b < 3; ++b) L.dl[a][b] = Real(0);
  }
  if constexpr (COORD == COORD_CYL) {
    Real r = __ldg(m.r_c + i), ir = __ldg(m.inv_r + i);
    L.h[1] = r;
    L.dl[0][1] = ir;
    L.d123[0] = ir;
  } else if constexpr (COORD == COORD_SPH) {
    Real r = __ldg(m.r_c + i), ir = __ldg(m.inv_r + i), cot = __ldg(m.cot_c2 + j);
    L.h[1] = r;
    L.h[2] = r * __ldg(m.sin_c2 + j);
    L.dl[0][1] = ir;
    L.dl[0][2] = ir;
    L.dl[1][2] = cot;
    L.d123[0] = __ldg(m.two_inv_r + i);
    L.d123[1] = cot;
  }
}

// The float32 build trades IEEE division/sqrt for the approximate SFU
// instructions (<= 2 ulp); the float64 build keeps the reference's exact
// operation sequence.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 1 / x of a metric factor: the approximate reciprocal and one Newton step, which
// leaves little more than the rounding of the result, at two operations (a
// correctly rounded division per column made a heat stage of short pieces 2 to 5 %
// longer).
__device__ __forceinline__ float rcp_newton(float x) {
  const float r = rcp_approx(x);
  return fmaf(fmaf(-x, r, 1.f), r, r);
}

// float32 metric factors of a cell for the register-blocked kernels, as
// products of one per-column value c1 and table entries: the divergence takes
// face areas over the cell volume, S_a / V (the x3 length cancels in S1 / V and
// S2 / V), and the curvilinear terms the three non-zero d_a ln h_b / h_a of the
// supported coordinates, la = dl01/h0, lb = dl02/h0, lc = dl12/h1.
//
// The x1 faces come as half sum and half difference of S1 / V,
//   S1+ F+ - S1- F- = V (s1 (F+ - F-) + d1 (F+ + F-)):
// with the two quotients themselves the pressure, the largest term of both
// fluxes, left a residue of their rounding, an acceleration of the column that
// stays from step to step (cylindrical 96x128x64, error after ten steps 5.55e-8,
// so 3.94e-8).
template <int COORD>
struct ColMetric {
  float a1p, a1m;  // S1 / V of the upper and lower x1 face
  float s1, d1;    // half their sum and half their difference
  float c1;        // cylindrical dx1 / a1, spherical a1 / b1
  float ir;        // 1 / r
  __device__ __forceinline__ void load(const Metric<float>& m, int i) {
    if constexpr (COORD == COORD_CART) {
      a1p = a1m = s1 = __ldg(m.inv_dx1 + i);
      d1 = c1 = ir = 0.f;
    } else if constexpr (COORD == COORD_CYL) {
      const float ia = rcp_newton(__ldg(m.a1 + i));
      a1p = __ldg(m.r_f + i + 1) * ia;
      a1m = __ldg(m.r_f + i) * ia;
      c1 = __ldg(m.dx1 + i) * ia;
      s1 = __ldg(m.inv_dx1 + i);
      d1 = 0.5f * c1;
      ir = __ldg(m.inv_r + i);
    } else {
      const float ib = rcp_newton(__ldg(m.b1 + i)), rp = __ldg(m.r_f2 + i + 1), rm = __ldg(m.r_f2 + i);
      a1p = rp * ib;
      a1m = rm * ib;
      d1 = c1 = __ldg(m.a1 + i) * ib;
      s1 = 0.5f * (rp + rm) * ib;
      ir = __ldg(m.inv_r + i);
    }
  }
  // S2 / V of cell row j at its face fj (j or j + 1)
  __device__ __forceinline__ float a2(const Metric<float>& m, int j, int fj) const {
    if constexpr (COORD == COORD_CART) return __ldg(m.inv_dx2 + j);
    else if constexpr (COORD == COORD_CYL) return c1 * __ldg(m.inv_dx2 + j);
    else return (c1 * __ldg(m.sin_f2 + fj)) * rcp_approx(__ldg(m.c2 + j));
  }
  // S3 / V at a plane with inverse length idz
  __device__ __forceinline__ float a3(const Metric<float>& m, int j, float idz) const {
    if constexpr (COORD == COORD_SPH) return ((c1 * __ldg(m.dx2 + j)) * rcp_approx(__ldg(m.c2 + j))) * idz;
    else return idz;
  }
  __device__ __forceinline__ float la() const { return ir; }
  __device__ __forceinline__ float lb() const { return COORD == COORD_SPH ? ir : 0.f; }
  __device__ __forceinline__ float lc(const Metric<float>& m, int j) const {
    return COORD == COORD_SPH ? ir * __ldg(m.cot_c2 + j) : 0.f;
  }
};

// ------------------------------------------------------- packed float32 ----
// Two float32 values in one 64-bit register, with the packed add, subtract,
// multiply and fused multiply-add of sm_100a: each half rounds as the scalar
// instruction does, and one issue slot does two cells' work.
struct F2 {
  unsigned long long v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
  __device__ __forceinline__ explicit F2(float a) : F2(a, a) {}
  __device__ __forceinline__ float lo() const { return __uint_as_float((unsigned)v); }
  __device__ __forceinline__ float hi() const { return __uint_as_float((unsigned)(v >> 32)); }
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
  return d;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return d;
}

// ------------------------------------------------------------ limiters ----
__device__ __forceinline__ float sgn(float x) { return x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f); }

// The float64 limiters give the reference's values without its float64 sign
// sums: where the signs of a and b agree (sign bits, an integer operation) the
// sign factor is +-1 or, for the three-sign test, +-1 too.
__device__ __forceinline__ bool same_sign(double a, double b) { return (__double2hiint(a) ^ __double2hiint(b)) >= 0; }
__device__ __forceinline__ double abs_min(double a, double b) { return fabs(a) < fabs(b) ? a : b; }
// slope_limiters.py:13-39
__device__ __forceinline__ double lim_minmod(double a, double b) { return same_sign(a, b) ? abs_min(a, b) : 0.0; }
// slope_limiters.py:42-73 (three-sign test divided by 3: opposite slopes keep
// a third of the sign of their sum)
__device__ __forceinline__ double lim_mc(double a, double b) {
  const double c = 0.5 * (a + b);
  const double m = fabs(abs_min(c, 2.0 * abs_min(a, b)));
  return copysign(same_sign(a, b) ? m : (1.0 / 3.0) * m, c);
}
// slope_limiters.py:76-105
__device__ __forceinline__ double lim_vanleer(double a, double b) {
  const double ab = (2.0 * a) * b, den = fabs(a) + fabs(b);
  return same_sign(a, b) && den > 0.0 ? copysign(ab / den, a) : 0.0;
}
template <int LIM>
__device__ __forceinline__ double limiter(double a, double b) {
  if constexpr (LIM == LIM_MINMOD) return lim_minmod(a, b);
  else if constexpr (LIM == LIM_MC) return lim_mc(a, b);
  else return lim_vanleer(a, b);
}
// ------------------------------------------- float32 fast arithmetic ----
template <typename R>
__device__ __forceinline__ R recip(R x) {
  if constexpr (sizeof(R) == 4) return rcp_approx(x);
  else return R(1) / x;
}
// Quotients x / y by one y.  float32: the approximate reciprocal.  float64: the
// correctly rounded reciprocal r once, then per x the product q = x r and one
// residual correction q + (x - q y) r with fused multiply-adds (Markstein 1990),
// which rounds to the quotient itself: three operations in place of a division
// of about 25 instructions.  (x or 1/y infinite gives NaN where the division
// gives infinity; such a state is already flagged.)  The float64 viscous stage
// divided 120 times per cell and 26 times by a shared denominator.
template <typename R>
struct Quot {
  R y, r;
  __device__ __forceinline__ explicit Quot(R y_) : y(y_), r(recip(y_)) {}
  __device__ __forceinline__ R operator()(R x) const {
    if constexpr (sizeof(R) == 4) return x * r;
    else {
      const R q = x * r;
      return __fma_rn(__fma_rn(-q, y, x), r, q);
    }
  }
};
// Limiters are positively homogeneous of degree one, so limiter(a/L, b/L)*L
// equals limiter(a, b); the float32 path evaluates that form directly.
__device__ __forceinline__ float flim_minmod(float a, float b) {
  return a * b > 0.f ? copysignf(fminf(fabsf(a), fabsf(b)), a) : 0.f;
}
__device__ __forceinline__ float flim_vanleer(float a, float b) {
  const float ab = a * b;
  return ab > 0.f ? 2.f * ab * rcp_approx(a + b) : 0.f;
}
__device__ __forceinline__ float flim_mc(float a, float b) {
  const float c = 0.5f * (a + b);
  const float ss = (sgn(c) + sgn(a) + sgn(b)) * (1.f / 3.f);
  return ss * fminf(fabsf(c), 2.f * fminf(fabsf(a), fabsf(b)));
}

// MUSCL slope of a cell (reconstructors.py:120-132): limiter(bwd/L, fwd/L)*L.
template <int LIM, typename R>
__device__ __forceinline__ R muscl_slope(R fm, R f0, R fp, const Quot<R>& L) {
  if constexpr (LIM == LIM_PC) return R(0);
  else if constexpr (sizeof(R) == 4) {
    const float a = f0 - fm, b = fp - f0;
    if constexpr (LIM == LIM_MINMOD) return flim_minmod(a, b);
    else if constexpr (LIM == LIM_MC) return flim_mc(a, b);
    else return flim_vanleer(a, b);
  } else {
    return limiter<LIM>(L(f0 - fm), L(fp - f0)) * L.y;
  }
}

// Device-resident time-loop scalars.
struct Clock {
  double t, t_end, dt, cfl, dt_fixed;
  long long steps;
  int active;
  unsigned long long red[2];  // running maxima (bit patterns of non-negative doubles)
};

// --------------------------------------------------------- PTX helpers ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait on an mbarrier phase: gives up after `limit_ns` and reports it.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > limit_ns) return false;
  }
  return true;
}
// TMA: 4D tiled load (x, y, z, var) into shared memory, completion on `bar`.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ------------------------------------------------------- stage epilogue ----
struct StageCoef {
  int mode, accmode;
  double ca, cb, wacc;  // mode constants (see StageMode), acc weight
  int u0_is_input;      // the stage input buffer is the step base U0 (first stage)
};

// Ask L2 for the 128-byte line holding p (the epilogue's U0/acc rows), so the
// dependent loads at the end of a z-march step hit L2 instead of DRAM.
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
// One 4-byte asynchronous copy global -> shared (completion: cp_async_wait_all
// by the issuing thread, after which the thread may read the destination).
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Combine one variable.  `k` is the residual, `ucur` the stage input, `u0`
// the step's base state, `acc` the running k-sum.  Op order follows
// time_integrators.py:47,91-103,147-159,203-221.
template <typename R>
__device__ __forceinline__ R stage_combine(const StageCoef& c, R dt, R k, R ucur, R u0, R acc) {
  switch (c.mode) {
    case MODE_RHS: return k;
    case MODE_EULER: return ucur + dt * k;
    case MODE_AXPY: return u0 + (R(c.ca) * dt) * k;
    case MODE_SSP:
      // float32: U0 + cb((Ucur - U0) + dt k), equal to ca U0 + cb (Ucur + dt k)
      // because ca + cb = 1, and exact when nothing changes (the float32
      // coefficients 1/3, 2/3 do not sum to one and would bias the totals)
      if constexpr (sizeof(R) == 4) return u0 + R(c.cb) * ((ucur - u0) + dt * k);
      else return R(c.ca) * u0 + R(c.cb) * (ucur + dt * k);
    default:
      // float32 keeps acc = U0 + (dt/6) sum_s w_s k_s (low storage: the last
      // stage reads only its input and acc); float64 keeps the k-sum and the
      // reference's summation order U0 + (dt/6)(k1 + w k2 + ... + k_last)
      if constexpr (sizeof(R) == 4) return acc + (dt / R(6)) * k;
      else return u0 + (dt / R(6)) * (acc + k);
  }
}

// stage_combine and acc_update of the float32 build with the step's constants
// formed once per launch (they are float64 in StageCoef, and dt / 6 a division):
// every mode but MODE_SSP is base + c k.
struct StripCoef {
  int mode;
  bool set;
  float c, cb, dt, w;
  __device__ __forceinline__ StripCoef(const StageCoef& s, float dt_) : mode(s.mode), set(s.accmode == ACC_SET), dt(dt_) {
    c = mode == MODE_RHS ? 1.f : (mode == MODE_AXPY ? float(s.ca) * dt : (mode == MODE_FINAL ? dt / 6.f : dt));
    cb = float(s.cb);
    w = set ? dt / 6.f : (float(s.wacc) * dt) / 6.f;
  }
  __device__ __forceinline__ float combine(float k, float ucur, float u0, float acc) const {
    if (mode == MODE_SSP) return fmaf(cb, fmaf(dt, k, ucur - u0), u0);
    const float base = mode == MODE_AXPY ? u0 : (mode == MODE_FINAL ? acc : (mode == MODE_EULER ? ucur : 0.f));
    return fmaf(c, k, base);
  }
  __device__ __forceinline__ float acc(float k, float u0, float a) const { return fmaf(w, k, set ? u0 : a); }
};

// The stage epilogue needs U0 from memory (not from the input ring)?
template <typename R>
__device__ __forceinline__ bool needs_u0(const StageCoef& c) {
  if (c.mode < MODE_AXPY) return false;
  if constexpr (sizeof(R) == 4) {
    if (c.mode == MODE_FINAL) return false;
  }
  return true;
}
__device__ __forceinline__ bool needs_acc(const StageCoef& c) {
  return c.mode == MODE_FINAL || c.accmode == ACC_ADD;
}
// New accumulator value after this stage (see stage_combine).
template <typename R>
__device__ __forceinline__ R acc_update(const StageCoef& c, R dt, R k, R u0, R acc) {
  if constexpr (sizeof(R) == 4) {
    if (c.accmode == ACC_SET) return u0 + (dt / R(6)) * k;
    return acc + ((R(c.wacc) * dt) / R(6)) * k;
  } else {
    if (c.accmode == ACC_SET) return k;
    return acc + R(c.wacc) * k;
  }
}

}  // namespace fvm
