// Float32 Navier-Stokes stage kernel with register-blocked columns, for every
// coordinate system:
// residual (navier_stokes.py:588-711) + Runge-Kutta stage combination in one
// pass, built to issue few instructions per cell.
//
// Tile: 32 columns (x1) x TY = NW*R rows (x2), marching a chunk of planes
// along x3.  Output warp w (< NW) owns the strip of R rows w*R .. w*R+R-1;
// lane l owns column l.  One more warp (the halo warp) forms, for every tile
// row, the x1 data that lies outside the warp: the slopes of the cell left of
// the tile and the flux through the tile's right edge, and the pressure of
// the tile's halo cells.
//
// Per step K (ghosted output plane K; the TMA ring holds planes K, K+1 and,
// once it has arrived, K+2):
//   1. thread 0 issues the TMA of plane K+2 into the slot that plane K-1 left,
//      and of this plane's U0 / k-accumulator tile when the stage combination
//      reads them;
//   2. x1 and x2 for plane K: x1 slopes of both rows with the left slope and the
//      right-face flux from neighbouring lanes by shuffle (lane 0 / lane 31 from
//      the halo warp's data), then x2 slopes and fluxes in registers (the strip
//      computes its three faces itself).  The halo warp meanwhile forms that data
//      for plane K+1;
//   3. every thread waits (bounded) for plane K+2;
//   4. P of plane K+2: own cells by their owners (kept in registers), halo
//      cells by the halo warp (navier_stokes.py:94-100);
//   5. x3: slope of plane K+1 at the thread's cells and the face flux at
//      K+1/2; the left state and the flux at K-1/2 are carried in registers;
//   6. divergence with the face areas over the cell volume (cartesian: the
//      inverse cell lengths), gravity and curvilinear sources, stage combination
//      with U0 / acc from shared memory, coalesced stores;
//   7. one block barrier per step (after it, plane K's slot is free).
// Face values are the reference's: MUSCL slopes limiter(f_i - f_i-1,
// f_i+1 - f_i) (zero in ghost cells, reconstructors.py:120-132), states
// f +- s/2, Euler flux from the face U and the reconstructed face P, HLL or
// Rusanov (riemann_solvers.py:13-89).  float32 arithmetic with the
// approximate reciprocal and square root; HLL's three-way choice is written
// with clamped wave speeds (s- = min(s_min, 0), s+ = max(s_max, 0)), which is
// the same function.
#pragma once
#include <cfloat>
#include "stage_ns.cuh"

namespace fvm {

template <int R, int NW>
struct NsStripCfg {
  static constexpr int TX = 32, TY = R * NW;
  static constexpr int NO = 32 * NW;  // output threads
  static constexpr int NT = NO + 32;  // + the halo warp
  static constexpr int NV = 5, NF = 6, HH = 2;
  static constexpr int W = 40;  // ring column c <-> tile x offset c - 4
  static constexpr int ROWS = TY + 2 * HH;
  static constexpr int PL = ROWS * W;
  static constexpr int NSLOT = 3;  // planes K, K+1 and K+2 (arriving)
  static constexpr int SLOT = round_up(NV * PL, 32);
  static constexpr int W2 = TX + 4, R2 = TY + 4, PL2 = W2 * R2;  // P plane: tile + 2
  static constexpr int NBORDER = 4 * W2 + 4 * TY;                 // P halo cells per plane
  static constexpr int STG = NV * TY * TX;                        // one staged U0 / acc tile
  static constexpr int OFF_U = 0;
  static constexpr int OFF_P = OFF_U + NSLOT * SLOT;
  static constexpr int OFF_HL = OFF_P + 3 * PL2;       // [parity][field][row]: slopes left of the tile
  static constexpr int OFF_FR = OFF_HL + 2 * NF * TY;  // [parity][var][row]: right-edge fluxes
  static constexpr int END = OFF_FR + 2 * NV * TY;
  static constexpr int NBAR = NSLOT + 1;               // ring slots + the staged tiles
  static constexpr int BAR_BYTES = round_up(END * 4, 8);
  static constexpr int STG_OFF_BYTES = round_up(BAR_BYTES + NBAR * 8, 128);
  static constexpr unsigned TX_BYTES = NV * PL * 4;
  static constexpr unsigned STG_BYTES = STG * 4;
  // dynamic shared memory with `nbuf` staged tiles (0: none, 1: U0 or acc, 2: both)
  static constexpr int bytes(int nbuf) { return STG_OFF_BYTES + nbuf * (int)STG_BYTES; }
  static_assert(R == 2, "the two rows of a thread's strip share packed registers");
  static_assert(2 * TY <= 32, "one halo lane per tile row and task");
  static_assert((SLOT * 4) % 128 == 0 && (STG_BYTES % 128) == 0, "TMA destinations need 128-byte alignment");
};

// Tensor maps and parameters of one launch: the ring map of the stage input
// and the maps of the U0 / accumulator buffers (box 32 x TY x 1 x 5).
struct NsStripSource {
  CUtensorMap tmap, u0map, accmap;
  NsParams<float> p;
};

// min(|a|, |b|), positive where a and b have the same sign, negative where not.
__device__ __forceinline__ float min_xorsign(float a, float b) {
  float d;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// Limited slope from the backward and forward differences (float32; zero for
// piecewise constant), up to the factor 2 strip_half<LIM>: a face state is
// f +- strip_half * strip_slope, the reference's f +- slope / 2.  The factor
// carries the constants of the limiters (slope_limiters.py:13-105).
// A ghost cell's slope is zero by one value per cell, its gate, instead of a
// select per field: the factor, zero in a ghost cell, or for van Leer the bound
// that the product of the differences has to pass, infinite in a ghost cell,
// where the product may overflow to an infinity that a zero factor would turn into
// NaN (a predicate in place of that bound: 256^3 stage 651 us, so 610).
// The kernels are bound by issue and latency: with the limiters in four to
// eleven instructions, a select per slope, flux vectors formed per state and
// float64 stage constants converted per cell, the stage launches took 717 us
// (inviscid 256^3), 1497 (viscous 256^3), 95 (97x130x61, three-sign limiter) and
// 291 (Maxwell 128x128x256); in this form 600, 1291, 54 and 200 (542, 1092, 48 and
// 186 with what the comments at strip_slope2, the flat march, the viscous and the
// Maxwell kernel say).
template <int LIM>
__host__ __device__ constexpr float strip_half() {
  return LIM == LIM_MC ? 0.25f : (LIM == LIM_VANLEER ? 1.f : 0.5f);
}
// A cell's gate, and the factor of its slope.
template <int LIM>
__device__ __forceinline__ float strip_gate(bool ghost) {
  if constexpr (LIM == LIM_VANLEER) return ghost ? __int_as_float(0x7f800000) : 0.f;
  else return ghost ? 0.f : strip_half<LIM>();
}
template <int LIM>
__device__ __forceinline__ float strip_factor(float gate) {
  if constexpr (LIM == LIM_VANLEER) return strip_half<LIM>();
  else return gate;
}
template <int LIM>
__device__ __forceinline__ float strip_slope(float a, float b, float gate = strip_gate<LIM>(false)) {
  if constexpr (LIM == LIM_PC) return 0.f;
  else if constexpr (LIM == LIM_MINMOD) return copysignf(fmaxf(min_xorsign(a, b), 0.f), a);
  else if constexpr (LIM == LIM_MC) {
    // the three-sign form: opposite slopes keep a third, with the sign of a + b
    const float s = a + b, t = min_xorsign(a, b);
    const float m = fminf(fabsf(s), fabsf(4.f * t));
    return copysignf(t > 0.f ? m : m * (1.f / 3.f), s);
  } else {
    // a b / (a + b) where a b > 0; a + b = 0 only where a b <= 0
    const float ab = a * b;
    return ab > gate ? ab * rcp_approx(a + b) : 0.f;
  }
}

// a F(qL) + b F(qR) + c (qR - qL) of the Euler flux F along axis D, with the
// normal velocities v and sound speeds c of the two states: F's terms all carry
// v, so a v and b v multiply the states directly.
template <int D, int RIEM>
__device__ __forceinline__ void strip_combine(const float* qL, const float* qR, float vL, float vR, float cL, float cR,
                                              float* F) {
  float a, b, c;
  if constexpr (RIEM == RIEM_HLL) {
    const float sl = fminf(fminf(vL - cL, vR - cR), 0.f);
    const float sr = fmaxf(fmaxf(vL + cL, vR + cR), 0.f);
    const float rd = rcp_approx(fmaxf(sr - sl, 1e-30f));
    a = sr * rd;
    b = -sl * rd;
    c = sl * a;
  } else {
    a = b = 0.5f;
    c = -0.5f * fmaxf(fabsf(vL) + cL, fabsf(vR) + cR);
  }
  const float av = a * vL, bv = b * vR;
  F[0] = fmaf(a, qL[1 + D], fmaf(b, qR[1 + D], c * (qR[0] - qL[0])));
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    // (the normal momentum with its pressure, the largest term, rounded per state:
    // adding both pressures at the end rounded the sum once more, error of five
    // steps 3.36e-8, so 3.34e-8)
    if (k == 1 + D) F[k] = fmaf(a, fmaf(vL, qL[k], qL[5]), fmaf(b, fmaf(vR, qR[k], qR[5]), c * (qR[k] - qL[k])));
    else F[k] = fmaf(av, qL[k], fmaf(bv, qR[k], c * (qR[k] - qL[k])));
  }
  F[4] = fmaf(av, qL[4] + qL[5], fmaf(bv, qR[4] + qR[5], c * (qR[4] - qL[4])));
}

// Inviscid Riemann flux along axis D from face states q = {rho, m1, m2, m3, E, P}
// (navier_stokes.py:159-214 fluxes, :280-355 wave speeds).
template <int D, int RIEM>
__device__ __forceinline__ void strip_flux(const float* qL, const float* qR, float gam, float* F) {
  const float irL = rcp_approx(qL[0]), irR = rcp_approx(qR[0]);
  const float vL = qL[1 + D] * irL, vR = qR[1 + D] * irR;
  const float cL = sqrt_approx((gam * qL[5]) * irL), cR = sqrt_approx((gam * qR[5]) * irR);
  strip_combine<D, RIEM>(qL, qR, vL, vR, cL, cR, F);
}

// strip_slope, strip_flux of two faces at once, one in each half of the packed
// registers: the kernel is bound by issue and latency, and the x1 and x3 faces of a
// strip's two rows, and two of its three x2 faces, cost their adds and multiplies
// once (837 -> 700 thread instructions per cell; 256^3 stage 575 -> 541 us,
// 97x130x61 51.6 -> 48.4, one-plane 64x64 5.99 -> 5.0).
template <int LIM>
__device__ __forceinline__ F2 strip_slope2(F2 a, F2 b, float gate) {
  return F2(strip_slope<LIM>(a.lo(), b.lo(), gate), strip_slope<LIM>(a.hi(), b.hi(), gate));
}
template <int LIM>
__device__ __forceinline__ F2 strip_state2(F2 h, F2 s, F2 q) {
  if constexpr (LIM == LIM_PC) return q;
  else return fma2(h, s, q);
}
template <int D, int RIEM, bool EARLY>
__device__ __forceinline__ void strip_flux2(const F2* qL, const F2* qR, float gam, F2* F) {
  const F2 g2(gam);
  const F2 irL(rcp_approx(qL[0].lo()), rcp_approx(qL[0].hi())), irR(rcp_approx(qR[0].lo()), rcp_approx(qR[0].hi()));
  const F2 vL = qL[1 + D] * irL, vR = qR[1 + D] * irR;
  // flux of the normal momentum: formed before the wave speeds (EARLY) or where it
  // is used, as the kernel's registers and schedule like it (ns_strip_kernel)
  auto normal = [](const F2* q, F2 v) { return fma2(v, q[1 + D], q[5]); };
  F2 nL, nR;
  if constexpr (EARLY) nL = normal(qL, vL), nR = normal(qR, vR);
  const F2 c2L = (g2 * qL[5]) * irL, c2R = (g2 * qR[5]) * irR;
  const F2 cL(sqrt_approx(c2L.lo()), sqrt_approx(c2L.hi())), cR(sqrt_approx(c2R.lo()), sqrt_approx(c2R.hi()));
  // c below is -c of strip_combine, with the states' difference turned round
  F2 a, b, c;
  if constexpr (RIEM == RIEM_HLL) {
    const F2 lL = cL - vL, lR = cR - vR, uL = vL + cL, uR = vR + cR;
    const F2 sl(fmaxf(fmaxf(lL.lo(), lR.lo()), 0.f), fmaxf(fmaxf(lL.hi(), lR.hi()), 0.f));  // -s-
    const F2 sr(fmaxf(fmaxf(uL.lo(), uR.lo()), 0.f), fmaxf(fmaxf(uL.hi(), uR.hi()), 0.f));
    const F2 dd = sr + sl;
    const F2 rd(rcp_approx(fmaxf(dd.lo(), 1e-30f)), rcp_approx(fmaxf(dd.hi(), 1e-30f)));
    a = sr * rd;
    b = sl * rd;
    c = sl * a;
  } else {
    const F2 h(0.5f);
    const F2 uL = F2(fabsf(vL.lo()), fabsf(vL.hi())) + cL, uR = F2(fabsf(vR.lo()), fabsf(vR.hi())) + cR;
    a = b = h;
    c = h * F2(fmaxf(uL.lo(), uR.lo()), fmaxf(uL.hi(), uR.hi()));
  }
  const F2 av = a * vL, bv = b * vR;
  F[0] = fma2(a, qL[1 + D], fma2(b, qR[1 + D], c * (qL[0] - qR[0])));
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    if (k == 1 + D) {
      if constexpr (!EARLY) nL = normal(qL, vL), nR = normal(qR, vR);
      F[k] = fma2(a, nL, fma2(b, nR, c * (qL[k] - qR[k])));
    } else {
      F[k] = fma2(av, qL[k], fma2(bv, qR[k], c * (qL[k] - qR[k])));
    }
  }
  F[4] = fma2(av, qL[4] + qL[5], fma2(bv, qR[4] + qR[5], c * (qL[4] - qR[4])));
}

// P = (gamma - 1)(E - |m|^2 / (2 rho)) of one ring cell (navier_stokes.py:94-100).
// Cells outside the ghosted grid hold zeros; the clamp of the reciprocal keeps
// their P, which a ghost cell's discarded slope reads, finite (a clamp of the
// density would change the pressure of thin states: in units with densities of
// 1e-31 a clamp at 1e-30 was wrong by 3 %).
__device__ __forceinline__ float strip_pressure(const float* u, int PL, float gm1) {
  const float rho = u[0], m1 = u[PL], m2 = u[2 * PL], m3 = u[3 * PL], E = u[4 * PL];
  const float ke = fmaf(m1, m1, fmaf(m2, m2, m3 * m3)) * (0.5f * fminf(rcp_approx(rho), FLT_MAX));
  return gm1 * (E - ke);
}

// Geometric source of a cell (navier_stokes.py:437-452), added to s[1..3]: q =
// {rho, m1, m2, m3, E}, pressure P and, with viscosity, the stress components
// {t11, t22, t33, t12, t13, t23} tau[0], tau[stride], ... .
template <int COORD>
__device__ __forceinline__ void curvilinear_source(const ColMetric<COORD>& cm, const Metric<float>& m, int j,
                                                   const float* q, float P, const float* tau, float* s,
                                                   int stride = 0) {
  const float ir = rcp_approx(q[0]), la = cm.la(), lb = cm.lb(), lc = cm.lc(m, j);
  const float v1 = q[1] * ir, v2 = q[2] * ir, v3 = q[3] * ir;
  float n2 = fmaf(q[2], v2, P), n3 = fmaf(q[3], v3, P), s12 = q[1] * v2, s13 = q[1] * v3, s23 = q[2] * v3;
  (void)v1;
  if (tau) {
    n2 -= tau[stride];
    n3 -= tau[2 * stride];
    s12 -= tau[3 * stride];
    s13 -= tau[4 * stride];
    s23 -= tau[5 * stride];
  }
  s[1] = fmaf(n2, la, s[1]);
  s[2] = fmaf(-s12, la, s[2]);
  if constexpr (COORD == COORD_SPH) {
    s[1] = fmaf(n3, lb, s[1]);
    s[2] = fmaf(n3, lc, s[2]);
    s[3] = fmaf(-s13, lb, fmaf(-s23, lc, s[3]));
  }
}

// One piece of the stage (a run of planes of one tile column, or of row tiles
// of a flat grid).  `bars` holds the ring
// barriers (indices 0..2, phase bits 0..2), `gbar` the staged-tile barrier with
// phase bit `gbit`; `phase_bits` and `pending` carry over from tile to tile.
// Returns false when a wait ran out: the block must stop and drain.
template <int LIM, int RIEM, int R, int NW, int COORD, bool flat, bool EARLY>
__device__ __forceinline__ bool ns_strip_tile(const NsParams<float>& p, const CUtensorMap* tmap,
                                              const CUtensorMap* u0map, const CUtensorMap* accmap, const Piece& pc,
                                              unsigned char* smem_raw, uint64_t* bars, uint64_t* gbar, int gbit,
                                              unsigned& phase_bits, unsigned& pending) {
  using C = NsStripCfg<R, NW>;
  constexpr int TX = C::TX, TY = C::TY, W = C::W, PL = C::PL, HH = C::HH, NF = C::NF, W2 = C::W2;
  constexpr int PL2 = C::PL2;
  constexpr float HS = strip_half<LIM>();
  float* sm = reinterpret_cast<float*>(smem_raw);
  float* uring = sm + C::OFF_U;
  float* pring = sm + C::OFF_P;
  float* hl = sm + C::OFF_HL;
  float* fr = sm + C::OFF_FR;
  float* gst = reinterpret_cast<float*>(smem_raw + C::STG_OFF_BYTES);
  const int tid = threadIdx.x;
  const Layout& L = p.lay;
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const float gam = float(p.gamma), gm1 = float(p.gamma) - 1.f;
  const StripCoef sc(p.coef, float(*p.dt));
  const float gx = float(p.g1), gy = float(p.g2), gz = float(p.g3);
  const bool need_u0 = needs_u0<float>(p.coef) && !p.coef.u0_is_input;
  const bool need_acc = needs_acc(p.coef);
  const unsigned stg_bytes = (need_u0 ? C::STG_BYTES : 0u) + (need_acc ? C::STG_BYTES : 0u);
  const float* gu0 = gst;                            // staged U0 tile [var][row][column]
  const float* gacc = gst + (need_u0 ? C::STG : 0);  // staged acc tile
  const int w = tid >> 5, lane = tid & 31;
  const bool is_out = w < NW;
  {
    // A one-plane grid whose x3 ghosts copy the plane ("flat") has x3 fluxes
    // that cancel exactly: plane 1 alone, no x3 pipeline.  Its piece marches
    // instead over row tiles along x2 (the steps of the march), each step's
    // plane copy issued one step ahead into the next ring slot.  A
    // template argument: with both marches in one body the hot loop spread over
    // code it jumped across, and warps waited for instructions (256^3 stage
    // 599 -> 575 us, a mixed batch's stage 340 -> 301, when they were parted).
    const int Z0 = flat ? 1 : 1 + pc.u0;  // first ghosted output plane
    const int Zl = flat ? 1 : pc.u1;      // last ghosted output plane
    const int x0 = (pc.col % p.ntx) * TX, ybase = flat ? pc.u0 * TY : (pc.col / p.ntx) * TY;
    int y0 = ybase;  // the current step's first row
    const int nsteps = pc.u1 - pc.u0;
    const int Kfirst = flat ? Z0 : Z0 - 2, Plast = flat ? Zl : Zl + HH;
    const int i = x0 + lane;
    ColMetric<COORD> cm;
    cm.load(p.met, min(i, nx - 1));

    // plane pl of the rows from yrow - HH into ring slot s
    auto issue_at = [&](int pl, int s, int yrow) {
      pending |= 1u << s;
      fence_proxy_async();
      mbar_arrive_expect_tx(&bars[s], C::TX_BYTES + p.extra_tx);
      tma_load_4d(&uring[s * C::SLOT], tmap, &bars[s], x0 - 3 + L.padx, yrow + 1 - HH, pl, 0);
    };
    auto issue = [&](int pl) { issue_at(pl, pmod(pl, C::NSLOT), y0); };
    // planes Kfirst .. Kfirst + 2 (the first step's; a flat grid's first row tile)
    if (tid == 0) {
      if (flat) issue_at(Kfirst, 0, ybase);
      else
        for (int pl = Kfirst; pl <= Kfirst + 2; ++pl) issue(pl);
    }

    // Halo warp: x1 data of plane Kh (ring plane uH, P plane pH) outside the
    // warps: lanes 0..TY-1 the slopes of the cell left of the tile, lanes
    // TY..2TY-1 the flux through the tile's right edge
    auto halo_x1 = [&](int Kh, const float* uH, const float* pH) {
      const int row = lane < TY ? lane : lane - TY;
      const int j = y0 + row;
      if (Kh >= Z0 && Kh <= Zl && lane < 2 * TY && j < ny) {
        const int hpar = Kh & 1;
        auto ldh = [&](float* f, int tx) {
          const int o = (row + HH) * W + tx + 4;
#pragma unroll
          for (int v = 0; v < 5; ++v) f[v] = uH[v * PL + o];
          f[5] = pH[(row + 2) * W2 + tx + 2];
        };
        if (lane < TY) {
          float a[NF], b[NF], c[NF];
          ldh(a, -2);
          ldh(b, -1);
          ldh(c, 0);
#pragma unroll
          for (int f = 0; f < NF; ++f)  // zero on the left ghost column
            hl[(hpar * NF + f) * TY + row] = x0 == 0 ? 0.f : strip_slope<LIM>(b[f] - a[f], c[f] - b[f]);
        } else {
          float F[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
          if (x0 + TX <= nx) {  // the face between x0 + 31 and x0 + 32 is needed
            float a[NF], b[NF], c[NF], d[NF], ql[NF], qr[NF];
            ldh(a, TX - 2);
            ldh(b, TX - 1);
            ldh(c, TX);
            ldh(d, TX + 1);
            const float g32 = strip_gate<LIM>(x0 + TX >= nx);  // x0 + 32 is the right ghost column
#pragma unroll
            for (int f = 0; f < NF; ++f) {
              ql[f] = fmaf(HS, strip_slope<LIM>(b[f] - a[f], c[f] - b[f]), b[f]);
              qr[f] = fmaf(-strip_factor<LIM>(g32), strip_slope<LIM>(c[f] - b[f], d[f] - c[f], g32), c[f]);
            }
            strip_flux<0, RIEM>(ql, qr, gam, F);
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) fr[(hpar * 5 + v) * TY + row] = F[v];
        }
      }
    };
    // Halo warp: P of ring plane usrc on the cells of the P plane no output
    // thread owns
    auto border_p = [&](float* pdst, const float* usrc) {
      for (int b = lane; b < C::NBORDER; b += 32) {
        int x, y;
        if (b < 2 * W2) {
          y = b / W2 - 2;
          x = b % W2 - 2;
        } else if (b < 4 * W2) {
          y = TY + (b - 2 * W2) / W2;
          x = (b - 2 * W2) % W2 - 2;
        } else {
          const int c = b - 4 * W2;
          y = c >> 2;
          x = (c & 3) < 2 ? (c & 3) - 2 : (c & 3) + 30;
        }
        pdst[(y + 2) * W2 + x + 2] = strip_pressure(usrc + (y + HH) * W + x + 4, PL, gm1);
      }
    };

    // x3 state carried from step to step, per own cell: the left state of the
    // face above the last slope plane and the flux of the face below the
    // output plane
    F2 qlz[NF], fzp[5];
#pragma unroll
    for (int f = 0; f < NF; ++f) qlz[f] = F2(0.f);
#pragma unroll
    for (int v = 0; v < 5; ++v) fzp[v] = F2(0.f);
    // P of plane u at the thread's two cells, into P plane pp
    auto pressure2 = [&](const float* u, float* pp) {
      const int o = (w * R + HH) * W + lane + 4, op = (w * R + 2) * W2 + lane + 2;
      const F2 P(strip_pressure(u + o, PL, gm1), strip_pressure(u + o + W, PL, gm1));
      pp[op] = P.lo();
      pp[op + W2] = P.hi();
      return P;
    };

    static_assert(C::NSLOT == 3, "the U and P rings turn together");
    int slot = flat ? 0 : pmod(Kfirst, C::NSLOT);
    const int nstep = flat ? nsteps : Zl - Kfirst + 1;
    for (int st = 0; st < nstep; ++st) {
      const int K = flat ? Kfirst : Kfirst + st;
      if (flat) y0 = ybase + st * TY;
      const int sK = slot, pK0 = flat ? 0 : slot;
      slot = slot == C::NSLOT - 1 ? 0 : slot + 1;
      const bool outstep = K >= Z0;
      const int sK1 = sK == C::NSLOT - 1 ? 0 : sK + 1, sK2 = sK1 == C::NSLOT - 1 ? 0 : sK1 + 1;
      const int pK1i = pK0 == 2 ? 0 : pK0 + 1, pK2i = pK1i == 2 ? 0 : pK1i + 1;
      const float* uK = uring + sK * C::SLOT;
      const float* uK1 = uring + sK1 * C::SLOT;
      const float* uK2 = uring + sK2 * C::SLOT;
      float* pK = pring + pK0 * PL2;
      float* pK1 = pring + pK1i * PL2;
      float* pK2 = pring + pK2i * PL2;
      // ------------------------------------------------------------ 1 ----
      if (tid == 0) {
        if (flat) {
          // the next row tile's plane, into the slot two steps back left
          if (st + 1 < nstep) issue_at(Kfirst, (st + 1) % C::NSLOT, y0 + TY);
        } else if (K > Kfirst && K + 2 <= Plast) {
          issue(K + 2);
        }
        if (outstep && stg_bytes) {
          pending |= 1u << gbit;
          fence_proxy_async();
          mbar_arrive_expect_tx(gbar, stg_bytes);
          const int gxc = x0 + 1 + L.padx;
          if (need_u0) tma_load_4d(gst, u0map, gbar, gxc, y0 + 1, K, 0);
          if (need_acc) tma_load_4d(gst + (need_u0 ? C::STG : 0), accmap, gbar, gxc, y0 + 1, K, 0);
        }
      }
      F2 kv[5];  // flux differences of the two rows
#pragma unroll
      for (int v = 0; v < 5; ++v) kv[v] = F2(0.f);
      if constexpr (flat) {
        // the plane itself, its P over the tile + 2 and the halo warp's x1
        // data, before the sweep
        const bool g = mbar_wait_bounded(&bars[sK], (phase_bits >> sK) & 1u, p.wait_ns);
        if (g) {
          phase_bits ^= 1u << sK;
          if (tid == 0) pending &= ~(1u << sK);
          if (is_out) {
            pressure2(uK, pK);
          } else {
            border_p(pK, uK);
          }
        } else {
          atomicOr(p.status, ST_TMA_TIMEOUT);
        }
        if (!__syncthreads_and(g)) return false;
        if (!is_out) halo_x1(K, uK, pK);
        __syncthreads();
      }
      // ------------------------------------------------------------ 2 ----
      if (is_out) {
        if (outstep) {
          const int par = K & 1;
          const int jb = y0 + w * R;  // first row of the strip
          auto ld = [&](int f, int ty, int tx) {
            return f < 5 ? uK[f * PL + (ty + HH) * W + tx + 4] : pK[(ty + 2) * W2 + tx + 2];
          };
          auto ld2 = [&](int f, int ty, int tx) { return F2(ld(f, ty, tx), ld(f, ty + 1, tx)); };
          const int ty = w * R;  // first row of the strip
          {
            // x1 of both rows (cells i, rows jb and jb + 1): the flux through
            // the cells' left faces, the right faces' from the next lane
            F2 qlx[NF], qrx[NF], F[5];
            const float xgate = strip_gate<LIM>(i >= nx);  // i == nx: the right ghost column
            const F2 hx(-strip_factor<LIM>(xgate));
#pragma unroll
            for (int f = 0; f < NF; ++f) {
              const F2 fm = ld2(f, ty, lane - 1), f0 = ld2(f, ty, lane), fp = ld2(f, ty, lane + 1);
              const F2 s1 = strip_slope2<LIM>(f0 - fm, fp - f0, xgate);
              const float ua = __shfl_up_sync(0xffffffffu, s1.lo(), 1), ub = __shfl_up_sync(0xffffffffu, s1.hi(), 1);
              const float* h = hl + (par * NF + f) * TY + ty;
              qlx[f] = strip_state2<LIM>(F2(HS), lane == 0 ? F2(h[0], h[1]) : F2(ua, ub), fm);
              qrx[f] = strip_state2<LIM>(hx, s1, f0);
            }
            strip_flux2<0, RIEM, EARLY>(qlx, qrx, gam, F);
#pragma unroll
            for (int v = 0; v < 5; ++v) {
              const float da = __shfl_down_sync(0xffffffffu, F[v].lo(), 1), db = __shfl_down_sync(0xffffffffu, F[v].hi(), 1);
              const float* e = fr + (par * 5 + v) * TY + ty;
              const F2 fe = lane == 31 ? F2(e[0], e[1]) : F2(da, db);
              kv[v] = (fe - F[v]) * F2(cm.s1);
              if constexpr (COORD != COORD_CART) kv[v] = fma2(fe + F[v], F2(cm.d1), kv[v]);
            }
          }
          {
            // x2: slopes of rows jb - 1 .. jb + 2 (zero in a ghost cell), the
            // faces below rows jb and jb + 1 as a pair and the one above
            F2 ql[NF], qr[NF], F[5];
            float ql1[NF], qr1[NF], F1[5];
            float ygate[4];
            float hy[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              ygate[r] = strip_gate<LIM>(jb + r - 1 < 0 || jb + r - 1 >= ny);
              hy[r] = strip_factor<LIM>(ygate[r]);
            }
#pragma unroll
            for (int f = 0; f < NF; ++f) {
              float g[6], s[4];
#pragma unroll
              for (int r = 0; r < 6; ++r) g[r] = ld(f, ty - 2 + r, lane);
#pragma unroll
              for (int r = 0; r < 4; ++r) s[r] = strip_slope<LIM>(g[r + 1] - g[r], g[r + 2] - g[r + 1], ygate[r]);
              ql[f] = strip_state2<LIM>(F2(hy[0], hy[1]), F2(s[0], s[1]), F2(g[1], g[2]));
              qr[f] = strip_state2<LIM>(F2(-hy[1], -hy[2]), F2(s[1], s[2]), F2(g[2], g[3]));
              ql1[f] = fmaf(hy[2], s[2], g[3]);
              qr1[f] = fmaf(-hy[3], s[3], g[4]);
            }
            strip_flux2<1, RIEM, EARLY>(ql, qr, gam, F);
            strip_flux<1, RIEM>(ql1, qr1, gam, F1);
            const int ja = min(jb, ny - 1), jc = min(jb + 1, ny - 1);
            const F2 lower(-cm.a2(p.met, ja, ja), -cm.a2(p.met, jc, jc));
            const F2 upper(cm.a2(p.met, ja, ja + 1), cm.a2(p.met, jc, jc + 1));
#pragma unroll
            for (int v = 0; v < 5; ++v) kv[v] = fma2(F2(F[v].hi(), F1[v]), upper, fma2(F[v], lower, kv[v]));
          }
        }
      } else {
        // --------------------------------------------------- halo warp ----
        // x1 data of plane K+1, the next output plane (a flat grid's was
        // formed before the sweep)
        if constexpr (!flat) halo_x1(K + 1, uK1, pK1);
      }
      // ------------------------------------------------------------ 3 ----
      // Every thread waits for the plane itself; nothing read after the wait
      // was written by another thread in this step, so the block needs no
      // barrier here.  A thread whose wait ran out skips the rest of the step
      // and the barrier at its end takes the block out.
      bool got = true;
      for (int pl = (flat ? K + 3 : (K == Kfirst ? Kfirst : K + 2)); pl <= K + 2; ++pl) {
        const int s = pl == K + 2 ? sK2 : pl == K + 1 ? sK1 : sK;
        const bool g = got && mbar_wait_bounded(&bars[s], (phase_bits >> s) & 1u, p.wait_ns);
        if (g) {
          phase_bits ^= 1u << s;
          if (tid == 0) pending &= ~(1u << s);
        }
        got = g;
      }
      if (!got) atomicOr(p.status, ST_TMA_TIMEOUT);
      bool step_ok = got;
      if (!got) {
        // skip to the barrier
      } else if (is_out) {
        if constexpr (!flat) {  // x3 (a flat grid has none)
          // ------------------------------------------------------------ 4 ----
          const int ty = w * R;
          const int o = (ty + HH) * W + lane + 4, op = (ty + 2) * W2 + lane + 2;
          const F2 pnew = pressure2(uK2, pK2);
          if (K == Kfirst) {
            pressure2(uK, pK);
            pressure2(uK1, pK1);
          }
          // ------------------------------------------------------------ 5 ----
          // slope of plane K+1 (zero on a ghost plane) and the flux at K+1/2
          const float zgate = strip_gate<LIM>(K + 1 <= 0 || K + 1 >= nz + 1);
          const float hz = strip_factor<LIM>(zgate);
          const bool zface = K >= Z0 - 1;
          const float idz = outstep ? __ldg(p.met.inv_dx3 + (K - 1)) : 0.f;
          F2 qr[NF], qn[NF];
#pragma unroll
          for (int f = 0; f < NF; ++f) {
            const float* b0 = f < 5 ? uK + f * PL + o : pK + op;
            const float* b1 = f < 5 ? uK1 + f * PL + o : pK1 + op;
            const int up = f < 5 ? W : W2;  // one row up
            const F2 a0(b0[0], b0[up]), a1(b1[0], b1[up]);
            const F2 a2 = f < 5 ? F2(uK2[f * PL + o], uK2[f * PL + o + W]) : pnew;
            const F2 s = strip_slope2<LIM>(a1 - a0, a2 - a1, zgate);
            qr[f] = strip_state2<LIM>(F2(-hz), s, a1);
            qn[f] = strip_state2<LIM>(F2(hz), s, a1);
          }
          if (zface) {
            F2 F[5];
            strip_flux2<2, RIEM, EARLY>(qlz, qr, gam, F);
            const F2 a3(cm.a3(p.met, min(y0 + ty, ny - 1), idz), cm.a3(p.met, min(y0 + ty + 1, ny - 1), idz));
#pragma unroll
            for (int v = 0; v < 5; ++v) {
              kv[v] = fma2(F[v] - fzp[v], a3, kv[v]);
              fzp[v] = F[v];
            }
          }
#pragma unroll
          for (int f = 0; f < NF; ++f) qlz[f] = qn[f];
        }
        // ------------------------------------------------------------ 6 ----
        if (outstep) {
          bool staged_ok = true;
          if (stg_bytes) {
            staged_ok = mbar_wait_bounded(gbar, (phase_bits >> gbit) & 1u, p.wait_ns);
            if (staged_ok) {
              phase_bits ^= 1u << gbit;
              if (tid == 0) pending &= ~(1u << gbit);
            }
          }
          step_ok = step_ok && staged_ok;
          unsigned bad = staged_ok ? 0u : ST_TMA_TIMEOUT;
          const int ty = w * R, jb = y0 + ty;
          if (i < nx && jb < ny && staged_ok) {
            const bool two = jb + 1 < ny;  // the strip's second row is inside the grid
            // where the combination reads U, U0 and the accumulator of the two
            // cells: first cell, next variable, next row
            struct Src {
              const float* q;
              int var, row;
              __device__ __forceinline__ F2 operator[](int v) const { return F2(q[v * var], q[v * var + row]); }
            };
            const Src cur{uK + (ty + HH) * W + lane + 4, PL, W};
            const Src u0 = need_u0 ? Src{gu0 + ty * TX + lane, TY * TX, TX} : cur;
            const Src ac = need_acc ? Src{gacc + ty * TX + lane, TY * TX, TX} : cur;
            const Src base = sc.mode == MODE_AXPY ? u0 : (sc.mode == MODE_FINAL ? ac : cur);
            const Src abase = sc.set ? u0 : ac;
            F2 q[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) q[v] = cur[v];
            // gravity (navier_stokes.py:499-504): rho g and rho g.v = g.m
            const F2 gx2(gx), gy2(gy), gz2(gz);
            F2 k[5];
            k[0] = F2(0.f) - kv[0];
            k[1] = q[0] * gx2 - kv[1];
            k[2] = q[0] * gy2 - kv[2];
            k[3] = q[0] * gz2 - kv[3];
            k[4] = fma2(gx2, q[1], fma2(gy2, q[2], gz2 * q[3])) - kv[4];
            if constexpr (COORD != COORD_CART) {
              float s[2][4], qs[2][5];
#pragma unroll
              for (int v = 0; v < 5; ++v) qs[0][v] = q[v].lo(), qs[1][v] = q[v].hi();
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                s[r][1] = s[r][2] = s[r][3] = 0.f;
                curvilinear_source<COORD>(cm, p.met, min(jb + r, ny - 1), qs[r], pK[(ty + r + 2) * W2 + lane + 2],
                                          nullptr, s[r]);
              }
#pragma unroll
              for (int v = 1; v < 4; ++v) k[v] = k[v] + F2(s[0][v], s[1][v]);
            }
            // (read once: a batch's parameters lie in global memory, and a load
            // between the stores would have to be repeated after each)
            const long long g = L.idx(0, K, jb + 1, i + 1), pitch = L.pitch, var_stride = L.var_stride;
            const F2 dt2(sc.dt), c2(sc.c), cb2(sc.cb), w2(sc.w);
            bool fin0 = true, fin1 = true;
            float* po = p.out + g;
            float* pa = p.acc + g;
            const bool wacc = p.coef.accmode != ACC_NONE, ssp = sc.mode == MODE_SSP, rhs = sc.mode == MODE_RHS;
#pragma unroll
            for (int v = 0; v < 5; ++v) {
              F2 o;
              if (ssp) {
                const F2 b = u0[v];
                o = fma2(cb2, fma2(dt2, k[v], q[v] - b), b);
              } else {
                o = fma2(c2, k[v], rhs ? F2(0.f) : base[v]);
              }
              po[0] = o.lo();
              if (two) po[pitch] = o.hi();
              fin0 = fin0 && isfinite(o.lo());
              fin1 = fin1 && isfinite(o.hi());
              if (v == 0 && !rhs) {
                if (!(o.lo() > 0.f) || (two && !(o.hi() > 0.f))) bad |= ST_DENSITY;
              }
              if (wacc) {
                const F2 na = fma2(w2, k[v], abase[v]);
                pa[0] = na.lo();
                if (two) pa[pitch] = na.hi();
              }
              po += var_stride;
              pa += var_stride;
            }
            if (!fin0 || (two && !fin1)) bad |= ST_NONFINITE;
          }
          if (bad) atomicOr(p.status, bad);
        }
      } else {
        // P of plane K+2 (and on the first step of K, K+1) on the cells of
        // the P plane no output thread owns
        if constexpr (!flat) {
          border_p(pK2, uK2);
          if (K == Kfirst) {
            border_p(pK, uK);
            border_p(pK1, uK1);
          }
        }
      }
      // ------------------------------------------------------------ 7 ----
      if (!__syncthreads_and(step_ok)) return false;
    }
  }
  return true;
}

template <int LIM, int RIEM, int R, int NW, int MINB, int COORD, bool FLAT>
__global__ void __launch_bounds__(NsStripCfg<R, NW>::NT, MINB)
    ns_strip_kernel(const __grid_constant__ NsStripSource src) {
  using C = NsStripCfg<R, NW>;
  // where strip_flux2 forms its normal flux, by what was measured: 256^3 HLL stage
  // 542 us early, 563 late, Rusanov 558 and 533, the one-plane march the same, grids
  // of 128^3 in the mixed-batch kernel 314 and 302
  constexpr bool EARLY = RIEM == RIEM_HLL && !FLAT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::BAR_BYTES);
  const NsParams<float>& p = src.p;
  if (smem_u32(smem_raw) & 127u) {  // TMA destinations need 128-byte alignment
    if (threadIdx.x == 0) atomicOr(p.status, ST_TMA_TIMEOUT);
    return;
  }
  if (p.active && !*p.active) return;  // the clock passed t_end: the stage is a no-op
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int s = 0; s < C::NBAR; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
    tma_prefetch_desc(&src.tmap);
    if (needs_u0<float>(p.coef) && !p.coef.u0_is_input) tma_prefetch_desc(&src.u0map);
    if (needs_acc(p.coef)) tma_prefetch_desc(&src.accmap);
  }
  __syncthreads();
  unsigned phase_bits = 0;  // expected parity per barrier (identical in the threads that wait)
  unsigned pending = 0;     // barriers with a copy in flight (thread 0)
  const OneGrid<NsParams<float>> grid{p};
  TileWalk<OneGrid<NsParams<float>>> walk(grid);
  Piece pc;
  int inst;
  bool ok = true;
  while (ok && walk.next(grid, inst, pc))
    ok = ns_strip_tile<LIM, RIEM, R, NW, COORD, FLAT, EARLY>(p, &src.tmap, &src.u0map, &src.accmap, pc, smem_raw, bars,
                                                             bars + C::NSLOT, C::NSLOT, phase_bits, pending);
  // On a timeout, wait (bounded) for every copy this block may still have in flight.
  if (!ok && tid == 0) {
    for (int s = 0; s < C::NBAR; ++s)
      if ((pending >> s) & 1u) mbar_wait_bounded(&bars[s], (phase_bits >> s) & 1u, p.drain_ns);
  }
}

}  // namespace fvm
