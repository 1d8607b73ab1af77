// Float32 heat stage kernel for piecewise-constant face states (the centred
// diffusion scheme): residual (heat.py:354-473) + Runge-Kutta stage in one
// pass with few instructions per cell.
//
// With piecewise-constant faces the face flux is the mean of the two cell
// fluxes phi_a = -k dT/dx_a (centred, zero in ghost cells, heat.py:85-95), so
//   rhs = q - [ A1+ (phi1_i + phi1_i+1) - A1- (phi1_i-1 + phi1_i)
//             + A2+ (phi2_j + phi2_j+1) - A2- (phi2_j-1 + phi2_j)
//             + A3  (phi3_k+1 - phi3_k-1) ]
// with A_a+- = S_a(face +-1/2) / (2 V) and phi_a = g_a (U_+1 - U_-1),
// g_a = -k / (2 rho cp L_a) (T = U / (rho cp), heat.py:74).  Every grid metric
// is a product of per-axis factors (geometry.py:37-171), so the A and g of a
// cell column are formed once per tile in registers; only 1/dx3 of the plane
// varies along the z-march.
//
// Written out per cell, each direction is three products of a coefficient and a
// difference d_a = U_+1 - U_-1 at the cell and its two neighbours, so every
// coefficient is formed once per tile column and the differences are shared:
//   x1: a1+ g(i+1) d(i+1) + (a1+ - a1-) g(i) d(i) - a1- g(i-1) d(i-1), and x2 alike.
//
// Tile: 32 columns x TY = NW*VX rows.  A thread owns VX consecutive columns of
// one row and reads the TMA ring (tile + 2 halo, planes K..K+2) with VX-wide
// loads: own, left and right group, the four neighbour rows and the plane above,
// 8 wide loads per VX cells; with one column and four rows per thread (10 loads
// per cell, 2 barriers a plane) a 192x256x128 stage took 37.7 us, this takes
// 24.5.  phi3 of planes K-1 and K stay in registers; one block barrier a plane.
#pragma once
#include "stage_heat.cuh"

namespace fvm {

template <int VX>
struct alignas(VX * 4) FloatVec {
  float v[VX];
};
template <int VX>
__device__ __forceinline__ FloatVec<VX> vload(const float* p) {
  return *reinterpret_cast<const FloatVec<VX>*>(p);
}

template <int VX, int NW>
struct HeatPcCfg {
  static constexpr int TX = 32, TY = VX * NW, NT = 32 * NW, HH = 2;
  static constexpr int W = 40;  // ring column c <-> tile x offset c - 4
  static constexpr int ROWS = TY + 2 * HH, PL = ROWS * W;
  static constexpr int NSLOT = 6;  // planes K..K+2 in use, K+3..K+5 in flight
  static constexpr int SLOT = round_up(PL, 32);
  static constexpr int BYTES = NSLOT * SLOT * 4 + NSLOT * 8;
  static constexpr unsigned TX_BYTES = PL * 4;
  static_assert((SLOT * 4) % 128 == 0, "TMA destinations need 128-byte alignment");
};

// One piece of the stage (a run of planes of one tile column) with the ring
// barriers `bars` (phase bits 0..5); `phase_bits` and `pending` carry over from
// piece to piece.  Returns false when a wait ran out: the block must stop and drain.
template <int COORD, int VX, int NW>
__device__ __forceinline__ bool heat_pc_tile(const HeatParams<float>& p, const CUtensorMap* tmap, const Piece& pc,
                                             unsigned char* smem_raw, uint64_t* bars, unsigned& phase_bits,
                                             unsigned& pending) {
  using C = HeatPcCfg<VX, NW>;
  using V = FloatVec<VX>;
  constexpr int TX = C::TX, TY = C::TY, W = C::W, HH = C::HH, LX = TX / VX;  // LX lanes per row
  float* uring = reinterpret_cast<float*>(smem_raw);
  const int tid = threadIdx.x;
  const Layout& L = p.lay;
  const Metric<float>& m = p.met;
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const float qsrc = float(p.q);
  const StripCoef sc(p.coef, float(*p.dt));
  const float gk = -0.5f * float(p.k * p.inv_rho_cp);  // phi = gk / L * (U_+1 - U_-1)
  const bool need_u0 = needs_u0<float>(p.coef) && !p.coef.u0_is_input;
  const bool need_acc = needs_acc(p.coef);
  const int w = tid >> 5, lane = tid & 31;
  const int x0 = (pc.col % p.ntx) * TX, y0 = (pc.col / p.ntx) * TY;
  const int Z0 = 1 + pc.u0, Zl = pc.u1;
  const int Kfirst = Z0 - 2, Plast = Zl + 2;
  const int ty = w * VX + lane / LX, tx = (lane % LX) * VX;
  const int i0 = x0 + tx, j = y0 + ty;

  int next_pl = Kfirst;  // the next plane to issue (thread 0)
  auto issue_to = [&](int last) {
    for (; next_pl <= last && next_pl <= Plast; ++next_pl) {
      const int s = pmod(next_pl, C::NSLOT);
      pending |= 1u << s;
      fence_proxy_async();
      mbar_arrive_expect_tx(&bars[s], C::TX_BYTES + p.extra_tx);
      tma_load_4d(&uring[s * C::SLOT], tmap, &bars[s], x0 - 3 + L.padx, y0 + 1 - HH, next_pl, 0);
    }
  };
  if (tid == 0) issue_to(Kfirst + C::NSLOT - 1);

  // coefficients of the own cells (clamped indices in lanes outside the grid;
  // zero where a neighbour is a ghost cell: phi is zero-padded there)
  const int jc = min(j, ny - 1);
  auto gx = [&](int i) { return i >= 0 && i < nx ? gk * __ldg(m.inv_dx1 + i) : 0.f; };
  auto gy = [&](int jj) { return jj >= 0 && jj < ny ? gk * __ldg(m.inv_dx2 + jj) : 0.f; };
  const float ic2 = COORD == COORD_SPH ? rcp_newton(__ldg(m.c2 + jc)) : 1.f;
  float cxm[VX], cx0[VX], cxp[VX], cy[VX], cz[VX];
#pragma unroll
  for (int c = 0; c < VX; ++c) {
    const int ic = min(i0 + c, nx - 1);
    ColMetric<COORD> cm;
    cm.load(m, ic);
    const float c1 = COORD == COORD_CART ? 1.f : cm.c1;
    cxp[c] = 0.5f * cm.a1p * gx(i0 + c + 1);
    cxm[c] = -0.5f * cm.a1m * gx(i0 + c - 1);
    cx0[c] = cm.d1 * gx(ic);
    cy[c] = 0.5f * c1 * (COORD == COORD_CART ? 1.f : cm.ir);
    cz[c] = 0.5f * gk;
    if constexpr (COORD == COORD_SPH)
      cz[c] *= (c1 * __ldg(m.dx2 + jc)) * ic2 * (cm.ir * __ldg(m.inv_sin_c2 + jc));
  }
  // S2 / V without its column factor, at the upper and lower x2 face
  float pu, pl_;
  if constexpr (COORD == COORD_SPH) {
    pu = __ldg(m.sin_f2 + jc + 1) * ic2;
    pl_ = __ldg(m.sin_f2 + jc) * ic2;
  } else {
    pu = pl_ = __ldg(m.inv_dx2 + jc);
  }
  const float cyp = pu * gy(j + 1), cy0 = (pu - pl_) * gy(jc), cym = -pl_ * gy(j - 1);

  const int o = (ty + HH) * W + tx + 4;
  auto ring = [&](int pl) { return uring + pmod(pl, C::NSLOT) * C::SLOT; };
  auto wait_planes = [&](int first, int last) {
    bool got = true;
    for (int pl = first; pl <= last; ++pl) {
      const int s = pmod(pl, C::NSLOT);
      const bool g = got && mbar_wait_bounded(&bars[s], (phase_bits >> s) & 1u, p.wait_ns);
      if (g) {
        phase_bits ^= 1u << s;
        if (tid == 0) pending &= ~(1u << s);
      }
      got = g;
    }
    if (!__syncthreads_and(got)) {
      if (tid == 0) atomicOr(p.status, ST_TMA_TIMEOUT);
      return false;
    }
    return true;
  };
  // 1/dx3 of ghosted plane P, zero on a ghost plane
  auto idz_of = [&](int P) { return P <= 0 || P >= nz + 1 ? 0.f : __ldg(m.inv_dx3 + P - 1); };
  V ph0, ph1;  // d3 / dx3 of planes K-1 and K
  if (!wait_planes(Kfirst, Kfirst + 3)) return false;
  {
    const V um = vload<VX>(ring(Z0 - 2) + o), u0 = vload<VX>(ring(Z0 - 1) + o), u1 = vload<VX>(ring(Z0) + o),
            u2 = vload<VX>(ring(Z0 + 1) + o);
    const float za = idz_of(Z0 - 1), zb = idz_of(Z0);
#pragma unroll
    for (int c = 0; c < VX; ++c) {
      ph0.v[c] = za * (u1.v[c] - um.v[c]);
      ph1.v[c] = zb * (u2.v[c] - u0.v[c]);
    }
  }
  const bool in_y = j < ny, full = i0 + VX <= nx;
  for (int K = Z0, sK = pmod(Z0, C::NSLOT); K <= Zl; ++K, sK = (sK == C::NSLOT - 1 ? 0 : sK + 1)) {
    // U0 / acc of the own cells, before anything is stored in this step (rows
    // are padded to whole 16-byte groups, so the wide load stays in its row)
    V u0v, accv;
    const long long g = L.idx(0, K, j + 1, i0 + 1);
    const bool in = in_y && i0 < nx;
    if (in && need_u0) u0v = vload<VX>(p.u0 + g);
    if (in && need_acc) accv = vload<VX>(p.acc + g);
    if (!wait_planes(K + 2, K + 2)) return false;
    // every thread has left step K-1: its slot (on the first step, both planes
    // below Z0) takes the next copies
    if (tid == 0) issue_to(K + C::NSLOT - 1);
    const int s2 = sK + 2 >= C::NSLOT ? sK + 2 - C::NSLOT : sK + 2;
    const float* uK = uring + sK * C::SLOT + o;
    const V uc = vload<VX>(uK), up = vload<VX>(uring + s2 * C::SLOT + o);
    float ux[VX + 4];  // columns i0-2 .. i0+VX+1
    {
      const V l = vload<VX>(uK - VX), r = vload<VX>(uK + VX);
      ux[0] = l.v[VX - 2];
      ux[1] = l.v[VX - 1];
#pragma unroll
      for (int c = 0; c < VX; ++c) ux[2 + c] = uc.v[c];
      ux[VX + 2] = r.v[0];
      ux[VX + 3] = r.v[1];
    }
    float d[VX + 2];  // x1 differences at columns i0-1 .. i0+VX
#pragma unroll
    for (int c = 0; c < VX + 2; ++c) d[c] = ux[c + 2] - ux[c];
    const V r1 = vload<VX>(uK + W), r2 = vload<VX>(uK + 2 * W), l1 = vload<VX>(uK - W), l2 = vload<VX>(uK - 2 * W);
    const float idz = __ldg(m.inv_dx3 + (K - 1)), idz1 = idz_of(K + 1);
    float out[VX], ac[VX];
    bool fin = true;
#pragma unroll
    for (int c = 0; c < VX; ++c) {
      float div = fmaf(cxp[c], d[c + 2], fmaf(cx0[c], d[c + 1], cxm[c] * d[c]));
      const float dy = fmaf(cyp, r2.v[c] - uc.v[c], fmaf(cy0, r1.v[c] - l1.v[c], cym * (uc.v[c] - l2.v[c])));
      div = fmaf(cy[c], dy, div);
      const float ph2 = idz1 * (up.v[c] - uc.v[c]);
      div = fmaf(cz[c] * idz, ph2 - ph0.v[c], div);
      ph0.v[c] = ph1.v[c];
      ph1.v[c] = ph2;
      const float k = qsrc - div, b = need_u0 ? u0v.v[c] : uc.v[c], a = need_acc ? accv.v[c] : 0.f;
      out[c] = sc.combine(k, uc.v[c], b, a);
      ac[c] = sc.acc(k, b, a);
      if (i0 + c < nx) fin = fin && isfinite(out[c]);
    }
    if (in) {
      if (full) {
        V ov;
#pragma unroll
        for (int c = 0; c < VX; ++c) ov.v[c] = out[c];
        *reinterpret_cast<V*>(p.out + g) = ov;
        if (p.coef.accmode != ACC_NONE) {
#pragma unroll
          for (int c = 0; c < VX; ++c) ov.v[c] = ac[c];
          *reinterpret_cast<V*>(p.acc + g) = ov;
        }
      } else {
#pragma unroll
        for (int c = 0; c < VX; ++c)
          if (i0 + c < nx) {
            p.out[g + c] = out[c];
            if (p.coef.accmode != ACC_NONE) p.acc[g + c] = ac[c];
          }
      }
      if (!fin) atomicOr(p.status, ST_NONFINITE);
    }
  }
  __syncthreads();  // the next piece's first copies reuse every slot
  return true;
}

template <int COORD, int VX, int NW>
__global__ void __launch_bounds__(HeatPcCfg<VX, NW>::NT)
    heat_pc_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ HeatParams<float> p) {
  using C = HeatPcCfg<VX, NW>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + C::NSLOT * C::SLOT * 4);
  if (smem_u32(smem_raw) & 127u) {
    if (threadIdx.x == 0) atomicOr(p.status, ST_TMA_TIMEOUT);
    return;
  }
  if (p.active && !*p.active) return;  // the clock passed t_end
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int s = 0; s < C::NSLOT; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmap);
  }
  __syncthreads();
  unsigned phase_bits = 0, pending = 0;
  const OneGrid<HeatParams<float>> grid{p};
  TileWalk<OneGrid<HeatParams<float>>> walk(grid);
  Piece pc;
  int inst;
  bool ok = true;
  while (ok && walk.next(grid, inst, pc)) ok = heat_pc_tile<COORD, VX, NW>(p, &tmap, pc, smem_raw, bars, phase_bits, pending);
  if (!ok && tid == 0)
    for (int s = 0; s < C::NSLOT; ++s)
      if ((pending >> s) & 1u) mbar_wait_bounded(&bars[s], (phase_bits >> s) & 1u, p.drain_ns);
}

}  // namespace fvm
