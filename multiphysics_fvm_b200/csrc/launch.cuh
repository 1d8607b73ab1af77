// Launch helpers for the fused stage kernels: persistent grids sized from the
// occupancy of each instantiation, runtime dispatch over the scheme enums.
#pragma once
#include <algorithm>
#include <atomic>
#include <type_traits>
#include "stage_ns.cuh"
#include "stage_ns_strip.cuh"
#include "stage_ns_strip_visc.cuh"
#include "stage_heat.cuh"
#include "stage_heat_pc.cuh"
#include "stage_batch_mixed.cuh"
#include "stage_maxwell.cuh"
#include "stage_maxwell_strip.cuh"

namespace fvm {

// Tile rows of the Navier-Stokes kernel and the blocks per SM it is built
// for: viscous 6 rows (float32 2 blocks of 256 threads, ~109 KB each; float64
// one, 215 KB: 4 rows, 6 warps per SM and twice the stress per cell took 529 us
// where 6 rows take 372, 96^3), inviscid 8 rows (float32 3 blocks; float64 one:
// two blocks of 4 rows ran the same, 177 us at 96^3 minmod).
template <typename Real, bool VISC>
constexpr int ns_tile_ty() { return VISC ? 6 : 8; }
template <typename Real, bool VISC>
constexpr int ns_min_blocks() { return std::is_same<Real, double>::value ? 1 : (VISC ? 2 : 3); }
constexpr int HEAT_TY = 8, HEAT_TY_ALT = 4;

// Resident blocks per SM of the kernel that prepare_kernel last looked at on
// this thread (of a kernel with several shared-memory sizes, its largest).
inline thread_local int prepared_blocks = 0;

// Resident blocks per SM of one kernel with each of its N shared-memory sizes.
// The launchers' are process-wide and handles may be made and stepped from
// several threads: blocks[0], written last, says that all are there.
template <int N>
struct Residency {
  std::atomic<int> blocks[N] = {};
  bool known() const { return blocks[0].load(std::memory_order_acquire) != 0; }
  long long operator[](int k) const { return blocks[k].load(std::memory_order_relaxed); }
};

// Prepare a kernel that runs with bytes[0] < bytes[1] < ... of dynamic shared
// memory: its limit goes to the largest at once, and never below what another
// thread may be launching with.
template <typename K, int N>
static cudaError_t prepare_kernel(K kern, int threads, const int (&bytes)[N], Residency<N>& res) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes[N - 1]);
  if (e != cudaSuccess) return e;
  // all of the unified L1/shared array as shared memory: the ring planes are
  // the blocks' working set, so more resident blocks beat a larger L1
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int blocks[N];
  for (int k = 0; k < N; ++k) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[k], kern, threads, bytes[k]);
    if (e != cudaSuccess) return e;
    if (blocks[k] < 1) return cudaErrorInvalidConfiguration;
  }
  for (int k = N - 1; k > 0; --k) res.blocks[k].store(blocks[k], std::memory_order_relaxed);
  res.blocks[0].store(blocks[0], std::memory_order_release);
  prepared_blocks = blocks[N - 1];
  return cudaSuccess;
}
// Blocks of a persistent launch over `ntiles` tiles.
inline int grid_blocks(long long ntiles, long long resident, int nsm) { return (int)std::min(ntiles, resident * nsm); }

// nsm < 0: only set the kernel's shared-memory attribute and query its
// occupancy (done once, outside any stream capture).
template <typename Real, int LIM, int RIEM, int COORD, bool VISC, class Src>
cudaError_t launch_ns_src(const Src& src, long long ntiles, cudaStream_t s, int nsm) {
  constexpr int TY = ns_tile_ty<Real, VISC>();
  using C = NsCfg<Real, VISC, TY>;
  auto kern = ns_stage_kernel<Real, LIM, RIEM, COORD, VISC, TY, ns_min_blocks<Real, VISC>(), Src>;
  static Residency<1> res;
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::BYTES}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  if (ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[0], nsm);
  kern<<<grid, C::NT, C::BYTES, s>>>(src);
  return cudaGetLastError();
}

// One grid: float64, the viscous float32 grids' second block shape, and single
// calls on a float32 member of a batch that runs these kernels.
template <typename Real, int LIM, int RIEM, int COORD, bool VISC>
cudaError_t launch_ns_one(const CUtensorMap& map, NsParams<Real> p, cudaStream_t s, int nsm) {
  SingleSource<NsParams<Real>> src;
  src.tmap = map;
  set_tiles(p, ns_tile_ty<Real, VISC>());
  src.p = p;
  return launch_ns_src<Real, LIM, RIEM, COORD, VISC>(src, tile_total(p), s, nsm);
}

template <typename Real, int COORD>
cudaError_t launch_ns_coord(int lim, int riem, bool visc, const CUtensorMap& map, const NsParams<Real>& p,
                            cudaStream_t s, int nsm) {
#define FVM_NS_CASE(L, R)                                                          \
  if (lim == L && riem == R)                                                       \
    return visc ? launch_ns_one<Real, L, R, COORD, true>(map, p, s, nsm)           \
                : launch_ns_one<Real, L, R, COORD, false>(map, p, s, nsm);
  FVM_NS_CASE(LIM_PC, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_PC, RIEM_HLL)
  FVM_NS_CASE(LIM_MINMOD, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_MINMOD, RIEM_HLL)
  FVM_NS_CASE(LIM_MC, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_MC, RIEM_HLL)
  FVM_NS_CASE(LIM_VANLEER, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_VANLEER, RIEM_HLL)
#undef FVM_NS_CASE
  return cudaErrorInvalidValue;
}

// Batched launch: every instance shares the kernel specialisation; the tile
// counts of each instance's params must already be filled in.
template <typename Real, int COORD>
cudaError_t launch_ns_batch_coord(int lim, int riem, bool visc, const BatchSource<NsParams<Real>>& src,
                                  long long ntiles, cudaStream_t s, int nsm) {
#define FVM_NS_CASE(L, R)                                                                                \
  if (lim == L && riem == R)                                                                             \
    return visc ? launch_ns_src<Real, L, R, COORD, true>(src, ntiles, s, nsm)                            \
                : launch_ns_src<Real, L, R, COORD, false>(src, ntiles, s, nsm);
  FVM_NS_CASE(LIM_PC, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_PC, RIEM_HLL)
  FVM_NS_CASE(LIM_MINMOD, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_MINMOD, RIEM_HLL)
  FVM_NS_CASE(LIM_MC, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_MC, RIEM_HLL)
  FVM_NS_CASE(LIM_VANLEER, RIEM_RUSANOV)
  FVM_NS_CASE(LIM_VANLEER, RIEM_HLL)
#undef FVM_NS_CASE
  return cudaErrorInvalidValue;
}

// Declarations of the per-(precision, coordinate) instantiations.
#define FVM_DECLARE_NS(REAL, COORD)                                                                      \
  extern template cudaError_t launch_ns_coord<REAL, COORD>(int, int, bool, const CUtensorMap&,          \
                                                          const NsParams<REAL>&, cudaStream_t, int);    \
  extern template cudaError_t launch_ns_batch_coord<REAL, COORD>(                                        \
      int, int, bool, const BatchSource<NsParams<REAL>>&, long long, cudaStream_t, int);
FVM_DECLARE_NS(float, COORD_CART)
FVM_DECLARE_NS(float, COORD_CYL)
FVM_DECLARE_NS(float, COORD_SPH)
FVM_DECLARE_NS(double, COORD_CART)
FVM_DECLARE_NS(double, COORD_CYL)
FVM_DECLARE_NS(double, COORD_SPH)

template <typename Real>
cudaError_t launch_ns_batch(int lim, int riem, int coord, bool visc, const BatchSource<NsParams<Real>>& src,
                            long long ntiles, cudaStream_t s, int nsm) {
  if (coord == COORD_CART) return launch_ns_batch_coord<Real, COORD_CART>(lim, riem, visc, src, ntiles, s, nsm);
  if (coord == COORD_CYL) return launch_ns_batch_coord<Real, COORD_CYL>(lim, riem, visc, src, ntiles, s, nsm);
  return launch_ns_batch_coord<Real, COORD_SPH>(lim, riem, visc, src, ntiles, s, nsm);
}

template <typename Real>
cudaError_t launch_ns(int lim, int riem, int coord, bool visc, const CUtensorMap& map, const NsParams<Real>& p,
                      cudaStream_t s, int nsm) {
  if (coord == COORD_CART) return launch_ns_coord<Real, COORD_CART>(lim, riem, visc, map, p, s, nsm);
  if (coord == COORD_CYL) return launch_ns_coord<Real, COORD_CYL>(lim, riem, visc, map, p, s, nsm);
  return launch_ns_coord<Real, COORD_SPH>(lim, riem, visc, map, p, s, nsm);
}

// ---------------------------------------------------------- float32 NS ----
// Register-blocked stage kernel (stage_ns_strip.cuh) for float32 inviscid
// grids, 2 rows per thread: TY = 8 (4 output warps, 3 blocks/SM at
// 128 registers) or 16 (8 output warps, 2 blocks/SM).
constexpr int NS_STRIP_TY = 8, NS_STRIP_TY_ALT = 16;

template <int LIM, int RIEM, int COORD, int TY, bool FLAT>
cudaError_t launch_ns_strip_ty(const NsStripSource& src, int nbuf, cudaStream_t s, int nsm) {
  constexpr int R = 2, NW = TY / R;
  using C = NsStripCfg<R, NW>;
  auto kern = ns_strip_kernel<LIM, RIEM, R, NW, TY == 8 ? 3 : 2, COORD, FLAT>;
  static Residency<3> res;  // with 0, 1 and 2 staged tiles
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::bytes(0), C::bytes(1), C::bytes(2)}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  const long long ntiles = tile_total(src.p);
  if (ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[nbuf], nsm);
  kern<<<grid, C::NT, C::bytes(nbuf), s>>>(src);
  return cudaGetLastError();
}

template <int LIM, int RIEM, int COORD>
cudaError_t launch_ns_strip_lr(NsStripSource& src, int ty, int nbuf, cudaStream_t s, int nsm) {
  NsParams<float>& p = src.p;
  set_tiles(p, ty, p.flat != 0);
  const bool alt = ty == NS_STRIP_TY_ALT;
  // (a handle prepares the march of its steps; a residual of a one-plane grid runs
  // the x3 march and prepares it on its first call)
  if (p.flat)
    return alt ? launch_ns_strip_ty<LIM, RIEM, COORD, NS_STRIP_TY_ALT, true>(src, nbuf, s, nsm)
               : launch_ns_strip_ty<LIM, RIEM, COORD, NS_STRIP_TY, true>(src, nbuf, s, nsm);
  return alt ? launch_ns_strip_ty<LIM, RIEM, COORD, NS_STRIP_TY_ALT, false>(src, nbuf, s, nsm)
             : launch_ns_strip_ty<LIM, RIEM, COORD, NS_STRIP_TY, false>(src, nbuf, s, nsm);
}

template <int COORD>
cudaError_t launch_ns_strip_coord(int lim, int riem, NsStripSource& src, int ty, int nbuf, cudaStream_t s, int nsm) {
#define FVM_STRIP_CASE(L, R) \
  if (lim == L && riem == R) return launch_ns_strip_lr<L, R, COORD>(src, ty, nbuf, s, nsm);
  FVM_STRIP_CASE(LIM_PC, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_PC, RIEM_HLL)
  FVM_STRIP_CASE(LIM_MINMOD, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_MINMOD, RIEM_HLL)
  FVM_STRIP_CASE(LIM_MC, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_MC, RIEM_HLL)
  FVM_STRIP_CASE(LIM_VANLEER, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_VANLEER, RIEM_HLL)
#undef FVM_STRIP_CASE
  return cudaErrorInvalidValue;
}
extern template cudaError_t launch_ns_strip_coord<COORD_CART>(int, int, NsStripSource&, int, int, cudaStream_t, int);
extern template cudaError_t launch_ns_strip_coord<COORD_CYL>(int, int, NsStripSource&, int, int, cudaStream_t, int);
extern template cudaError_t launch_ns_strip_coord<COORD_SPH>(int, int, NsStripSource&, int, int, cudaStream_t, int);
inline cudaError_t launch_ns_strip(int lim, int riem, int coord, NsStripSource& src, int ty, int nbuf, cudaStream_t s,
                                   int nsm) {
  return coord == COORD_CART  ? launch_ns_strip_coord<COORD_CART>(lim, riem, src, ty, nbuf, s, nsm)
         : coord == COORD_CYL ? launch_ns_strip_coord<COORD_CYL>(lim, riem, src, ty, nbuf, s, nsm)
                              : launch_ns_strip_coord<COORD_SPH>(lim, riem, src, ty, nbuf, s, nsm);
}

// Viscous float32 grids (stage_ns_strip_visc.cuh): 1 row per
// thread, TY = 7 (7 output warps + the halo warp, 2 blocks/SM: 16 warps per SM,
// 4 per scheduler, fit 128 registers without spills; 8 output warps left 96
// registers and spilled, 2-row strips held 168 and ran 8 warps per SM).  It is
// these grids' default block shape; the second one runs the general kernel
// (stage_ns.cuh).
constexpr int NS_STRIP_VISC_TY = 7;

template <int LIM, int RIEM, int COORD, int TY>
cudaError_t launch_ns_strip_visc_ty(const NsStripSource& src, int nbuf, cudaStream_t s, int nsm) {
  constexpr int R = 1, NW = TY / R;
  using C = NsStripViscCfg<R, NW>;
  auto kern = ns_strip_visc_kernel<LIM, RIEM, R, NW, 2, COORD>;
  static Residency<3> res;  // with 0, 1 and 2 staged tiles
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::bytes(0), C::bytes(1), C::bytes(2)}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  const long long ntiles = tile_total(src.p);
  if (ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[nbuf], nsm);
  kern<<<grid, C::NT, C::bytes(nbuf), s>>>(src);
  return cudaGetLastError();
}

template <int LIM, int RIEM, int COORD>
cudaError_t launch_ns_strip_visc_lr(NsStripSource& src, int ty, int nbuf, cudaStream_t s, int nsm) {
  NsParams<float>& p = src.p;
  set_tiles(p, ty);
  return launch_ns_strip_visc_ty<LIM, RIEM, COORD, NS_STRIP_VISC_TY>(src, nbuf, s, nsm);
}

template <int COORD>
cudaError_t launch_ns_strip_visc_coord(int lim, int riem, NsStripSource& src, int ty, int nbuf, cudaStream_t s, int nsm) {
#define FVM_STRIP_CASE(L, R) \
  if (lim == L && riem == R) return launch_ns_strip_visc_lr<L, R, COORD>(src, ty, nbuf, s, nsm);
  FVM_STRIP_CASE(LIM_PC, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_PC, RIEM_HLL)
  FVM_STRIP_CASE(LIM_MINMOD, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_MINMOD, RIEM_HLL)
  FVM_STRIP_CASE(LIM_MC, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_MC, RIEM_HLL)
  FVM_STRIP_CASE(LIM_VANLEER, RIEM_RUSANOV)
  FVM_STRIP_CASE(LIM_VANLEER, RIEM_HLL)
#undef FVM_STRIP_CASE
  return cudaErrorInvalidValue;
}
extern template cudaError_t launch_ns_strip_visc_coord<COORD_CART>(int, int, NsStripSource&, int, int, cudaStream_t, int);
extern template cudaError_t launch_ns_strip_visc_coord<COORD_CYL>(int, int, NsStripSource&, int, int, cudaStream_t, int);
extern template cudaError_t launch_ns_strip_visc_coord<COORD_SPH>(int, int, NsStripSource&, int, int, cudaStream_t, int);
inline cudaError_t launch_ns_strip_visc(int lim, int riem, int coord, NsStripSource& src, int ty, int nbuf,
                                        cudaStream_t s, int nsm) {
  return coord == COORD_CART  ? launch_ns_strip_visc_coord<COORD_CART>(lim, riem, src, ty, nbuf, s, nsm)
         : coord == COORD_CYL ? launch_ns_strip_visc_coord<COORD_CYL>(lim, riem, src, ty, nbuf, s, nsm)
                              : launch_ns_strip_visc_coord<COORD_SPH>(lim, riem, src, ty, nbuf, s, nsm);
}

// ---------------------------------------------------------------- heat ----
template <typename Real, int LIM, int COORD, class Src, int TY = HEAT_TY>
cudaError_t launch_heat_src(const Src& src, long long ntiles, cudaStream_t s, int nsm) {
  using C = HeatCfg<Real, LIM, TY>;
  auto kern = heat_stage_kernel<Real, LIM, COORD, TY, Src>;
  static Residency<1> res;
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::BYTES}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0 || ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[0], nsm);
  kern<<<grid, C::NT, C::BYTES, s>>>(src);
  return cudaGetLastError();
}

template <typename Real, class Src, int TY = HEAT_TY>
cudaError_t launch_heat_any(int lim, int coord, const Src& src, long long ntiles, cudaStream_t s, int nsm) {
#define FVM_HEAT_CASE(L)                                                                               \
  if (lim == L) {                                                                                      \
    if (coord == COORD_CART) return launch_heat_src<Real, L, COORD_CART, Src, TY>(src, ntiles, s, nsm); \
    if (coord == COORD_CYL) return launch_heat_src<Real, L, COORD_CYL, Src, TY>(src, ntiles, s, nsm);   \
    return launch_heat_src<Real, L, COORD_SPH, Src, TY>(src, ntiles, s, nsm);                           \
  }
  FVM_HEAT_CASE(LIM_PC)
  FVM_HEAT_CASE(LIM_MINMOD)
  FVM_HEAT_CASE(LIM_MC)
  FVM_HEAT_CASE(LIM_VANLEER)
#undef FVM_HEAT_CASE
  return cudaErrorInvalidValue;
}

// Float32 piecewise-constant heat (stage_heat_pc.cuh): 4 columns per thread,
// TY = 16 (4 warps) or 8 (2 warps); mixed-batch members also run 20 (5 warps)
// and 10 (2 columns per thread, 5 warps).
constexpr int HEAT_PC_TY = 16, HEAT_PC_TY_ALT = 8;

template <int COORD, int TY>
cudaError_t launch_heat_pc_ty(const CUtensorMap& map, const HeatParams<float>& p, cudaStream_t s, int nsm) {
  constexpr int VX = TY % 4 == 0 ? 4 : 2, NW = TY / VX;
  using C = HeatPcCfg<VX, NW>;
  auto kern = heat_pc_kernel<COORD, VX, NW>;
  static Residency<1> res;
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::BYTES}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  const long long ntiles = tile_total(p);
  if (ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[0], nsm);
  kern<<<grid, C::NT, C::BYTES, s>>>(map, p);
  return cudaGetLastError();
}

cudaError_t launch_heat_pc(int coord, const CUtensorMap& map, HeatParams<float> p, cudaStream_t s, int nsm, int ty);

// Mixed batch (stage_batch_mixed.cuh): navier_stokes (limiter, Riemann
// solver) and heat (coordinate system) tiles in one launch.
template <int LIM, int RIEM, int HCOORD, int HR>
cudaError_t launch_mixed_lrc(const MixedSource& src, long long ntiles, int nbuf, cudaStream_t s, int nsm) {
  auto kern = batch_mixed_kernel<LIM, RIEM, HCOORD, HR>;
  static Residency<3> res;  // with 0, 1 and 2 staged tiles
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, MIX_NT, {mixed_bytes(0), mixed_bytes(1), mixed_bytes(2)}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0 || ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[nbuf], nsm);
  kern<<<grid, MIX_NT, mixed_bytes(nbuf), s>>>(src);
  return cudaGetLastError();
}
// heat_ty: the heat members' tile rows (MIX_HEAT_TY or MIX_HEAT_TY_ALT)
cudaError_t launch_mixed_h4(int lim, int riem, int hcoord, const MixedSource& src, long long ntiles, int nbuf,
                            cudaStream_t s, int nsm);
cudaError_t launch_mixed_h2(int lim, int riem, int hcoord, const MixedSource& src, long long ntiles, int nbuf,
                            cudaStream_t s, int nsm);
inline cudaError_t launch_mixed(int lim, int riem, int hcoord, int heat_ty, const MixedSource& src, long long ntiles,
                                int nbuf, cudaStream_t s, int nsm) {
  return heat_ty == MIX_HEAT_TY_ALT ? launch_mixed_h2(lim, riem, hcoord, src, ntiles, nbuf, s, nsm)
                                    : launch_mixed_h4(lim, riem, hcoord, src, ntiles, nbuf, s, nsm);
}

template <typename Real>
cudaError_t launch_heat(int lim, int coord, const CUtensorMap& map, const HeatParams<Real>& p0, cudaStream_t s,
                        int nsm, int ty) {
  HeatParams<Real> p = p0;
  SingleSource<HeatParams<Real>> src;
  src.tmap = map;
  if constexpr (std::is_same<Real, float>::value) {
    if (ty == HEAT_TY_ALT) {
      set_tiles(p, HEAT_TY_ALT);
      src.p = p;
      return launch_heat_any<Real, SingleSource<HeatParams<Real>>, HEAT_TY_ALT>(
          lim, coord, src, tile_total(p), s, nsm);
    }
  }
  set_tiles(p, HEAT_TY);
  src.p = p;
  return launch_heat_any<Real>(lim, coord, src, tile_total(p), s, nsm);
}
template <typename Real>
cudaError_t launch_heat_batch(int lim, int coord, const BatchSource<HeatParams<Real>>& src, long long ntiles,
                              cudaStream_t s, int nsm) {
  return launch_heat_any<Real>(lim, coord, src, ntiles, s, nsm);
}
extern template cudaError_t launch_heat<float>(int, int, const CUtensorMap&, const HeatParams<float>&, cudaStream_t, int,
                                              int);
extern template cudaError_t launch_heat<double>(int, int, const CUtensorMap&, const HeatParams<double>&, cudaStream_t,
                                               int, int);
extern template cudaError_t launch_heat_batch<float>(int, int, const BatchSource<HeatParams<float>>&, long long,
                                                     cudaStream_t, int);
extern template cudaError_t launch_heat_batch<double>(int, int, const BatchSource<HeatParams<double>>&, long long,
                                                      cudaStream_t, int);

// ------------------------------------------------------------- maxwell ----
// Float64 Maxwell: 8 rows x 32 columns, one block per SM.
constexpr int MAXWELL_TY = 8;

template <typename Real, int LIM, int RIEM, int COORD>
cudaError_t launch_maxwell_one(const CUtensorMap& map, MaxwellParams<Real> p, cudaStream_t s, int nsm) {
  static_assert(std::is_same<Real, double>::value, "float32 grids run stage_maxwell_strip.cuh");
  constexpr int TY = MAXWELL_TY;
  using C = MaxwellCfg<Real, TY>;
  auto kern = maxwell_stage_kernel<Real, LIM, RIEM, COORD, TY>;
  static Residency<1> res;
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::BYTES}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  set_tiles(p, TY);
  const long long ntiles = tile_total(p);
  const int grid = grid_blocks(ntiles, res[0], nsm);
  kern<<<grid, C::NT, C::BYTES, s>>>(map, p);
  return cudaGetLastError();
}

template <typename Real, int COORD>
cudaError_t launch_maxwell_coord(int lim, int riem, const CUtensorMap& map, const MaxwellParams<Real>& p,
                                 cudaStream_t s, int nsm) {
#define FVM_MX_CASE(L)                                                                           \
  if (lim == L) return riem == RIEM_HLL ? launch_maxwell_one<Real, L, RIEM_HLL, COORD>(map, p, s, nsm) \
                                        : launch_maxwell_one<Real, L, RIEM_RUSANOV, COORD>(map, p, s, nsm);
  FVM_MX_CASE(LIM_PC)
  FVM_MX_CASE(LIM_MINMOD)
  FVM_MX_CASE(LIM_MC)
  FVM_MX_CASE(LIM_VANLEER)
#undef FVM_MX_CASE
  return cudaErrorInvalidValue;
}
#define FVM_DECLARE_MX(REAL, COORD)                                                                      \
  extern template cudaError_t launch_maxwell_coord<REAL, COORD>(int, int, const CUtensorMap&,           \
                                                               const MaxwellParams<REAL>&, cudaStream_t, int);
FVM_DECLARE_MX(double, COORD_CART)
FVM_DECLARE_MX(double, COORD_CYL)
FVM_DECLARE_MX(double, COORD_SPH)

template <typename Real>
cudaError_t launch_maxwell(int lim, int riem, int coord, const CUtensorMap& map, const MaxwellParams<Real>& p,
                           cudaStream_t s, int nsm) {
  if (coord == COORD_CART) return launch_maxwell_coord<Real, COORD_CART>(lim, riem, map, p, s, nsm);
  if (coord == COORD_CYL) return launch_maxwell_coord<Real, COORD_CYL>(lim, riem, map, p, s, nsm);
  return launch_maxwell_coord<Real, COORD_SPH>(lim, riem, map, p, s, nsm);
}

// Float32 Maxwell (stage_maxwell_strip.cuh): TY = 8 (2 rows per thread, 4
// output warps) or 16 (4 rows per thread, 4 output warps).
constexpr int MX_STRIP_TY = 8, MX_STRIP_TY_ALT = 16;

template <int LIM, int COORD, int TY>
cudaError_t launch_mx_strip_ty(const MxStripSource& src, int nbuf, cudaStream_t s, int nsm) {
  constexpr int R = TY == 8 ? 2 : 4, NW = TY / R;
  using C = MxStripCfg<R, NW>;
  auto kern = mx_strip_kernel<LIM, COORD, R, NW, TY == 8 ? 3 : 2>;
  static Residency<3> res;  // with 0, 1 and 2 staged tiles
  if (nsm < 0 || !res.known()) {
    const cudaError_t e = prepare_kernel(kern, C::NT, {C::bytes(0), C::bytes(1), C::bytes(2)}, res);
    if (e != cudaSuccess) return e;
  }
  if (nsm < 0) return cudaSuccess;
  const long long ntiles = tile_total(src.p);
  if (ntiles <= 0) return cudaSuccess;
  const int grid = grid_blocks(ntiles, res[nbuf], nsm);
  kern<<<grid, C::NT, C::bytes(nbuf), s>>>(src);
  return cudaGetLastError();
}

cudaError_t launch_mx_strip(int lim, int coord, MxStripSource& src, int ty, int nbuf, cudaStream_t s, int nsm);

}  // namespace fvm

