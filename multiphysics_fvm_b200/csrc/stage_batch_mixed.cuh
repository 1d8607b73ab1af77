// One persistent launch per stage for a batch of float32 grids of two kinds:
// inviscid cartesian Navier-Stokes (the register-blocked body of
// stage_ns_strip.cuh, 8-row tiles) and piecewise-constant heat (the body of
// stage_heat_pc.cuh, 20-row tiles).  A flat work-list of tiles over all grids
// drives the launch; a block finds its grid by binary search over the tile
// offsets and runs that grid's body on the tile, with the grid's own
// parameters (stage coefficients, time step, clock) and tensor maps.  Both
// bodies use 160 threads and share the block's mbarriers: ring barriers 0..5
// (Navier-Stokes uses 0..2) and the Navier-Stokes staged-tile barrier 6, so
// each barrier's phase is tracked by the same threads across tiles of either
// kind.
#pragma once
#include "stage_ns_strip.cuh"
#include "stage_heat_pc.cuh"

namespace fvm {

constexpr int MIX_NS_R = 2, MIX_NS_NW = 4;  // Navier-Stokes: 2-row strips, 8-row tiles
constexpr int MIX_HEAT_NW = 5;              // heat: 4 columns per thread (20-row tiles) or 2 (10-row tiles)
constexpr int MIX_NT = 160;
constexpr int MIX_NBAR = 7;
// Relative cost of a unit in the balanced split of the launch: a Navier-Stokes
// plane (or row tile) of 32 x 8 cells against a heat plane of 32 x 20 (or 32 x
// 10).  Alone, warm-up included, a unit kept a block busy for 3.95 us (one-plane
// 256^2 grids), 4.1 to 4.5 (128^3, 64^3, 96x96x32) and 1.48 (cylindrical heat
// 96x160x48): 2.7 to 3.1 to 1.  (5:2 ran a batch of 64 + 32 grids at 1195 us a step,
// 3:1 at 1178, 7:2 at 1197.)
constexpr int MIX_NS_COST = 6, MIX_HEAT_COST = 2, MIX_HEAT_COST_ALT = 1;
constexpr int MIX_NS_TY = MIX_NS_R * MIX_NS_NW, MIX_HEAT_TY = 4 * MIX_HEAT_NW, MIX_HEAT_TY_ALT = 2 * MIX_HEAT_NW;
static_assert(NsStripCfg<MIX_NS_R, MIX_NS_NW>::NT == MIX_NT && HeatPcCfg<4, MIX_HEAT_NW>::NT == MIX_NT,
              "both bodies run on the same block");

// Shared memory of a launch with `nbuf` staged Navier-Stokes tiles: the larger
// body, then the barriers.
__host__ __device__ constexpr int mixed_bar_offset(int nbuf) {
  return round_up(cmax(NsStripCfg<MIX_NS_R, MIX_NS_NW>::bytes(nbuf),
                       HeatPcCfg<4, MIX_HEAT_NW>::NSLOT * HeatPcCfg<4, MIX_HEAT_NW>::SLOT * 4),
                  8);
}
// ... and the parameters of the Navier-Stokes piece in work.  (Read from global
// memory they are loaded again after every store of a step, in which the compiler
// must suppose an alias; a heat piece, with registers to spare, copies its own
// to them.  Stage of 64 + 32 grids 301 -> 262 us.)
__host__ __device__ constexpr int mixed_param_offset(int bar_off) { return (bar_off + MIX_NBAR * 8 + 15) & ~15; }
__host__ __device__ constexpr int mixed_bytes(int nbuf) {
  return mixed_param_offset(mixed_bar_offset(nbuf)) + (int)sizeof(NsParams<float>);
}

// Per grid and stage: what a tile of that grid needs.
struct alignas(64) MixedInst {
  CUtensorMap tmap;    // ring map of the stage input
  CUtensorMap u0map;   // staged U0 tile (Navier-Stokes)
  CUtensorMap accmap;  // staged accumulator tile (Navier-Stokes)
  NsParams<float> ns;
  HeatParams<float> heat;
  int kind;  // 0 Navier-Stokes, 1 heat
  int ncol, nunit, zchunk, weight;  // tile_walk.cuh; weight: relative cost of a unit
};

struct MixedSource {
  const MixedInst* inst;    // per grid, this stage
  const long long* starts;  // ninst + 1 prefix sums of unit costs (or pieces)
  int ninst;
  int bal;                  // the launch is balanced (depth 0)
  int bar_off;              // byte offset of the barriers in shared memory
  __device__ __forceinline__ bool balanced() const { return bal != 0; }
  __device__ __forceinline__ long long total() const { return __ldg(starts + ninst); }
  __device__ __forceinline__ int instance(long long pos) const { return find_instance(starts, ninst, pos); }
  __device__ __forceinline__ long long start(int i) const { return __ldg(starts + i); }
  __device__ __forceinline__ const MixedInst& params(int i) const { return inst[i]; }
  __device__ __forceinline__ int weight(int i) const { return inst[i].weight; }
};

// HVX: heat columns per thread (4: 20-row heat tiles, 2: 10-row).
template <int LIM, int RIEM, int HCOORD, int HVX>
__global__ void __launch_bounds__(MIX_NT, 3) batch_mixed_kernel(const __grid_constant__ MixedSource src) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + src.bar_off);
  const int tid = threadIdx.x;
  if (smem_u32(smem_raw) & 127u) {  // TMA destinations need 128-byte alignment
    if (tid == 0) {
      const MixedInst& in = src.inst[0];
      atomicOr(in.kind == 0 ? in.ns.status : in.heat.status, ST_TMA_TIMEOUT);
    }
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < MIX_NBAR; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
  }
  __syncthreads();
  unsigned phase_bits = 0, pending = 0;
  TileWalk<MixedSource> walk(src);
  Piece pc;
  int inst;
  bool ok = true;
  while (ok && walk.next(src, inst, pc)) {
    const MixedInst& in = src.inst[inst];
    if (in.kind == 0) {
      if (in.ns.active && !*in.ns.active) continue;  // this grid's clock passed t_end
      NsParams<float>& ns = *reinterpret_cast<NsParams<float>*>(smem_raw + mixed_param_offset(src.bar_off));
      // (the last piece's readers are past the barrier that ended it)
      for (int q = tid; q < (int)sizeof(ns); q += MIX_NT)  // by bytes, which may alias every field
        reinterpret_cast<unsigned char*>(&ns)[q] = reinterpret_cast<const unsigned char*>(&in.ns)[q];
      __syncthreads();
      if (ns.flat)
        ok = ns_strip_tile<LIM, RIEM, MIX_NS_R, MIX_NS_NW, COORD_CART, true, false>(
            ns, &in.tmap, &in.u0map, &in.accmap, pc, smem_raw, bars, bars + 6, 6, phase_bits, pending);
      else
        ok = ns_strip_tile<LIM, RIEM, MIX_NS_R, MIX_NS_NW, COORD_CART, false, false>(
            ns, &in.tmap, &in.u0map, &in.accmap, pc, smem_raw, bars, bars + 6, 6, phase_bits, pending);
    } else {
      if (in.heat.active && !*in.heat.active) continue;
      const HeatParams<float> heat = in.heat;
      ok = heat_pc_tile<HCOORD, HVX, MIX_HEAT_NW>(heat, &in.tmap, pc, smem_raw, bars, phase_bits, pending);
    }
  }
  // On a timeout, wait (bounded) for every copy this block may still have in flight.
  if (!ok && tid == 0) {
    const MixedInst& in = src.inst[0];
    const unsigned long long lim = in.kind == 0 ? in.ns.drain_ns : in.heat.drain_ns;
    for (int s = 0; s < MIX_NBAR; ++s)
      if ((pending >> s) & 1u) mbar_wait_bounded(&bars[s], (phase_bits >> s) & 1u, lim);
  }
}

}  // namespace fvm
