// How a persistent launch's blocks share a stage's work.
//
// The work of a grid is ncol columns (a tile's footprint in x1, x2) of nunit
// units each: a unit is one output plane of the z-march, or, on a one-plane
// grid of the register-blocked Navier-Stokes kernel, one row tile of the march
// along x2.  A piece is a run of consecutive units of one column; it costs its
// units plus a fixed warm-up (the planes below the first output plane).
//
// Balanced (depth 0, the default): the units of all columns in a row are cut
// into gridDim equal runs, one per block, so every block does the same number
// of units to within one, whatever the grid's size; a run that crosses a
// column boundary is two pieces.  Fixed depth (> 0): pieces of `zchunk` units
// dealt round-robin, ceil(pieces / blocks) rounds: a 256^3 grid in 64-plane
// pieces fills 2.3 rounds of 444 resident blocks and takes 3, and a 97x130x61
// one occupies 68 blocks.  Measured stage launches, fixed 64 -> balanced, when the
// split was introduced: inviscid NS 256^3 811 -> 715 us and 97x130x61 342 -> 95,
// viscous cylindrical 96x128x64 437 -> 147, Maxwell 128x128x256 395 -> 291, heat
// 192x256x128 89 -> 38, viscous 256^3 1547 -> 1497, 64x64x1 17.2 -> 6.6.
//
// What the balanced split costs: the warm-up is not counted, so a block whose run
// crosses a column boundary pays it twice (two planes of a run of 9 at 97x130x61);
// and neighbouring columns are marched at different heights, so a tile's halo is
// seldom still in L2.  At 192^3 the launches moved 1.71 (inviscid) and 2.65
// (viscous) times the algorithmic bytes, 1.07 and 1.10 in equal chunks.  Bandwidth
// does not bound those kernels, but a sweep over depths finds what is left: 256^3
// inviscid 543 us a stage, 508 at depth 48.
#pragma once
#include "fvm_common.cuh"

namespace fvm {

// One run of consecutive units of one column.
struct Piece {
  int col;     // column: col % ntx along x1, col / ntx along x2
  int u0, u1;  // units u0 .. u1 - 1 (unit u = interior plane u, or row tile u)
};

// The pieces of one block.  Src: total() and, per grid of the launch,
// instance(pos) / start(inst) (prefix sums of cost, balanced, or of pieces,
// fixed depth), params(inst) with ncol, nunit, zchunk, and weight(inst), the
// cost of a unit; balanced() tells the two orders apart.
template <class Src>
struct TileWalk {
  long long pos, end;
  __device__ __forceinline__ explicit TileWalk(const Src& src) {
    const long long total = src.total();
    if (src.balanced()) {
      pos = total * blockIdx.x / gridDim.x;
      end = total * (blockIdx.x + 1) / gridDim.x;
    } else {
      pos = blockIdx.x;
      end = total;
    }
  }
  // The next piece of this block, of grid `inst`; false when none is left.
  __device__ __forceinline__ bool next(const Src& src, int& inst, Piece& pc) {
    while (pos < end) {
      inst = src.instance(pos);
      const auto& p = src.params(inst);
      const long long at = src.start(inst);
      if (!src.balanced()) {
        const int tile = (int)(pos - at), zc = tile / p.ncol;
        pc.col = tile - zc * p.ncol;
        pc.u0 = zc * p.zchunk;
        pc.u1 = min(pc.u0 + p.zchunk, p.nunit);
        pos += gridDim.x;
        return true;
      }
      // the units whose cost interval starts inside this block's run
      const int w = src.weight(inst);
      const long long n = (long long)p.ncol * p.nunit;
      const long long u = (pos - at + w - 1) / w, ue = min(n, (end - at + w - 1) / w);
      if (u >= ue) {
        pos = u >= n ? at + n * w : end;
        continue;
      }
      pc.col = (int)(u / p.nunit);
      pc.u0 = (int)(u - (long long)pc.col * p.nunit);
      pc.u1 = (int)min((long long)p.nunit, pc.u0 + (ue - u));
      pos = at + (u + pc.u1 - pc.u0) * w;
      return true;
    }
    return false;
  }
};

// Tile sources: one grid (params + tensor map in kernel parameter space) or a
// batch of independent grids (per-instance params and maps in global memory,
// the instance of a position found by binary search over the prefix sums).
template <class P>
struct OneGrid {
  const P& p;
  __device__ __forceinline__ bool balanced() const { return p.zchunk == 0; }
  __device__ __forceinline__ long long total() const {
    return (long long)p.ncol * (p.zchunk == 0 ? p.nunit : (p.nunit + p.zchunk - 1) / p.zchunk);
  }
  __device__ __forceinline__ int instance(long long) const { return 0; }
  __device__ __forceinline__ long long start(int) const { return 0; }
  __device__ __forceinline__ const P& params(int) const { return p; }
  __device__ __forceinline__ int weight(int) const { return 1; }
};
template <class P>
struct SingleSource {
  CUtensorMap tmap;
  P p;
  __device__ __forceinline__ bool balanced() const { return p.zchunk == 0; }
  __device__ __forceinline__ long long total() const { return OneGrid<P>{p}.total(); }
  __device__ __forceinline__ int instance(long long) const { return 0; }
  __device__ __forceinline__ long long start(int) const { return 0; }
  __device__ __forceinline__ const P& params(int) const { return p; }
  __device__ __forceinline__ int weight(int) const { return 1; }
  __device__ __forceinline__ const CUtensorMap* map(int) const { return &tmap; }
};
// The grid whose interval [start[i], start[i+1]) holds pos.
__device__ __forceinline__ int find_instance(const long long* start, int ninst, long long pos) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(start + mid) <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
template <class P>
struct BatchSource {
  const P* prm;             // per instance (this stage)
  const CUtensorMap* maps;  // per instance: map of this stage's input buffer
  const long long* starts;  // ninst+1 prefix sums of units (or pieces)
  int ninst;
  int bal;                  // the launch is balanced (depth 0)
  __device__ __forceinline__ bool balanced() const { return bal != 0; }
  __device__ __forceinline__ long long total() const { return __ldg(starts + ninst); }
  __device__ __forceinline__ int instance(long long pos) const { return find_instance(starts, ninst, pos); }
  __device__ __forceinline__ long long start(int i) const { return __ldg(starts + i); }
  __device__ __forceinline__ const P& params(int i) const { return prm[i]; }
  __device__ __forceinline__ int weight(int) const { return 1; }
  __device__ __forceinline__ const CUtensorMap* map(int i) const { return maps + i; }
};

// Row tiles of a flat grid's piece in a fixed-depth launch.
constexpr int NS_FLAT_ROWS = 4;
// Host: columns and units of a grid in tiles of 32 x ty; `flat` marches over
// the row tiles of a one-plane grid.
template <class P>
void set_tiles(P& p, int ty, bool flat = false) {
  p.ntx = (p.lay.nx + 31) / 32;
  p.nty = (p.lay.ny + ty - 1) / ty;
  p.ncol = flat ? p.ntx : p.ntx * p.nty;
  p.nunit = flat ? p.nty : p.lay.nz;
  if (flat && p.zchunk > 0) p.zchunk = NS_FLAT_ROWS;
}
// Units (balanced) or pieces (fixed depth) of a grid.
template <class P>
long long tile_total(const P& p) {
  return (long long)p.ncol * (p.zchunk == 0 ? p.nunit : (p.nunit + p.zchunk - 1) / p.zchunk);
}

}  // namespace fvm
