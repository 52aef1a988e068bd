// Work split of the symmetric all-points sums (forward: pairsym.cu, adjoint:
// adjoint.cu): every unordered pair of a spectrum is evaluated once and added
// to both of its ends.
//
// Tile T holds TT = 256*R consecutive targets, R per thread; its sources are
// the tile itself (a full square, rows only) and everything after it (each
// pair feeds the target's row sum and the source's column sum).  The sources
// of a tile are cut into units of SYM_UB, the units of all tiles are numbered
// tile after tile, and CTA c of G takes the c-th of G equal runs of them, so
// the triangle is balanced to one unit whatever its size (fixed tiles of
// (T, S) pairs lose up to a wave: 820 items on 296 CTAs run as long as 888).
// A run crosses few tiles; the path (c, T) only moves forward, so c + T - T0
// numbers the row partials without gaps to clear.
//
// Column partials go to one slab per tile.  The slabs of all tiles of a large
// spectrum would not fit (16 GB at p = 1e6), so tiles run in phases of as
// many as the slab budget holds, each phase reduced before the next.
#pragma once

#include "common.cuh"

namespace shrk {

constexpr int SYM_NT = 256;   // threads per CTA
constexpr int SYM_UB = 64;    // sources per unit
constexpr int SYM_CH = 256;   // sources staged at a time

struct SymPlan {
  int64_t p;
  int64_t u0;        // units of tile 0
  int tt;            // targets per tile
  int t0, t1;        // tiles of this phase
  int64_t units;     // units of this phase
  int grid;          // CTAs: the first `rem` run per + 1 units, the others per
  int64_t per;
  int rem;

  // Units of the tiles before T, counted from tile 0 (tt is a multiple of
  // SYM_UB, so each tile has tt / SYM_UB units less than the one before).
  __host__ __device__ int64_t before(int64_t T) const {
    return T * u0 - (int64_t)(tt / SYM_UB) * (T * (T - 1) / 2);
  }
  __host__ __device__ int64_t first_unit(int c) const { return c * per + (c < rem ? c : rem); }
  // The tile of unit u (counted from the phase's first unit).
  __host__ __device__ int tile_of(int64_t u) const {
    const int64_t v = u + before(t0);
    int lo = t0, hi = t1 - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (before(mid) <= v) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
  // The CTA that runs unit u.
  __host__ __device__ int cta_of(int64_t u) const {
    const int64_t head = rem * (per + 1);
    return (int)(u < head ? u / (per + 1) : rem + (u - head) / per);
  }
};

// The plan of tiles [t0, t1) of a spectrum of p values.
inline SymPlan sym_plan(int64_t p, int tt, int t0, int t1, int ctas) {
  SymPlan pl;
  pl.p = p;
  pl.u0 = (p + SYM_UB - 1) / SYM_UB;
  pl.tt = tt;
  pl.t0 = t0;
  pl.t1 = t1;
  pl.units = pl.before(t1) - pl.before(t0);
  pl.grid = (int)(pl.units < ctas ? pl.units : ctas);
  pl.per = pl.units / pl.grid;
  pl.rem = (int)(pl.units % pl.grid);
  return pl;
}

}  // namespace shrk
