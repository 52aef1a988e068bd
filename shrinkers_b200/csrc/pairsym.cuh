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

__device__ __forceinline__ void sym_add(double& a, double b) { a += b; }
__device__ __forceinline__ void sym_add(double2& a, double2 b) {
  a.x += b.x;
  a.y += b.y;
}

// Reduction of a phase's partials: a CTA of SYM_NT threads takes 32 targets
// from t0 (one tile: tiles are multiples of 256 targets).  Warp w adds every
// eighth partial (the columns of the tiles before theirs, then their rows in
// CTA order); the eight sums are added in warp order after `acc`, the sums of
// the earlier phases (null in the first).  The result is valid in warp 0.  (A
// thread per target walked all its partials alone: 11 us at p = 4096, where
// the sums themselves take 12.)
template <typename V>
__device__ __forceinline__ V sym_collect(const SymPlan& pl, const V* __restrict__ rows,
                                         const V* __restrict__ cols, const V* acc, int64_t t0) {
  __shared__ V part[SYM_NT / 32][32];
  __shared__ int cs[2];
  constexpr int NW = SYM_NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t = t0 + lane < pl.p ? t0 + lane : pl.p - 1;
  const int tile = (int)(t0 / pl.tt);
  const bool own = tile >= pl.t0 && tile < pl.t1;
  if (threadIdx.x < 2 && own) {
    const int64_t base0 = pl.before(pl.t0);
    cs[threadIdx.x] = pl.cta_of(pl.before(tile + threadIdx.x) - base0 - threadIdx.x);
  }
  V sum{};
  const int nc = min(tile, pl.t1) - pl.t0;
#pragma unroll 4
  for (int k = warp; k < nc; k += NW) sym_add(sum, cols[(int64_t)k * pl.p + t]);
  __syncthreads();
  if (own) {
    const int c1 = cs[1];
    const V* row = rows + (int64_t)(tile - pl.t0) * pl.tt + (t - (int64_t)tile * pl.tt);
#pragma unroll 4
    for (int c = cs[0] + warp; c <= c1; c += NW) sym_add(sum, row[(int64_t)c * pl.tt]);
  }
  part[warp][lane] = sum;
  __syncthreads();
  if (warp == 0) {
    if (acc) sym_add(sum, acc[t]);
#pragma unroll
    for (int w = 1; w < NW; ++w) sym_add(sum, part[w][lane]);
  }
  return sum;
}

}  // namespace shrk
