// FFT grid convolution for the Stieltjes transform on sm_100a: the fft5
// family (fft5 / fft3 / fft2, and the real part of adaptive and dst) and the
// coarse-grid NUFFT preset over the same pipeline.
//
// Replaces the dual-convolution core of src/stieltjes/fft5.rs
// (Fft5Options 213-249, lagrange_weights 136-164, splat 175-185 / 259-318,
// fft_convolution 325-432, interp_at 191-211, interpolate_grid 440-476, entry
// points 559-625), the packing helpers of src/stieltjes/fftplan.rs:43-76 and
// the NUFFT policy of src/stieltjes/nufft.rs (33-126, entry points 164-220).
// Pipeline (all FP64), stencil width N = 2/4/6/8 a template parameter:
//
//   1. runs         a source's stencil cell is i0 = floor((v-lo)/dx); the
//                   sources are sorted, so the cells are too: one thread per
//                   source finds its cell and its N Lagrange weights, the
//                   sources at which the cell changes mark the runs of equal
//                   cells, and each run gets the sums of its weights.
//   2. pack         one thread per grid cell adds the weights of its sources
//                   (at most 32) run by run in ascending source order -- the
//                   order of the reference's sequential splat, so these
//                   densities are the same sums, without atomics; a denser
//                   cell adds the N run sums.  The N Lagrange weights of
//                   t = pos - i0 are recomputed where they are added
//                   (sources come from L2; no weight array).
//                   packed[c] = density[c] + i x_c/(x_c^2 + eta^2).
//   3. fft          four-step FFT m = m1*m2 (m1, m2 <= 2048): column FFTs of
//                   length m1 with the inter-pass twiddle, then row FFTs of
//                   length m2, in registers with exchanges through shared
//                   memory.  Twiddles and the analytic even-kernel spectrum
//                   are device tables cached per grid.
//   4. fft          inverse transform, whose column pass forms the spectral
//                   product on the way in: unpack the two real spectra
//                   (conjugate symmetry), Im_hat + i Re_hat = D*K_even +
//                   i D*K_odd.
//   5. interp       N-point interpolation at the query points, 1/m scale,
//                   fused FP64 epilogue.
#include "common.cuh"
#include "epilogue.cuh"
#include "internal.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <string>

namespace shrk {

namespace {

// nufft.rs:33-58
constexpr double NUFFT_PAD_ETA_MULT = 2000.0;
constexpr double NUFFT_PAD_RANGE_FRAC = 0.75;
constexpr double NUFFT_RESOLUTION = 5.0;
constexpr size_t NUFFT_MIN_GRID = 8192;
constexpr size_t NUFFT_MAX_GRID = 65536;

// fft5.rs:345-353: dx <= eta/8, m >= 8p, at most 2^20 cells.
constexpr size_t FFT5_MAX_AUTO_GRID = (size_t)1 << 20;

constexpr int FFT_MAXL = 2048;                  // longest in-shared-memory transform
constexpr int64_t FFT_MAX_M = (int64_t)FFT_MAXL * FFT_MAXL;

size_t next_pow2(size_t n) {  // mod.rs:529-535
  size_t p = 1;
  while (p < n) p <<= 1;
  return p;
}

// Rust's saturating float -> usize cast (NaN and negatives -> 0).
size_t sat_usize(double v) {
  if (!(v > 0.0)) return 0;
  if (v >= 18446744073709551616.0) return SIZE_MAX;
  return (size_t)v;
}

// x / den for a constant integer |den| < 2^13, correctly rounded without a
// division: q = x rc (rc the rounded reciprocal) is within 1.5 ulp and one
// residual step leaves q + r rc within 1.5 2^-53 ulp of x / den, while a
// quotient by den that is not itself a midpoint is at least ulp / (2 |den|)
// from the nearest one.  (The stencil divides by N constants a source and a
// query; the divisions were two thirds of the weights' time.)
__device__ __forceinline__ double div_const(double x, double den, double rc) {
  const double q = x * rc;
  return fma(fma(-q, den, x), rc, q);
}

// fft5.rs:136-164 lagrange_weights<N>, operation order preserved.
template <int N>
__device__ __forceinline__ void lagrange(double t, double w[N]) {
  const double q = (double)(N / 2);
  double pref[N], suf[N], acc = 1.0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    pref[j] = acc;
    acc *= t - (double)j + q - 1.0;
  }
  acc = 1.0;
#pragma unroll
  for (int j = N - 1; j >= 0; --j) {
    suf[j] = acc;
    acc *= t - (double)j + q - 1.0;
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    double den = 1.0;
#pragma unroll
    for (int l = 0; l < N; ++l)
      if (l != j) den *= (double)(j - l);
    w[j] = div_const(pref[j] * suf[j], den, 1.0 / den);
  }
}

// A grid's spacing with its rounded reciprocal (0 outside the range in which
// the quotients below are exact, so that they take the division).
struct Spacing {
  double dx, rdx;
};

Spacing spacing(double dx) {
  const double ax = std::fabs(dx);
  return {dx, ax > 1e-100 && ax < 1e100 ? 1.0 / dx : 0.0};
}

// a / dx, correctly rounded: two residual steps on a rdx (Markstein: a
// faithful quotient corrected once with the rounded reciprocal is the rounded
// quotient); anything outside the plain range, NaN included, divides.
__device__ __forceinline__ double grid_pos(double a, const Spacing& h) {
  double q = a * h.rdx;
  const double aq = fabs(q);
  if (!(aq > 1e-100 && aq < 1e100)) return a / h.dx;
  q = fma(fma(-q, h.dx, a), h.rdx, q);
  return fma(fma(-q, h.dx, a), h.rdx, q);
}

// floor((v - lo)/dx) as a cell index clamped to [-N - 1, m + N] (every slot
// of a source beyond that range lands on the same edge cell), and the
// fraction t = pos - floor(pos) of the unclamped position.
template <int N>
__device__ __forceinline__ int64_t cell_of(double v, double lo, const Spacing& h, int64_t m,
                                           double* t) {
  const double pos = grid_pos(v - lo, h);
  const double fl = floor(pos);
  *t = pos - fl;
  const double c = fmin(fmax(fl, -(double)N - 1.0), (double)(m + N));
  return (int64_t)c;
}

struct GridArgs {
  const double* src;  // ascending
  int64_t ns;
  int rev;            // 1: visit the sources in descending order (dx < 0)
  double lo;
  Spacing h;
  double eta;
  int64_t m;
  double2* packed;
  double* dens;       // non-null: write the density alone (the splat stage)
};

__device__ __forceinline__ double visited(const GridArgs& a, int64_t j) {
  return a.rev ? a.src[a.ns - 1 - j] : a.src[j];
}

template <int N>
__device__ __forceinline__ int clamped_cell(const GridArgs& a, double v, double* t) {
  const int64_t i0 = cell_of<N>(v, a.lo, a.h, a.m, t);
  return (int)(i0 < -N ? -N : (i0 > a.m + N ? a.m + N : i0));
}

constexpr int DENSE_MIN = 32;  // cells with more sources take their density from run sums

// The runs of equal stencil cells and their weight sums.  run[cell + N + 1] =
// the visited sources [x, y) of that cell, {0, 0} for an empty one (zero on
// entry).  The sources are cut in chunks of SPLAT_CHUNK, a CTA each: a run
// inside one chunk has its sums in sum[(cell + N + 1) N + k]; one that spans
// chunks has tail[] of the chunk it starts in plus head[] of the later ones,
// in that order.
struct Runs {
  int2* run;
  double* sum;
  double* head;  // [chunks][N]
  double* tail;
};

constexpr int SPLAT_CHUNK = 512;
constexpr int SPLAT_NT = 256;
constexpr int SPLAT_LONG = 32;  // longer pieces of a run are summed by a warp
// Runs of more sources have their heads added by a warp in the pack (by a lane,
// one after the other: 10^6 sources, half of them zeros as in a spectrum with a
// null space, nufft 218 us, so 107; 4 10^6: 745 and 181).
constexpr int HEADS_LONG = 8 * SPLAT_CHUNK;

// One chunk of sources: each source's cell and weights once, by a thread each
// (coalesced), into shared memory; the places where the cell changes cut the
// chunk in pieces; each piece's N sums in source order by a thread each, or by
// a warp for a long piece (lanes strided, a fixed butterfly).  Work follows
// the sources, whatever their spread: a thread per cell that bisected for its
// run's start spent 51 us on the 2^20 cells of 200 003 sources (mostly empty
// ones), and a warp a run 14 us more on runs of ten sources; this takes 8, and
// 14 us for 10^6 sources on 65 536 cells, where those took 41.  FP64-bound:
// about 60 operations a source at N = 4, 90 at N = 8.
template <int N>
__global__ void __launch_bounds__(SPLAT_NT) splat_kernel(const GridArgs a, const Runs R) {
  constexpr int W = SPLAT_CHUNK + 1;
  constexpr int PER = SPLAT_CHUNK / SPLAT_NT;
  extern __shared__ double wsm[];       // [N][W]
  __shared__ int cell_sh[SPLAT_CHUNK + 2];  // of the sources j0 - 1 .. j0 + SPLAT_CHUNK
  __shared__ int start[SPLAT_CHUNK + 1];    // pieces, in source order
  __shared__ int longs[SPLAT_CHUNK / SPLAT_LONG];
  __shared__ int base[PER * SPLAT_NT / 32 + 1];
  __shared__ int n_long;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int64_t j0 = (int64_t)blockIdx.x * SPLAT_CHUNK;
  const int n = (int)(a.ns - j0 < SPLAT_CHUNK ? a.ns - j0 : SPLAT_CHUNK);
  if (tid == 0) n_long = 0;
#pragma unroll
  for (int it = 0; it < PER; ++it) {
    const int i = tid + it * SPLAT_NT;
    if (i < n) {
      double t, w[N];
      cell_sh[i + 1] = clamped_cell<N>(a, visited(a, j0 + i), &t);
      lagrange<N>(t, w);
#pragma unroll
      for (int k = 0; k < N; ++k) wsm[k * W + i] = w[k];
    }
  }
  if (tid == 0 || tid == 32) {  // the neighbours; INT_MIN is no cell
    const int64_t j = tid ? j0 + n : j0 - 1;
    double t;
    cell_sh[tid ? n + 1 : 0] = j >= 0 && j < a.ns ? clamped_cell<N>(a, visited(a, j), &t) : INT_MIN;
  }
  __syncthreads();
  // pieces: a source whose cell differs from the one before it, and source 0
  unsigned flags[PER];
#pragma unroll
  for (int it = 0; it < PER; ++it) {
    const int i = tid + it * SPLAT_NT;
    const bool f = i < n && (i == 0 || cell_sh[i + 1] != cell_sh[i]);
    flags[it] = __ballot_sync(0xffffffffu, f);
    if (lane == 0) base[it * (SPLAT_NT / 32) + wib + 1] = __popc(flags[it]);
  }
  if (tid == 0) base[0] = 0;
  __syncthreads();
  if (wib == 0) {  // inclusive scan of the PER * SPLAT_NT / 32 <= 32 counts
    constexpr int NB = PER * SPLAT_NT / 32;
    static_assert(NB <= 32, "one warp scans the counts");
    int v = lane < NB ? base[lane + 1] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane < NB) base[lane + 1] = v;
  }
  __syncthreads();
  const int pieces = base[PER * SPLAT_NT / 32];
#pragma unroll
  for (int it = 0; it < PER; ++it) {
    const int i = tid + it * SPLAT_NT;
    if ((flags[it] >> lane) & 1u) {
      start[base[it * (SPLAT_NT / 32) + wib] + __popc(flags[it] & ((1u << lane) - 1u))] = i;
      // the run's ends, each written once
      const int c = cell_sh[i + 1], before = cell_sh[i];
      if (c != before) {
        R.run[c + N + 1].x = (int)(j0 + i);
        if (before != INT_MIN) R.run[before + N + 1].y = (int)(j0 + i);
      }
    }
  }
  if (tid == 0) {
    start[pieces] = n;
    if (j0 + n == a.ns) R.run[cell_sh[n] + N + 1].y = (int)a.ns;
  }
  __syncthreads();
  const auto out = [&](int p, int p0, int p1) -> double* {
    const int c = cell_sh[p0 + 1];
    if (p == 0 && cell_sh[0] == c) return R.head + (int64_t)blockIdx.x * N;
    if (p1 == n && cell_sh[n + 1] == c) return R.tail + (int64_t)blockIdx.x * N;
    return R.sum + (int64_t)(c + N + 1) * N;
  };
  for (int u = tid; u < pieces * N; u += SPLAT_NT) {
    const int p = u / N, k = u % N, p0 = start[p], p1 = start[p + 1];
    if (p1 - p0 > SPLAT_LONG) {
      if (k == 0) longs[atomicAdd(&n_long, 1)] = p;
      continue;
    }
    double s = 0.0;
    for (int i = p0; i < p1; ++i) s += wsm[k * W + i];
    out(p, p0, p1)[k] = s;
  }
  __syncthreads();
  for (int u = wib; u < n_long * N; u += SPLAT_NT / 32) {
    const int p = longs[u / N], k = u % N, p0 = start[p], p1 = start[p + 1];
    double s = 0.0;
    for (int i = p0 + lane; i < p1; i += 32) s += wsm[k * W + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out(p, p0, p1)[k] = s;
  }
}

// The density of cell c is the sum of weight k over the run of sources with
// cell c + N/2 - 1 - k, k = N-1 .. 0 (fft5.rs:175-185).  A cell with at most
// DENSE_MIN sources adds them one by one, runs in ascending cell order and
// each run in ascending source order -- the order of the reference's
// sequential splat, so these densities are the same sums, without atomics;
// a denser cell adds the N run sums in that run order (deterministic, not the
// sequential order).  The two edge cells also collect every clamped slot.
// packed[c] = density[c] + i x_c/(x_c^2 + eta^2) (fft5.rs:364-376).
// The odd kernel's sample x_c/(x_c^2 + eta^2).
__device__ __forceinline__ double odd_kernel(const GridArgs& a, int64_t c) {
  const int64_t half = a.m / 2;
  const double sd = (c <= half) ? (double)c : (double)c - (double)a.m;
  const double x = sd * a.h.dx;
  return x / (x * x + a.eta * a.eta);
}

// The long runs of a warp's window: for each, the warp adds its heads but the
// first, a chunk a lane, all N sums together, and leaves the run as its tail and
// one head to the lanes' own sums; the result is what those miss in the lane's
// cell.  (Out of line: its registers are the pack's only where it runs.)
template <int N>
__device__ __noinline__ double add_heads(const double* __restrict__ head, int2* run, int lane,
                                         double* tot) {
  double extra = 0.0;
  for (int e = 0; e < 32 + N; ++e) {
    const int2 q = run[e];
    if (q.y - q.x <= HEADS_LONG) continue;
    double t[N] = {};
    const int c0 = q.x / SPLAT_CHUNK, c1 = (q.y - 1) / SPLAT_CHUNK;
#pragma unroll 2
    for (int h = c0 + 2 + lane; h <= c1; h += 32) {
#pragma unroll
      for (int k = 0; k < N; ++k) t[k] += __ldg(head + (int64_t)h * N + k);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
      if (lane == 0) tot[k] = t[k];
    }
    if (lane == 0) run[e].y = (c0 + 1) * SPLAT_CHUNK + 1;
    __syncwarp();
    const int i = e - lane;
    if (i >= 0 && i < N) extra += tot[N - 1 - i];
    __syncwarp();
  }
  return extra;
}

// A cell's sources are one stretch [A, B) of the sorted sources.  The sparse
// cells of a warp share theirs 32 sources at a time: a lane per source finds
// its cell and weights into shared memory, then every lane adds its own cell's
// in source order.  (Each lane walking its own sources was a serial chain of
// up to 32 loads and stencils; a lot of 32 sources takes 2 700 clk, and the
// kernel on 2^20 cells 14 us where it took 18.)
// Most cells of a large grid are empty: a warp whose window has no run stores
// its odd kernel and ends.
template <int N>
__global__ void __launch_bounds__(256, 6) pack_kernel(const GridArgs a, const Runs R) {
  constexpr int H = N / 2;
  constexpr int NP = N == 6 ? 8 : N;
  __shared__ double wsm[8][32 * NP];
  __shared__ __align__(16) int off_sh[8][32];
  __shared__ int2 run_sh[8][32 + N];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, cw = c - lane;
  const int64_t m = a.m;
  const int2* run = R.run + N + 1;  // run[cell] for -N - 1 <= cell <= m + N
  // the warp's window: the runs of the cells cw - H .. cw + 31 + H
  const int64_t e0 = cw - H + lane, e1 = e0 + 32;
  const int2 w0 = e0 <= m + N ? __ldg(run + e0) : make_int2(0, 0);
  const int2 w1 = lane < N && e1 <= m + N ? __ldg(run + e1) : make_int2(0, 0);
  const double odd = a.dens || c >= m ? 0.0 : odd_kernel(a, c);
  double dens = 0.0;
  const bool edge = cw == 0 || cw + 32 >= m;
  if (edge || __any_sync(0xffffffffu, w0.y > w0.x || w1.y > w1.x)) {
    const bool longs = __any_sync(0xffffffffu, max(w0.y - w0.x, w1.y - w1.x) > HEADS_LONG);
    run_sh[wib][lane] = w0;
    if (lane < N) run_sh[wib][32 + lane] = w1;
    __syncwarp();
    const int2* r = run_sh[wib] + lane;  // r[i]: the run of cell c - H + i
    unsigned A = UINT_MAX, B = 0;
    if (c > 0 && c < m - 1) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (r[i].y > r[i].x) {
          A = min(A, (unsigned)r[i].x);
          B = (unsigned)r[i].y;
        }
    }
    const bool any = B > A;
    const bool sparse = any && B - A <= DENSE_MIN;
    int64_t ahead = -1;
    double v_ahead = 0.0;
    for (unsigned pos = 0;;) {
      unsigned next = sparse && B > pos ? max(A, pos) : UINT_MAX;
      next = __reduce_min_sync(0xffffffffu, next);
      if (next == UINT_MAX) break;
      const int64_t j = (int64_t)next + lane;
      const double v = ahead == j ? v_ahead : j < a.ns ? visited(a, j) : 0.0;
      ahead = j + 32;  // mostly the next lot's
      if (ahead < a.ns) v_ahead = visited(a, ahead);
      if (j < a.ns) {
        double t, w[N];
        // the weight of cell c is entry off + 32 (c - cw), k = c + H - 1 - cell
        off_sh[wib][lane] = lane + 32 * (int)(cw + H - 1 - clamped_cell<N>(a, v, &t));
        lagrange<N>(t, w);
#pragma unroll
        for (int k = 0; k < N; ++k) wsm[wib][k * 32 + lane] = w[k];
      }
      __syncwarp();
      pos = next + 32;
      if (sparse) {
        const int i1 = (int)(min(B, pos) - next);
#pragma unroll 8
        for (int i = (int)(max(A, next) - next); i < i1; ++i)  // k < N; masked for cells
          dens += wsm[wib][(off_sh[wib][i] + 32 * lane) & (32 * NP - 1)];  // out of order (NaN)
      }
      __syncwarp();
    }
    double extra = 0.0;
    if (longs)
      extra = add_heads<N>(R.head, run_sh[wib], lane, reinterpret_cast<double*>(off_sh[wib]));
    if (c > 0 && c < m - 1) {
      if (any && !sparse) {
        double s[N];  // the run's sum, or its tail: N loads in flight (9 000 clk one by one)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int k = N - 1 - i, c0 = r[i].x / SPLAT_CHUNK;
          const double* at = R.sum + (c - H + i + N + 1) * N + k;
          if (c0 < (r[i].y - 1) / SPLAT_CHUNK) at = R.tail + (int64_t)c0 * N + k;
          s[i] = r[i].y > r[i].x ? __ldg(at) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int c1 = (r[i].y - 1) / SPLAT_CHUNK;
          if (r[i].y > r[i].x)
            for (int h = r[i].x / SPLAT_CHUNK + 1; h <= c1; ++h)
              s[i] += R.head[(int64_t)h * N + N - 1 - i];
          dens += s[i];
        }
        dens += extra;
      }
    } else if (c < m) {
      // edge cell: every slot whose clamped index lands here, sources then slots
      int j0 = c == 0 ? 0 : (int)a.ns, j1 = c == 0 ? 0 : (int)a.ns;
      if (c == 0)
        for (int64_t e = -N; e < H; ++e) j1 = max(j1, run[e].y);
      else
        for (int64_t e = m - 1 - H; e <= m + N; ++e) {
          const int2 r = run[e];
          if (r.y > r.x) j0 = min(j0, r.x);
        }
      for (int j = j0; j < j1; ++j) {
        double t;
        const int i0 = clamped_cell<N>(a, visited(a, j), &t);
        double w[N];
        lagrange<N>(t, w);
#pragma unroll
        for (int k = 0; k < N; ++k) {
          int64_t cell = (int64_t)i0 - H + 1 + k;
          cell = cell < 0 ? 0 : (cell > m - 1 ? m - 1 : cell);
          if (cell == c) dens += w[k];
        }
      }
    }
  }
  if (c >= m) return;
  if (a.dens) a.dens[c] = dens;
  else a.packed[c] = make_double2(dens, odd);
}

// The evaluation stage's input: packed[c] from a given density (the sum of
// the splat stages of several source sets).
__global__ void pack_density_kernel(const GridArgs a, const double* __restrict__ density) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < a.m) a.packed[c] = make_double2(density[c], odd_kernel(a, c));
}

// ---------------------------------------------------------------- FFT --
// Unnormalised DFT, forward sign e^{-2 pi i jk/m}, inverse e^{+2 pi i jk/m}
// (the contract of the reference's transform, rustfft).  m = m1*m2 by the
// four-step method; each row transform of length L = 2^LOG (8 <= L <= 2048) is
// a mixed-radix Stockham FFT (radix 8, then one radix-4 or radix-2 stage) by
// L/8 threads of eight elements each.  Thread q loads the elements q + r L/8,
// which are its first butterfly, and ends with the outputs q + r L/8, so the
// first stage takes its inputs, and the last leaves its outputs, in registers;
// only the exchanges between stages go through shared memory (one pad slot per
// 8 elements).  Every twiddle is a table entry, those between the passes the
// product of two, so the rounding is that of a transform with exact twiddles
// (rms error 3.2e-16 at 2^20 points; with a butterfly's twiddles formed as
// powers of one entry 5.8e-16, 3 us less for the two passes).  With the loads,
// the stores and every twiddle staged in shared memory a pass over 2^20 points
// took 36 (columns) and 21 us (rows), now 20 and 13 (16 + 16 MB each way
// through L2); bound by the latency of a CTA's chain of load, four butterflies
// with three exchanges, and store, 3 or 4 CTAs an SM overlapping.
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// The transform's products, fused (two operations fewer, one rounding less).
__device__ __forceinline__ double2 cmulf(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
// v e^{i pi/4 sign}
__device__ __forceinline__ double2 mul_w8(double2 v, double sign) {
  const double h = 0.70710678118654752440;  // sqrt(1/2)
  return make_double2(h * (v.x - sign * v.y), h * (v.y + sign * v.x));
}
// v * (sign * i)
__device__ __forceinline__ double2 mul_si(double2 v, double sign) {
  return make_double2(-sign * v.y, sign * v.x);
}
__device__ __forceinline__ int padi(int i) { return i + (i >> 3); }

// R-point DFTs in registers, W_R = e^{sign 2 pi i/R}.
__device__ __forceinline__ void dft4(double2& v0, double2& v1, double2& v2, double2& v3,
                                     double sign) {
  const double2 t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3);
  const double2 t3 = mul_si(csub(v1, v3), sign);
  v0 = cadd(t0, t2);
  v1 = cadd(t1, t3);
  v2 = csub(t0, t2);
  v3 = csub(t1, t3);
}
__device__ __forceinline__ void dft8(double2* v, double sign) {
  double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  double2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4(e0, e1, e2, e3, sign);
  dft4(o0, o1, o2, o3, sign);
  o1 = mul_w8(o1, sign);
  o2 = mul_si(o2, sign);
  o3 = mul_si(mul_w8(o3, sign), sign);
  v[0] = cadd(e0, o0);
  v[1] = cadd(e1, o1);
  v[2] = cadd(e2, o2);
  v[3] = cadd(e3, o3);
  v[4] = csub(e0, o0);
  v[5] = csub(e1, o1);
  v[6] = csub(e2, o2);
  v[7] = csub(e3, o3);
}

// w or its conjugate: a table entry for the transform's sign.
__device__ __forceinline__ double2 signed_tw(double2 w, double sign) {
  const int flip = __double2hiint(sign) & 0x80000000;
  w.y = __hiloint2double(__double2hiint(w.y) ^ flip, __double2loint(w.y));
  return w;
}

// Stage s >= 1 of a row transform combines Ns = 8^s points with radix R; its
// table holds W_{Ns R}^{k r}, k < Ns, r = 1 .. R - 1, at [r - 1][k] from entry
// stage_off(s) (7 x 8, 7 x 64 and 3 x 512 entries at most).
constexpr int STAGE_TAB = 2040;
__host__ __device__ constexpr int stage_off(int s) { return s <= 1 ? 0 : s == 2 ? 56 : 504; }

__global__ void stage_twiddle_kernel(double2* __restrict__ out, const double2* __restrict__ tw,
                                     int L, int64_t m) {
  const int idx = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int s = idx < 56 ? 1 : idx < 504 ? 2 : 3, Ns = 1 << (3 * s);
  if (idx >= STAGE_TAB || Ns >= L) return;
  const int R = L / Ns < 8 ? L / Ns : 8;
  const int r = (idx - stage_off(s)) / Ns + 1, k = (idx - stage_off(s)) & (Ns - 1);
  if (r < R) out[idx] = tw[(int64_t)k * r * (m / ((int64_t)Ns * R))];
}

// The stages S .. of a row: v holds stage S's inputs for S = 0 (the elements
// q + r L/8 in v[r]), otherwise they are in `row`; the outputs q + r L/8 end in
// v[r].  Every thread of the CTA calls it (the stages hold barriers).
template <int LOG, int S>
__device__ __forceinline__ void row_stages(double2 (&v)[8], double2* row,
                                           const double2* __restrict__ st, int q, double sign) {
  constexpr int L = 1 << LOG, TPR = L / 8, Ns = 1 << (3 * S);
  constexpr int R = L / Ns >= 8 ? 8 : L / Ns, B = 8 / R;
  const int k = q & (Ns - 1);
  if (S > 0) {
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = row[padi(q + r * TPR)];
  }
  // W_{Ns R}^{r (k + at)}
  const auto tw = [&](int r, int at) {
    return signed_tw(__ldg(st + stage_off(S) + (r - 1) * Ns + k + at), sign);
  };
  if constexpr (R == 8) {
    if (S > 0) {
#pragma unroll
      for (int r = 1; r < 8; ++r) v[r] = cmulf(v[r], tw(r, 0));
    }
    dft8(v, sign);
  } else if constexpr (R == 4) {  // butterflies q and q + Ns/2
    const double2 w2 = tw(2, 0);
#pragma unroll
    for (int b = 0; b < B; ++b) {
      v[b + 2] = cmulf(v[b + 2], tw(1, b * (Ns / 2)));
      v[b + 4] = cmulf(v[b + 4], b ? mul_si(w2, sign) : w2);
      v[b + 6] = cmulf(v[b + 6], tw(3, b * (Ns / 2)));
      dft4(v[b], v[b + 2], v[b + 4], v[b + 6], sign);
    }
  } else {  // butterflies q + b Ns/4, b < 4
    const double2 w = tw(1, 0), u = tw(1, Ns / 4);
    v[4] = cmulf(v[4], w);
    v[5] = cmulf(v[5], u);
    v[6] = cmulf(v[6], mul_si(w, sign));
    v[7] = cmulf(v[7], mul_si(u, sign));
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const double2 x = v[b], y = v[b + 4];
      v[b] = cadd(x, y);
      v[b + 4] = csub(x, y);
    }
  }
  if constexpr (Ns * R < L) {
    if (S > 0) __syncthreads();  // the row was read
    const int base = (q - k) * 8 + k;
#pragma unroll
    for (int r = 0; r < 8; ++r) row[padi(base + r * Ns)] = v[r];
    __syncthreads();
  }
}

template <int LOG, int S>
__device__ __forceinline__ void row_rest(double2 (&v)[8], double2* row,
                                         const double2* __restrict__ st, int q, double sign) {
  if constexpr ((1 << (3 * S)) < (1 << LOG)) {
    row_stages<LOG, S>(v, row, st, q, sign);
    row_rest<LOG, S + 1>(v, row, st, q, sign);
  }
}

// Row pitch for G rows side by side: lanes hold G rows of 8/G elements in a
// 128-byte wavefront, so the rows start 8/G slots apart modulo 8.
__host__ __device__ constexpr int row_pitch(int L, int G) {
  return L + (L >> 3) + (G >= 8 ? 1 : 8 / G);
}

// fftplan.rs:43-76: unpack D (density) and K (odd kernel) from the packed
// forward transform's entries k and m - k, multiply, repack as
// Im_hat + i Re_hat.
__device__ __forceinline__ double2 spectral(double2 ck, double2 cn, double ke) {
  const double2 cnc = make_double2(cn.x, -cn.y);
  const double2 s = make_double2(ck.x + cnc.x, ck.y + cnc.y);
  const double2 df = make_double2(ck.x - cnc.x, ck.y - cnc.y);
  const double2 D = make_double2(0.5 * s.x, 0.5 * s.y);
  const double2 K = make_double2(0.5 * df.y, -0.5 * df.x);  // (-0.5 i) * df
  const double2 rh = cmul(D, K);
  return make_double2(D.x * ke - rh.y, D.y * ke + rh.x);
}

// Pass 1: Y[k1*m2 + n2] = W_m^{n2 k1} * sum_n1 x[m2 n1 + n2] W_m1^{n1 k1}, for
// G columns n2 per CTA (G*m1/8 threads), lanes side by side in the columns.
// With ke the input is the spectral product of x, formed on the way in (a
// kernel of its own took 8 us at 2^20).
// Three CTAs an SM: in the 64 registers of four the table entries spill (both
// transforms of 2^19 points 49.8 us, here 48.3; 2^22 336, here 316).
template <int LOG>
__global__ void __launch_bounds__(256, 3) fft_pass1(const double2* __restrict__ x,
                                                    double2* __restrict__ y, int m2, int64_t m,
                                                    const double2* __restrict__ tw,
                                                    const double2* __restrict__ st, double sign,
                                                    const double* __restrict__ ke) {
  extern __shared__ double2 fsm[];
  constexpr int L = 1 << LOG, TPR = L / 8;
  const int G = blockDim.x / TPR, gl = __ffs(G) - 1;
  const int g = threadIdx.x & (G - 1), q = threadIdx.x >> gl;
  const int n2 = blockIdx.x * G + g;
  double2 v[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    v[r] = make_double2(0.0, 0.0);
    const int64_t k = (int64_t)m2 * (q + r * TPR) + n2;
    if (n2 < m2) v[r] = ke ? spectral(x[k], x[(m - k) & (m - 1)], ke[k]) : x[k];
  }
  row_rest<LOG, 0>(v, fsm + g * row_pitch(L, G), st, q, sign);
  if (n2 >= m2) return;
  // The outputs are column n2 at k1 = q + r L/8, their twiddles W_m^{n2 k1} =
  // W^{n2 q} W^{n2 r L/8}: two table entries, the second shared by the column.
  const double2 base = signed_tw(__ldg(tw + (unsigned)(n2 * q)), sign);
  const unsigned step = (unsigned)(n2 * TPR);  // m <= 2^22
  double2* out = y + (int64_t)q * m2 + n2;
  out[0] = cmulf(v[0], base);
#pragma unroll
  for (int r = 1; r < 8; ++r) {
    const double2 w = signed_tw(__ldg(tw + r * step), sign);
    out[(unsigned)(r * TPR * m2)] = cmulf(cmulf(v[r], w), base);
  }
}

// Pass 2: X[k1 + m1 k2] = sum_n2 Y[k1*m2 + n2] W_m2^{n2 k2}, G rows per CTA:
// lanes along the row for the loads and the first stage, side by side in the
// rows for the others and the stores.
template <int LOG>
__global__ void __launch_bounds__(256, 4) fft_pass2(const double2* __restrict__ y,
                                                    double2* __restrict__ x, int m1,
                                                    const double2* __restrict__ st, double sign) {
  extern __shared__ double2 fsm[];
  constexpr int L = 1 << LOG, TPR = L / 8;
  const int G = blockDim.x / TPR, gl = __ffs(G) - 1, Lp = row_pitch(L, G);
  const int k1_0 = blockIdx.x * G;
  double2 v[8];
  {
    const int g = threadIdx.x / TPR, q = threadIdx.x % TPR;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      v[r] = k1_0 + g < m1 ? y[(int64_t)(k1_0 + g) * L + q + r * TPR] : make_double2(0.0, 0.0);
    row_stages<LOG, 0>(v, fsm + g * Lp, st, q, sign);
  }
  const int g = threadIdx.x & (G - 1), q = threadIdx.x >> gl;  // the same for L = 8
  row_rest<LOG, 1>(v, fsm + g * Lp, st, q, sign);
  if (k1_0 + g >= m1) return;
#pragma unroll
  for (int r = 0; r < 8; ++r) x[(int64_t)(k1_0 + g) + (int64_t)m1 * (q + r * TPR)] = v[r];
}

// Transforms shorter than 64 points: direct DFT, one thread per output.
__global__ void dft_small(const double2* __restrict__ x, double2* __restrict__ y, int m,
                          const double2* __restrict__ tw, double sign) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  double2 acc = make_double2(0.0, 0.0);
  for (int n = 0; n < m; ++n) {
    const double2 w = tw[((int64_t)n * k) % m];
    acc = cadd(acc, cmul(x[n], make_double2(w.x, sign * w.y)));
  }
  y[k] = acc;
}

// The spectral product as a pass of its own, where the inverse transform does
// not read the grid itself (Bluestein's form, fewer than 64 points).
__global__ void spectral_kernel(const double2* __restrict__ C, const double* __restrict__ ke,
                                double2* __restrict__ out, int64_t m) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) out[k] = spectral(C[k], C[(m - k) % m], ke[k]);
}

struct InterpArgs {
  const double* q;
  int64_t nq;
  const double2* grid;
  int64_t m;
  double lo;
  Spacing h;
  double inv_m;
  Epilogue epi;
};

// fft5.rs:191-211 interp_at<N> + 440-476: re <- .im, im <- .re, times 1/m.
template <int N>
__global__ void interp_kernel(const InterpArgs a) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.nq) return;
  const double qv = a.q[t];
  double tt;
  const int64_t i0 = cell_of<N>(qv, a.lo, a.h, a.m, &tt);
  double w[N];
  lagrange<N>(tt, w);
  double ra = 0.0, ia = 0.0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    int64_t cell = i0 - N / 2 + 1 + j;
    cell = cell < 0 ? 0 : (cell > a.m - 1 ? a.m - 1 : cell);
    const double2 g = a.grid[cell];
    ia += g.x * w[j];
    ra += g.y * w[j];
  }
  epi_store(a.epi, t, qv, ra * a.inv_m, ia * a.inv_m);
}

// Twiddles (cos 2 pi j/m, sin 2 pi j/m) for j < m.
__global__ void twiddle_kernel(double2* tw, int64_t m) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  double s, c;
  sincospi(2.0 * (double)j / (double)m, &s, &c);
  tw[j] = make_double2(c, s);
}

// fft5.rs:404-416: K_even[k] = (pi/dx) r^|k|, |k| = min(k, m - k),
// r = exp(-2 pi eta/(m dx)).  The power is evaluated directly, not by the
// reference's running product (the two differ by that product's rounding,
// at most |k| ulp).
__global__ void even_kernel_spectrum(double* ke, int64_t m, double ke0, double r) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const int64_t half = m / 2;
  const int64_t kk = k <= half ? k : m - k;
  ke[k] = ke0 * pow(r, (double)kk);
}

// Grids whose size m is not a power of two (a forced fft5 grid_size; the
// reference plans any length through rustfft, fftplan.rs:21-28) take
// Bluestein's chirp-z form over the power-of-two transform of length
// M = next_pow2(2m - 1):  with c_j = e^{i pi j^2/m} and nk = (n^2 + k^2 -
// (k - n)^2)/2,
//   y_k = sum_n x_n e^{s 2 pi i nk/m} = c_k^s sum_n (x_n c_n^s) conj(c^s)_{k-n},
// a circular convolution of length M with the chirp filter, which is
// transformed once per m.  c^s is c for s = +1 and its conjugate for s = -1.

// c_j = e^{i pi (j^2 mod 2m)/m}, j < m; j^2 is exact in 64-bit integers for
// the m this path admits (m <= 2^21).
__global__ void chirp_kernel(double2* c, int64_t m) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const int64_t r = (j * j) % (2 * m);
  double sn, cs;
  sincospi((double)r / (double)m, &sn, &cs);
  c[j] = make_double2(cs, sn);
}

// The forward transform's filter conj(c^{-1})_j = c_j on the circular index
// range (-m, m) of length M, scaled by 1/M (a power of two: exact) so that
// the unnormalised inverse transform of the product is the convolution.
__global__ void chirp_filter_kernel(const double2* __restrict__ c, int64_t m, int64_t M,
                                    double2* __restrict__ b) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  const int64_t j = k < m ? k : (k > M - m ? M - k : -1);
  const double inv = 1.0 / (double)M;
  b[k] = j >= 0 ? make_double2(c[j].x * inv, c[j].y * inv) : make_double2(0.0, 0.0);
}

// a_n = x_n c^s_n for n < m, zero up to M.
__global__ void chirp_in_kernel(const double2* __restrict__ x, const double2* __restrict__ c,
                                int64_t m, int64_t M, double sign, double2* __restrict__ a) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  a[k] = k < m ? cmul(x[k], make_double2(c[k].x, sign * c[k].y)) : make_double2(0.0, 0.0);
}

// a_k *= B_k for the forward transform; for the inverse the filter is the
// conjugate chirp, whose transform is conj(B_{-k mod M}).
__global__ void chirp_mul_kernel(double2* __restrict__ a, const double2* __restrict__ bhat,
                                 int64_t M, int inverse) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  double2 h = bhat[inverse ? (M - k) & (M - 1) : k];
  if (inverse) h.y = -h.y;
  a[k] = cmul(a[k], h);
}

// y_k = c^s_k a_k, k < m.
__global__ void chirp_out_kernel(const double2* __restrict__ a, const double2* __restrict__ c,
                                 int64_t m, double sign, double2* __restrict__ y) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  y[k] = cmul(a[k], make_double2(c[k].x, sign * c[k].y));
}

// Length of the power-of-two (or direct, below 64 points) transform that
// serves a grid of m cells.
int64_t transform_len(int64_t m) {
  if (m < 64 || (m & (m - 1)) == 0) return m;
  return (int64_t)next_pow2((size_t)(2 * m - 1));
}

// Constant tables, cached per call context for the last transform length,
// m and (m, dx, eta); written and read on the context's stream.
struct Tables {
  double2* tw = nullptr;     // twiddles of the transform length, then the
  int64_t tw_m = 0;          // stage twiddles of its two passes [STAGE_TAB] each
  double2* chirp = nullptr;  // Bluestein: c_j (m) and the filter's transform (M)
  double2* bhat = nullptr;
  int64_t bs_m = 0, bs_cap = 0, bhat_cap = 0;
  double* ke = nullptr;
  int64_t ke_cap = 0;
  int64_t ke_m = 0;
  double ke_dx = 0.0, ke_eta = 0.0;
  ~Tables() {
    if (tw) cudaFree(tw);
    if (chirp) cudaFree(chirp);
    if (bhat) cudaFree(bhat);
    if (ke) cudaFree(ke);
  }
};

unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// m = m1 m2, the lengths of the two passes.
void fft_split(int64_t m, int* m1, int* m2) {
  int bits = 0;
  while ((int64_t(1) << bits) < m) ++bits;
  *m1 = 1 << ((bits + 1) / 2);
  *m2 = 1 << (bits / 2);
}

shrk_status fft(double2* buf, double2* tmp, int64_t m, const double2* tw, double sign,
                const char* family, cudaStream_t s);

shrk_status ensure_tables(int64_t m, double dx, double eta, const char* family, cudaStream_t s,
                          Tables** out) {
  Tables& T = ctx_state<Tables>(EXT_FFT_TABLES);
  const int64_t L = transform_len(m);
  if (T.tw_m != L) {
    if (T.tw) SHRK_CUDA(cudaFree(T.tw));
    T.tw = nullptr;
    T.tw_m = 0;
    SHRK_CUDA(cudaMalloc(&T.tw, sizeof(double2) * (L + 2 * STAGE_TAB)));
    twiddle_kernel<<<blocks_for(L, 256), 256, 0, s>>>(T.tw, L);
    SHRK_CUDA(cudaGetLastError());
    if (L >= 64) {
      int m1 = 0, m2 = 0;
      fft_split(L, &m1, &m2);
      stage_twiddle_kernel<<<blocks_for(STAGE_TAB, 256), 256, 0, s>>>(T.tw + L, T.tw, m1, L);
      SHRK_CUDA(cudaGetLastError());
      stage_twiddle_kernel<<<blocks_for(STAGE_TAB, 256), 256, 0, s>>>(T.tw + L + STAGE_TAB, T.tw, m2,
                                                                     L);
      SHRK_CUDA(cudaGetLastError());
    }
    T.tw_m = L;
  }
  if (L != m && T.bs_m != m) {
    T.bs_m = 0;
    if (T.bs_cap < m) {
      if (T.chirp) SHRK_CUDA(cudaFree(T.chirp));
      T.chirp = nullptr;
      T.bs_cap = 0;
      SHRK_CUDA(cudaMalloc(&T.chirp, sizeof(double2) * m));
      T.bs_cap = m;
    }
    if (T.bhat_cap < 2 * L) {  // the filter's transform and its scratch
      if (T.bhat) SHRK_CUDA(cudaFree(T.bhat));
      T.bhat = nullptr;
      T.bhat_cap = 0;
      SHRK_CUDA(cudaMalloc(&T.bhat, sizeof(double2) * 2 * L));
      T.bhat_cap = 2 * L;
    }
    chirp_kernel<<<blocks_for(m, 256), 256, 0, s>>>(T.chirp, m);
    SHRK_CUDA(cudaGetLastError());
    chirp_filter_kernel<<<blocks_for(L, 256), 256, 0, s>>>(T.chirp, m, L, T.bhat);
    SHRK_CUDA(cudaGetLastError());
    SHRK_TRY(fft(T.bhat, T.bhat + L, L, T.tw, -1.0, family, s));
    T.bs_m = m;
  }
  if (T.ke_m != m || T.ke_dx != dx || T.ke_eta != eta) {
    if (T.ke_cap < m) {
      if (T.ke) SHRK_CUDA(cudaFree(T.ke));
      T.ke = nullptr;
      T.ke_cap = 0;
      SHRK_CUDA(cudaMalloc(&T.ke, sizeof(double) * m));
      T.ke_cap = m;
    }
    const double r = std::exp(-2.0 * M_PI * eta / ((double)m * dx));
    even_kernel_spectrum<<<blocks_for(m, 256), 256, 0, s>>>(T.ke, m, M_PI / dx, r);
    SHRK_CUDA(cudaGetLastError());
    T.ke_m = m;
    T.ke_dx = dx;
    T.ke_eta = eta;
  }
  *out = &T;
  return SHRK_OK;
}

// Rows per CTA for a pass over `rows` transforms of length L: as many as fit
// 256 threads (8 elements each), but no more than keeps ~2 CTAs per SM, and at
// least two where they fit, whose neighbouring 16-byte elements fill a sector.
int rows_per_cta(int L, int rows) {
  const int cap = 2048 / L;
  int g = 1;
  while (g * 2 <= cap && (g == 1 || (int64_t)rows / (g * 2) >= 296)) g *= 2;
  return g;
}

struct PassKernels {
  void (*p1)(const double2*, double2*, int, int64_t, const double2*, const double2*, double,
             const double*);
  void (*p2)(const double2*, double2*, int, const double2*, double);
};

PassKernels pass_kernels(int L) {
  switch (L) {
    case 8: return {fft_pass1<3>, fft_pass2<3>};
    case 16: return {fft_pass1<4>, fft_pass2<4>};
    case 32: return {fft_pass1<5>, fft_pass2<5>};
    case 64: return {fft_pass1<6>, fft_pass2<6>};
    case 128: return {fft_pass1<7>, fft_pass2<7>};
    case 256: return {fft_pass1<8>, fft_pass2<8>};
    case 512: return {fft_pass1<9>, fft_pass2<9>};
    case 1024: return {fft_pass1<10>, fft_pass2<10>};
    default: return {fft_pass1<11>, fft_pass2<11>};
  }
}

// src -> dst (which may be src) through tmp, all of m >= 64 points; with ke the
// transform of the spectral product of src, which is then not dst.
shrk_status fft_from(const double2* src, double2* dst, double2* tmp, int64_t m, const double2* tw,
                     double sign, const double* ke, const char* family, cudaStream_t s) {
  int m1 = 0, m2 = 0;
  fft_split(m, &m1, &m2);
  {
    const int G = rows_per_cta(m1, m2);
    LaunchScope ls(family, s);
    pass_kernels(m1).p1<<<blocks_for(m2, G), G * (m1 >> 3), sizeof(double2) * G * row_pitch(m1, G),
                          s>>>(src, tmp, m2, m, tw, tw + m, sign, ke);
    SHRK_CUDA(cudaGetLastError());
  }
  {
    const int G = rows_per_cta(m2, m1);
    LaunchScope ls(family, s);
    pass_kernels(m2).p2<<<blocks_for(m1, G), G * (m2 >> 3), sizeof(double2) * G * row_pitch(m2, G),
                          s>>>(tmp, dst, m1, tw + m + STAGE_TAB, sign);
    SHRK_CUDA(cudaGetLastError());
  }
  return SHRK_OK;
}

shrk_status fft(double2* buf, double2* tmp, int64_t m, const double2* tw, double sign,
                const char* family, cudaStream_t s) {
  if (m < 64) {
    LaunchScope ls(family, s);
    dft_small<<<1, 64, 0, s>>>(buf, tmp, (int)m, tw, sign);
    SHRK_CUDA(cudaGetLastError());
    SHRK_CUDA(cudaMemcpyAsync(buf, tmp, sizeof(double2) * m, cudaMemcpyDeviceToDevice, s));
    return SHRK_OK;
  }
  return fft_from(buf, buf, tmp, m, tw, sign, nullptr, family, s);
}

// Unnormalised DFT of the m-cell grid in buf (sign -1 forward, +1 inverse):
// the power-of-two transform in place, or Bluestein's form through the
// M-point work buffers wa and wt.
shrk_status dft(double2* buf, int64_t m, const Tables* T, double sign, double2* wa, double2* wt,
                const char* family, cudaStream_t s) {
  const int64_t M = transform_len(m);
  if (M == m) return fft(buf, wt, m, T->tw, sign, family, s);
  {
    LaunchScope ls(family, s);
    chirp_in_kernel<<<blocks_for(M, 256), 256, 0, s>>>(buf, T->chirp, m, M, sign, wa);
    SHRK_CUDA(cudaGetLastError());
  }
  SHRK_TRY(fft(wa, wt, M, T->tw, -1.0, family, s));
  {
    LaunchScope ls(family, s);
    chirp_mul_kernel<<<blocks_for(M, 256), 256, 0, s>>>(wa, T->bhat, M, sign > 0.0 ? 1 : 0);
    SHRK_CUDA(cudaGetLastError());
  }
  SHRK_TRY(fft(wa, wt, M, T->tw, +1.0, family, s));
  {
    LaunchScope ls(family, s);
    chirp_out_kernel<<<blocks_for(m, 256), 256, 0, s>>>(wa, T->chirp, m, sign, buf);
    SHRK_CUDA(cudaGetLastError());
  }
  return SHRK_OK;
}

// One grid: stencil width, size, origin and spacing, and the launch families
// its kernels are timed under.
struct GridPlan {
  int order;
  int64_t m;
  double lo, dx;
  const char* fam_splat;
  const char* fam_fft;
  const char* fam_spectral;
  const char* fam_interp;
};

template <int N>
shrk_status eval_grid(double2* A, double2* B, double2* Wa, double2* Wt, const Tables* T,
                      const double* d_q, int64_t nq, const GridPlan& g, const Epilogue& epi,
                      cudaStream_t s);

// The whole grid convolution, or one of its two stages: with dens_out the
// splat alone (the density of the sources into dens_out[m], nothing else);
// with dens_in the evaluation alone from that density (no sources read).
template <int N>
shrk_status run_grid(const double* d_q, int64_t nq, const double* d_src, int64_t ns, double eta,
                     const GridPlan& g, const Epilogue& epi, cudaStream_t s,
                     const double* dens_in, double* dens_out) {
  const int64_t m = g.m;
  Tables* T = nullptr;
  if (!dens_out) SHRK_TRY(ensure_tables(m, g.dx, eta, g.fam_fft, s, &T));
  // slot 11: A (packed grid) | B (product) | Wt | Wa, the last two of the
  // transform length (Wa only for a Bluestein grid)
  const int64_t L = transform_len(m);
  void* w = nullptr;
  SHRK_TRY(scratch_get(11, sizeof(double2) * (size_t)(2 * m + (L == m ? L : 2 * L)), &w));
  double2* A = (double2*)w;
  double2* B = A + m;
  double2* Wt = B + m;
  double2* Wa = Wt + L;
  GridArgs ga{d_src, ns, g.dx < 0.0 ? 1 : 0, g.lo, spacing(g.dx), eta, m, A, dens_out};
  if (dens_in) {
    LaunchScope ls(g.fam_splat, s);
    pack_density_kernel<<<blocks_for(m, 256), 256, 0, s>>>(ga, dens_in);
    SHRK_CUDA(cudaGetLastError());
    return eval_grid<N>(A, B, Wa, Wt, T, d_q, nq, g, epi, s);
  }
  if (ns == 0) {  // no sources: a zero density
    if (dens_out) SHRK_CUDA(cudaMemsetAsync(dens_out, 0, sizeof(double) * m, s));
    return SHRK_OK;
  }
  // slot 24: runs [K], K = m + 2N + 2 keys from -N - 1 | run sums [K][N] |
  // chunk heads and tails [C][N] each, C = ceil(ns / SPLAT_CHUNK)
  const int64_t n_keys = m + 2 * N + 2;
  const int64_t chunks = (ns + SPLAT_CHUNK - 1) / SPLAT_CHUNK;
  const size_t run_bytes = (sizeof(int2) * (size_t)n_keys + 255) & ~(size_t)255;
  void* sw = nullptr;
  SHRK_TRY(scratch_get(24, run_bytes + sizeof(double) * N * (size_t)(n_keys + 2 * chunks), &sw));
  Runs runs;
  runs.run = (int2*)sw;
  runs.sum = (double*)((char*)sw + run_bytes);
  runs.head = runs.sum + (size_t)N * n_keys;
  runs.tail = runs.head + (size_t)N * chunks;
  SHRK_CUDA(cudaMemsetAsync(runs.run, 0, sizeof(int2) * (size_t)n_keys, s));
  {
    LaunchScope ls(g.fam_splat, s);
    splat_kernel<N><<<(unsigned)chunks, SPLAT_NT, sizeof(double) * N * (SPLAT_CHUNK + 1), s>>>(
        ga, runs);
    SHRK_CUDA(cudaGetLastError());
  }
  {
    LaunchScope ls(g.fam_splat, s);
    pack_kernel<N><<<blocks_for(m, 256), 256, 0, s>>>(ga, runs);
    SHRK_CUDA(cudaGetLastError());
  }
  if (dens_out) return SHRK_OK;
  return eval_grid<N>(A, B, Wa, Wt, T, d_q, nq, g, epi, s);
}

// Forward transform of the packed grid A, spectral product into B, inverse
// transform, interpolation at the queries with the epilogue.
template <int N>
shrk_status eval_grid(double2* A, double2* B, double2* Wa, double2* Wt, const Tables* T,
                      const double* d_q, int64_t nq, const GridPlan& g, const Epilogue& epi,
                      cudaStream_t s) {
  const int64_t m = g.m;
  SHRK_TRY(dft(A, m, T, -1.0, Wa, Wt, g.fam_fft, s));
  if (m >= 64 && transform_len(m) == m) {
    SHRK_TRY(fft_from(A, B, Wt, m, T->tw, +1.0, T->ke, g.fam_fft, s));
  } else {
    {
      LaunchScope ls(g.fam_spectral, s);
      spectral_kernel<<<blocks_for(m, 256), 256, 0, s>>>(A, T->ke, B, m);
      SHRK_CUDA(cudaGetLastError());
    }
    SHRK_TRY(dft(B, m, T, +1.0, Wa, Wt, g.fam_fft, s));
  }
  InterpArgs ia{d_q, nq, B, m, g.lo, spacing(g.dx), 1.0 / (double)m, epi};
  {
    LaunchScope ls(g.fam_interp, s);
    interp_kernel<N><<<blocks_for(nq, 256), 256, 0, s>>>(ia);
    SHRK_CUDA(cudaGetLastError());
  }
  return SHRK_OK;
}

shrk_status run_grid_order(const double* d_q, int64_t nq, const double* d_src, int64_t ns,
                           double eta, const GridPlan& g, const Epilogue& epi, cudaStream_t s,
                           const double* dens_in = nullptr, double* dens_out = nullptr) {
  // the runs hold 32-bit source indices
  if (ns > (int64_t)INT32_MAX) {
    set_error("fft grid methods: at most 2^31 - 1 sources per call");
    return SHRK_EINVAL;
  }
  switch (g.order) {
    case 2: return run_grid<2>(d_q, nq, d_src, ns, eta, g, epi, s, dens_in, dens_out);
    case 4: return run_grid<4>(d_q, nq, d_src, ns, eta, g, epi, s, dens_in, dens_out);
    case 6: return run_grid<6>(d_q, nq, d_src, ns, eta, g, epi, s, dens_in, dens_out);
    case 8: return run_grid<8>(d_q, nq, d_src, ns, eta, g, epi, s, dens_in, dens_out);
    default:
      set_error("fft5: the stencil order must be 2, 4, 6 or 8 nodes");
      return SHRK_EINVAL;
  }
}

}  // namespace

// nufft.rs:106-126 grid_size_for_range (a descending spectrum's range, and so the
// target, may be negative: the smallest grid).
size_t nufft_grid_size(double raw_range, double eta) {
  double pad = std::max(NUFFT_PAD_ETA_MULT * eta, NUFFT_PAD_RANGE_FRAC * raw_range);
  double range = raw_range + 2.0 * pad;
  size_t max_grid = std::max(std::max(NUFFT_MAX_GRID, NUFFT_MIN_GRID), (size_t)2);
  double target = NUFFT_RESOLUTION * range / eta;
  target = std::isfinite(target) ? std::min(target, (double)max_grid) : (double)max_grid;
  return std::min(next_pow2(std::max(sat_usize(std::ceil(target)), NUFFT_MIN_GRID)), max_grid);
}

// fft5.rs:339-361: pad = max(pad_eta_mult eta, pad_range_frac raw_range),
// m = next_pow2(min(max(ceil(8 range/eta), 8p), 2^20)), at least 2.
size_t fft5_grid_size(double lo_raw, double hi_raw, size_t p, double eta, double pad_eta_mult,
                      double pad_range_frac) {
  const double raw_range = hi_raw - lo_raw;
  const double pad = std::max(pad_eta_mult * eta, pad_range_frac * raw_range);
  const double lo = lo_raw - pad, hi = hi_raw + pad;
  const double range = hi - lo;
  size_t min_grid = sat_usize(std::ceil(8.0 * range / eta));
  const size_t p8 = p > SIZE_MAX / 8 ? SIZE_MAX : 8 * p;
  min_grid = std::min(std::max(min_grid, p8), FFT5_MAX_AUTO_GRID);
  return std::max(next_pow2(min_grid), (size_t)2);
}

// fft5.rs:339-361 with the NUFFT options (m fixed by the policy).
void nufft_geometry(double lo_raw, double hi_raw, double eta, int64_t* m, double* lo,
                    double* dx) {
  const double raw_range = hi_raw - lo_raw;
  *m = (int64_t)std::max(nufft_grid_size(raw_range, eta), (size_t)2);
  const double pad = std::max(NUFFT_PAD_ETA_MULT * eta, NUFFT_PAD_RANGE_FRAC * raw_range);
  *lo = lo_raw - pad;
  const double hi = hi_raw + pad;
  *dx = (hi - *lo) / (double)*m;
}

namespace {
GridPlan nufft_plan(int64_t m, double lo, double dx) {
  return GridPlan{4, m, lo, dx, "nufft_splat", "nufft_fft", "nufft_spectral", "nufft_interp"};
}
}  // namespace

shrk_status nufft_points(const double* d_q, int64_t nq, const double* d_src, int64_t ns,
                         double lo_raw, double hi_raw, double eta, const Epilogue& epi,
                         cudaStream_t s) {
  if (nq <= 0 || ns <= 0) return SHRK_OK;
  int64_t m = 0;
  double lo = 0.0, dx = 0.0;
  nufft_geometry(lo_raw, hi_raw, eta, &m, &lo, &dx);
  return run_grid_order(d_q, nq, d_src, ns, eta, nufft_plan(m, lo, dx), epi, s);
}

shrk_status nufft_density(const double* d_sorted_src, int64_t ns, int64_t m, double lo, double dx,
                          double* d_density, cudaStream_t s) {
  return run_grid_order(nullptr, 0, d_sorted_src, ns, 0.0, nufft_plan(m, lo, dx), Epilogue{}, s,
                        nullptr, d_density);
}

shrk_status nufft_eval(const double* d_density, int64_t m, double lo, double dx, double eta,
                       const double* d_q, int64_t nq, const Epilogue& epi, cudaStream_t s) {
  if (nq <= 0) return SHRK_OK;
  return run_grid_order(d_q, nq, nullptr, 0, eta, nufft_plan(m, lo, dx), epi, s, d_density,
                        nullptr);
}

shrk_status fft5_points(const double* d_q, int64_t nq, const double* d_src, int64_t ns,
                        double lo_raw, double hi_raw, double eta, const Fft5Opts& o,
                        const Epilogue& epi, cudaStream_t s) {
  if (nq <= 0 || ns <= 0) return SHRK_OK;
  const size_t m = o.m_override ? std::max(o.m_override, (size_t)2)
                                : fft5_grid_size(lo_raw, hi_raw, (size_t)ns, eta, o.pad_eta_mult,
                                                 o.pad_range_frac);
  if (m > (size_t)FFT_MAX_M || ((m & (m - 1)) != 0 && m > (size_t)FFT_MAX_M / 2)) {
    set_error("fft5: the grid size must be at most 2^22, or 2^21 when it is not a power of "
              "two (got " + std::to_string(m) + ")");
    return SHRK_ENOTIMPL;
  }
  const double raw_range = hi_raw - lo_raw;
  const double pad = std::max(o.pad_eta_mult * eta, o.pad_range_frac * raw_range);
  const double lo = lo_raw - pad, hi = hi_raw + pad;
  const double range = hi - lo;
  GridPlan g{o.order, (int64_t)m, lo, range / (double)m, "fft5_splat", "fft5_fft",
             "fft5_spectral", "fft5_interp"};
  return run_grid_order(d_q, nq, d_src, ns, eta, g, epi, s);
}

}  // namespace shrk
