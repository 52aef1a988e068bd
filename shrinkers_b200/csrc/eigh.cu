// Dense symmetric eigendecomposition and FP64 GEMM on sm_100a, for the matrix
// front-end (src/pipeline/mod.rs:502-585 symmetric_eigh; the reference runs a
// cyclic Jacobi iteration, and its docs name LAPACK's dsyevd as the fast
// path).  Written for the GPU instead of restating Jacobi:
//
//   1. tridiagonalisation  Householder reflections H_j = I - beta_j v_j v_j^T,
//                          one cooperative persistent kernel with the (full,
//                          symmetric) trailing matrix in shared memory: per
//                          column one walk applies the reflector and forms the
//                          next product, one exchange of vectors through L2
//                          and one grid barrier.  Above 2 048 rows a kernel
//                          that walks the matrix in global memory runs first.
//   2. eigenvalues         the tridiagonal T splits where an off-diagonal is
//                          negligible; each eigenvalue of each unreduced block
//                          by multisection on Sturm counts (8 to 32 probes a
//                          step), a warp serving several eigenvalues.
//   3. eigenvectors of T   inverse iteration (LU with partial pivoting,
//                          three solves from a fixed pseudo-random start),
//                          one thread per cluster of eigenvalues closer than
//                          CLUSTER_TOL ||T||, modified Gram-Schmidt inside a
//                          cluster; then as many Newton-Schulz steps
//                          Z <- Z (3I - Z^T Z)/2 on the whole basis as take
//                          the remaining O(eps ||T|| / gap) overlaps of close
//                          eigenvectors to rounding level.
//   4. back-transformation U = H_0 ... H_{p-3} Z in blocks of NB reflectors,
//                          each (I - Y T Y^T) in compact WY form, all blocks'
//                          T formed at once, then two GEMMs a block.
//
// The GEMM (dgemm): 128 x 128 tiles on the FP64 tensor instruction, the work
// of a product cut in as many equal runs as there are SMs; a 64 x 64 SIMT form
// for small products.
#include "common.cuh"
#include "internal.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

namespace shrk {

namespace cg = cooperative_groups;

namespace {

// ------------------------------------------------------------------ GEMM --
constexpr int GT = 64;   // output tile
constexpr int GK = 16;   // k per shared-memory stage

// Split-K: CTA z of gridDim.z sums k in [z kz, (z+1) kz) and, when the grid
// has several, writes alpha times its partial product to its own m x n slab
// of C (ldc = m, beta = 0); dgemm then adds the slabs in a fixed order.
template <bool TA, bool TB>
__global__ void __launch_bounds__(256) dgemm_kernel(int m, int n, int k, int kz, double alpha,
                                                    const double* __restrict__ A, int64_t lda,
                                                    const double* __restrict__ B, int64_t ldb,
                                                    double beta, double* __restrict__ C,
                                                    int64_t ldc, int lower) {
  if (lower && blockIdx.y > blockIdx.x) return;  // a tile wholly above the diagonal
  const int kb = blockIdx.z * kz, ke = min(k, kb + kz);
  if (gridDim.z > 1) C += (int64_t)blockIdx.z * m * n;
  __shared__ double As[GK][GT + 1];  // As[kk][i] = op(A)[i0 + i, k0 + kk]
  __shared__ double Bs[GK][GT + 1];  // Bs[kk][j] = op(B)[k0 + kk, j0 + j]
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i0 = blockIdx.x * GT, j0 = blockIdx.y * GT;
  double acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
  for (int k0 = kb; k0 < ke; k0 += GK) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int t = threadIdx.x + it * 256;
      int i, kk;
      if (!TA) { i = t & 63; kk = t >> 6; }   // A(i, kk) contiguous in i
      else { kk = t & 15; i = t >> 4; }       // A(kk, i) contiguous in kk
      const int gi = i0 + i, gk = k0 + kk;
      double v = 0.0;
      if (gi < m && gk < ke) v = !TA ? A[gi + (int64_t)gk * lda] : A[gk + (int64_t)gi * lda];
      As[kk][i] = v;
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int t = threadIdx.x + it * 256;
      int j, kk;
      if (!TB) { kk = t & 15; j = t >> 4; }   // B(kk, j) contiguous in kk
      else { j = t & 63; kk = t >> 6; }       // B(j, kk) contiguous in j
      const int gj = j0 + j, gk = k0 + kk;
      double v = 0.0;
      if (gj < n && gk < ke) v = !TB ? B[gk + (int64_t)gj * ldb] : B[gj + (int64_t)gk * ldb];
      Bs[kk][j] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      double a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = As[kk][tx + 16 * r];
#pragma unroll
      for (int c = 0; c < 4; ++c) b[c] = Bs[kk][ty + 16 * c];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int gj = j0 + ty + 16 * c;
    if (gj >= n) continue;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int gi = i0 + tx + 16 * r;
      if (gi >= m) continue;
      double* cp = C + gi + (int64_t)gj * ldc;
      *cp = beta == 0.0 ? alpha * acc[r][c] : fma(alpha, acc[r][c], beta * *cp);
    }
  }
}

// The large-problem form: 128 x 128 outputs per CTA of 256 threads on the
// FP64 tensor path (mma.sync m8n8k4 .f64; tcgen05 has no FP64 kind): each
// warp owns a 32 x 64 block, 4 x 8 tiles of 8 x 8 with two accumulators a
// lane; k staged 8 at a time through shared memory, two stages in flight
// (the next stage's global loads are issued before this stage's MMAs).  Rows
// of the staged tiles are 136 doubles apart (16 words mod 32 banks), so a
// fragment load -- 4 k rows x 8 consecutive entries -- takes the two
// wavefronts a 64-bit warp load needs and no more.
constexpr int GT2 = 128, GK2 = 8, GP2 = GT2 + 8;

// D = A B + D for one 8 x 8 x 4 FP64 tile: lane l holds A[l/4][l%4],
// B[l%4][l/4] and D[l/4][2(l%4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// One 128 x 128 tile of op(A) op(B) at (i0, j0) over k in [kb, ke).
struct GemmStage {
  double As[2][GK2][GP2];  // As[kk][i] = op(A)[i0 + i, k0 + kk]
  double Bs[2][GK2][GP2];  // Bs[kk][j] = op(B)[k0 + kk, j0 + j]
};

template <bool TA, bool TB>
__device__ __forceinline__ void gemm_tile(GemmStage& st, int m, int n, int kb, int ke, int i0,
                                          int j0, const double* __restrict__ A, int64_t lda,
                                          const double* __restrict__ B, int64_t ldb,
                                          double (&acc)[4][8][2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wi = (warp & 3) * 32, wj = (warp >> 2) * 64;  // the warp's block
  const int fr = lane >> 2, fk = lane & 3;                 // fragment row / k
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[r][c][0] = acc[r][c][1] = 0.0;
  double ra[4], rb[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int t = threadIdx.x + it * 256;
      int i, kk;
      if (!TA) { i = t & 127; kk = t >> 7; }  // A(i, kk) contiguous in i
      else { kk = t & 7; i = t >> 3; }        // A(kk, i) contiguous in kk
      const int gi = i0 + i, gk = k0 + kk;
      ra[it] = (gi < m && gk < ke) ? (!TA ? A[gi + (int64_t)gk * lda] : A[gk + (int64_t)gi * lda])
                                   : 0.0;
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int t = threadIdx.x + it * 256;
      int j, kk;
      if (!TB) { kk = t & 7; j = t >> 3; }    // B(kk, j) contiguous in kk
      else { j = t & 127; kk = t >> 7; }      // B(j, kk) contiguous in j
      const int gj = j0 + j, gk = k0 + kk;
      rb[it] = (gj < n && gk < ke) ? (!TB ? B[gk + (int64_t)gj * ldb] : B[gj + (int64_t)gk * ldb])
                                   : 0.0;
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int t = threadIdx.x + it * 256;
      if (!TA) st.As[buf][t >> 7][t & 127] = ra[it];
      else st.As[buf][t & 7][t >> 3] = ra[it];
      if (!TB) st.Bs[buf][t & 7][t >> 3] = rb[it];
      else st.Bs[buf][t >> 7][t & 127] = rb[it];
    }
  };
  fetch(kb);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = kb; k0 < ke; k0 += GK2) {
    const bool more = k0 + GK2 < ke;
    if (more) fetch(k0 + GK2);
#pragma unroll
    for (int k4 = 0; k4 < GK2; k4 += 4) {
      double a[4], b[8];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = st.As[buf][k4 + fk][wi + 8 * r + fr];
#pragma unroll
      for (int c = 0; c < 8; ++c) b[c] = st.Bs[buf][k4 + fk][wj + 8 * c + fr];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) mma_f64(acc[r][c][0], acc[r][c][1], a[r], b[c]);
    }
    if (more) {
      stash(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
}

// C(i, j) = alpha * tile + beta C (beta = 0: C is not read).  C's entries are
// read sixteen at a time before any is written (one after the other, as the
// compiler must keep them, they were 64 L2 round trips: 25 us a tile).
__device__ __forceinline__ void gemm_store(int m, int n, int i0, int j0, double alpha,
                                           const double (&acc)[4][8][2], double beta, double* C,
                                           int64_t ldc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wi = (warp & 3) * 32, wj = (warp >> 2) * 64, fr = lane >> 2, fk = lane & 3;
#pragma unroll
  for (int c0 = 0; c0 < 8; c0 += 2) {
    double old[2][2][4];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int gj = j0 + wj + 8 * (c0 + c) + 2 * fk + h, gi = i0 + wi + 8 * r + fr;
          old[c][h][r] = beta != 0.0 && gi < m && gj < n ? C[gi + (int64_t)gj * ldc] : 0.0;
        }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int gj = j0 + wj + 8 * (c0 + c) + 2 * fk + h, gi = i0 + wi + 8 * r + fr;
          if (gi >= m || gj >= n) continue;
          const double v = acc[r][c0 + c][h];
          C[gi + (int64_t)gj * ldc] =
              beta == 0.0 ? alpha * v : fma(alpha, v, beta * old[c][h][r]);
        }
  }
}

// The tiles' k steps (GK2 each) numbered tile after tile, CTA c taking the
// c-th of gridDim.x equal runs, so that every SM works to the end whatever the
// number of tiles (2048^3 is 256 tiles: two waves of 148, the second a third
// empty).  A run crosses whole tiles, written straight to C, and at most one
// tile's tail and one tile's head, kept in slots 2 c and 2 c + 1 of the
// workspace; dgemm_fixup_kernel adds a divided tile's parts in CTA order.
struct GemmRuns {
  int tm, tn;      // tiles along m and n
  int lower;       // only the tiles on or below the diagonal (tm = tn)
  int ksteps;      // steps a tile
  int64_t total;   // steps in all
  int64_t per;     // CTA c: [c per + min(c, rem), ...): the first rem have one more
  int rem;

  __host__ __device__ int64_t first(int64_t c) const { return c * per + (c < rem ? c : rem); }
  __host__ __device__ int cta_of(int64_t step) const {
    const int64_t head = (int64_t)rem * (per + 1);
    return (int)(step < head ? step / (per + 1) : rem + (step - head) / per);
  }
  // tile t -> (ti, tj), column by column
  __host__ __device__ void place(int t, int& ti, int& tj) const {
    if (!lower) {
      ti = t % tm;
      tj = t / tm;
      return;
    }
    tj = 0;
    while (t >= tm - tj) t -= tm - tj++;
    ti = tj + t;
  }
};

constexpr int GEMM_SLOT = GT2 * GT2;  // doubles of a partial tile, column-major

template <bool TA, bool TB>
__global__ void __launch_bounds__(256, 1) dgemm_big_kernel(GemmRuns g, int m, int n, int k,
                                                           double alpha,
                                                           const double* __restrict__ A,
                                                           int64_t lda,
                                                           const double* __restrict__ B,
                                                           int64_t ldb, double beta, double* C,
                                                           int64_t ldc, double* ws) {
  __shared__ GemmStage st;
  const int64_t s0 = g.first(blockIdx.x), s1 = g.first((int64_t)blockIdx.x + 1);
  for (int64_t s = s0; s < s1;) {
    const int t = (int)(s / g.ksteps), ks = (int)(s - (int64_t)t * g.ksteps);
    const int ke = (int)min((int64_t)g.ksteps, ks + (s1 - s));
    int ti, tj;
    g.place(t, ti, tj);
    double acc[4][8][2];
    __syncthreads();  // the last tile's readers are done with the stage
    gemm_tile<TA, TB>(st, m, n, ks * GK2, min(k, ke * GK2), ti * GT2, tj * GT2, A, lda, B, ldb,
                      acc);
    if (ks == 0 && ke == g.ksteps)
      gemm_store(m, n, ti * GT2, tj * GT2, alpha, acc, beta, C, ldc);
    else
      gemm_store(GT2, GT2, 0, 0, 1.0, acc, 0.0,
                 ws + (int64_t)(2 * blockIdx.x + (s == s0 ? 0 : 1)) * GEMM_SLOT, GT2);
    s += ke - ks;
  }
}

// The divided tiles: a CTA adds 2 048 entries of one tile, each thread its
// eight side by side, so that eight loads of a part are in flight (entry after
// entry, the parts of each one after the other, was a chain of L2 latencies:
// 15.7 us at p = 501, 18 at 2 048; now 10 and 13).
__global__ void __launch_bounds__(256) dgemm_fixup_kernel(GemmRuns g, int m, int n, double alpha,
                                                          double beta, double* __restrict__ C,
                                                          int64_t ldc,
                                                          const double* __restrict__ ws) {
  const int t = blockIdx.x;
  const int64_t a = (int64_t)t * g.ksteps;
  const int c0 = g.cta_of(a), c1 = g.cta_of(a + g.ksteps - 1);
  if (c0 == c1) return;
  int ti, tj;
  g.place(t, ti, tj);
  const double* p0 = ws + (int64_t)(2 * c0 + (g.first(c0) == a ? 0 : 1)) * GEMM_SLOT;
  const int e0 = blockIdx.y * 2048 + threadIdx.x;
  double v[8], old[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int e = e0 + 256 * u;
    const int gi = ti * GT2 + (e & (GT2 - 1)), gj = tj * GT2 + e / GT2;
    v[u] = p0[e];
    old[u] = beta != 0.0 && gi < m && gj < n ? C[gi + (int64_t)gj * ldc] : 0.0;
  }
#pragma unroll 2
  for (int c = c0 + 1; c <= c1; ++c) {
    const double* pc = ws + (int64_t)2 * c * GEMM_SLOT + e0;
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] += pc[256 * u];
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int e = e0 + 256 * u;
    const int gi = ti * GT2 + (e & (GT2 - 1)), gj = tj * GT2 + e / GT2;
    if (gi < m && gj < n)
      C[gi + (int64_t)gj * ldc] = beta == 0.0 ? alpha * v[u] : fma(alpha, v[u], beta * old[u]);
  }
}

// C = sum_z slab[z] + beta C, the split-K slabs added in order.
__global__ void dgemm_reduce_kernel(const double* __restrict__ ws, int splits, int m, int n,
                                    double beta, double* __restrict__ C, int64_t ldc) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)m * n) return;
  const int64_t i = idx % m, j = idx / m;
  double t = 0.0;
  for (int z = 0; z < splits; ++z) t += ws[(int64_t)z * m * n + idx];
  double* cp = C + i + j * ldc;
  *cp = beta == 0.0 ? t : t + beta * *cp;
}

// -------------------------------------------------------- tridiagonalise --
struct TriArgs {
  double* A;        // p x p column-major, symmetric (both triangles)
  int64_t p;
  double* d;        // [p] diagonal of T
  double* e;        // [p] off-diagonal of T (e[j] couples j and j+1)
  double* vhead;    // [p] first entry v_{j+1} of reflector j
  double* beta;     // [p] beta_j (0: no reflection)
  double* pv;       // [p] p = beta A22 v
  double* part;     // [gridDim.x] per-block partial sums of p^T v
  double* scal;     // [2] norm^2 and first entry of the next column below the diagonal
};

constexpr int TRI_NT = 512;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Norm^2 and first entry of A[c+1 .. p-1, c] by one warp; lane 0 writes them
// (and the final diagonal entry d[c]).
__device__ __forceinline__ void column_tail(const TriArgs& a, int64_t c, int lane) {
  const int64_t p = a.p;
  const double* col = a.A + c * p;
  double s = 0.0;
  for (int64_t k = c + 1 + lane; k < p; k += 32) s += col[k] * col[k];
  s = warp_sum(s);
  if (lane == 0) {
    a.scal[0] = s;
    a.scal[1] = c + 1 < p ? col[c + 1] : 0.0;
    a.d[c] = col[c];
  }
}

__global__ void __launch_bounds__(TRI_NT, 1) tridiag_kernel(const TriArgs a) {
  cg::grid_group grid = cg::this_grid();
  __shared__ double s_red[TRI_NT / 32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  constexpr int WPB = TRI_NT / 32;
  const int64_t gw = (int64_t)blockIdx.x * WPB + wib;  // global warp: owns columns gw mod nw
  const int64_t nw = (int64_t)gridDim.x * WPB;
  const int64_t p = a.p;
  double* A = a.A;
  if (gw == 0) column_tail(a, 0, lane);
  grid.sync();
  for (int64_t j = 0; j + 2 < p; ++j) {
    // the reflector of column j, from the norm its owner left in scal
    const double norm2 = a.scal[0], x0 = a.scal[1];
    const double sig = norm2 - x0 * x0;
    double beta = 0.0, v0 = x0;
    if (sig > 0.0) {
      const double nrm = sqrt(norm2);
      const double alpha = x0 >= 0.0 ? -nrm : nrm;
      v0 = x0 - alpha;
      beta = 2.0 / (sig + v0 * v0);
      if (gw == 0 && lane == 0) a.e[j] = alpha;
    } else if (gw == 0 && lane == 0) {
      a.e[j] = x0;  // already reduced: H_j = I
    }
    if (gw == 0 && lane == 0) {
      a.vhead[j] = v0;
      a.beta[j] = beta;
    }
    const double* vcol = A + j * p;  // v_k = vcol[k] for k >= j + 2
    const int64_t k0 = j + 1;
    // (1) p = beta A22 v over the owned columns, and p^T v
    double dot = 0.0;
    if (beta != 0.0) {
      int64_t c = k0 + ((gw - k0) % nw + nw) % nw;
      for (; c < p; c += nw) {
        const double* col = A + c * p;
        double s = 0.0;
        for (int64_t k = k0 + lane; k < p; k += 32) {
          const double vk = k == k0 ? v0 : vcol[k];
          s = fma(col[k], vk, s);
        }
        s = warp_sum(s) * beta;
        if (lane == 0) a.pv[c] = s;
        dot = fma(s, c == k0 ? v0 : vcol[c], dot);
      }
    }
    if (lane == 0) s_red[wib] = dot;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < WPB; ++w) t += s_red[w];
      a.part[blockIdx.x] = t;
    }
    grid.sync();
    // (2) A22 -= v w^T + w v^T, w = p - (beta/2)(p^T v) v, by owned columns;
    // the owner of column j+1 then measures the next column
    if (beta != 0.0) {
      double g = 0.0;
      for (int b = lane; b < (int)gridDim.x; b += 32) g += a.part[b];
      const double K = 0.5 * beta * warp_sum(g);
      int64_t c = k0 + ((gw - k0) % nw + nw) % nw;
      for (; c < p; c += nw) {
        double* col = A + c * p;
        const double vc = c == k0 ? v0 : vcol[c];
        const double wc = a.pv[c] - K * vc;
        for (int64_t k = k0 + lane; k < p; k += 32) {
          const double vk = k == k0 ? v0 : vcol[k];
          const double wk = a.pv[k] - K * vk;
          col[k] = col[k] - (vk * wc + wk * vc);
        }
      }
    }
    if (gw == k0 % nw) {
      __syncwarp();
      column_tail(a, k0, lane);
    }
    grid.sync();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (p >= 2) a.e[p - 2] = a.scal[1];
    a.d[p - 1] = A[(p - 1) + (p - 1) * p];
    if (p == 1) a.d[0] = A[0];
  }
}


// The same reduction with ONE grid barrier per column.  Phase j applies
// reflector j to the trailing columns and, in the same pass over each
// column, forms the next product p_{j+1} = beta_{j+1} A^{(j+1)} v_{j+1}.
// That needs v_{j+1} at the start of the phase: every CTA derives it itself
// from the stale column j+1 and the previous phase's p_j (w = p_j - K v_j),
// bit-identically in every CTA (same reads, same reduction order), into its
// own buffer.  Column j+1 is then never written: reflector j+1 goes to row
// j+1 of the upper triangle (a part no later phase reads), and only rows
// >= j+2 of the trailing columns are updated.  p and the partial sums of
// p^T v alternate between two buffers.
struct Tri1Args {
  double* A;       // p x p column-major, symmetric (both triangles)
  int64_t p;
  double* d;
  double* e;
  double* vhead;   // [p] reflector heads
  double* beta;    // [p]
  double* pv;      // [2][p]
  double* part;    // [2][gridDim.x]
  double* vb;      // [gridDim.x][2][p] per-CTA reflector copies (global form)
  double* wb;      // [gridDim.x][p] per-CTA w = p_j - K v_j (global form)
  int64_t stop;    // phases to run (the resident kernel takes over there), at most p - 2
};

// The per-CTA vectors (two reflectors and w, 3 p doubles) live in shared
// memory up to this many bytes, else in global memory.
constexpr size_t TRI1_SMEM_MAX = 200 * 1024;

__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  __syncthreads();  // red may still be read from the previous call
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  const int nw = blockDim.x >> 5;
  for (int w = 0; w < nw; ++w) t += red[w];
  return t;
}

// Reflector of x = v[k0 .. p): on return v[k0] holds the head x0 - alpha and
// the rest is x; beta = 0 (and alpha = x0) when x is already reduced.
__device__ __forceinline__ void make_reflector(double* v, int64_t k0, int64_t p, double* red,
                                               double& beta, double& alpha) {
  double s = 0.0;
  for (int64_t k = k0 + threadIdx.x; k < p; k += blockDim.x) s += v[k] * v[k];
  const double norm2 = block_sum(s, red);
  const double x0 = v[k0];
  const double sig = norm2 - x0 * x0;
  double head = x0;
  beta = 0.0;
  alpha = x0;
  if (sig > 0.0) {
    const double nrm = sqrt(norm2);
    alpha = x0 >= 0.0 ? -nrm : nrm;
    head = x0 - alpha;
    beta = 2.0 / (sig + head * head);
  }
  __syncthreads();  // every thread has read v[k0]
  if (threadIdx.x == 0) v[k0] = head;
  __syncthreads();
}

template <bool SH, int R = 16>
__global__ void __launch_bounds__(TRI_NT, 1) tridiag1_kernel(const Tri1Args a) {
  cg::grid_group grid = cg::this_grid();
  __shared__ double red[TRI_NT / 32];
  extern __shared__ double tri_sh[];
  const int lane = threadIdx.x & 31;
  constexpr int WPB = TRI_NT / 32;
  const int64_t gw = (int64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
  const int64_t nw = (int64_t)gridDim.x * WPB;
  const int64_t G = gridDim.x;
  const int64_t p = a.p;
  double* A = a.A;
  const bool lead = blockIdx.x == 0;
  if (p < 3) {
    if (lead && threadIdx.x == 0) {
      a.d[0] = A[0];
      if (p == 2) {
        a.e[0] = A[1];
        a.d[1] = A[3];
      }
    }
    return;
  }
  // the reflectors v_j, v_{j+1} and w_j = p_j - K v_j for the rows >= j+2,
  // read by every warp of the CTA for every trailing column
  double* vb = SH ? tri_sh : a.vb + (int64_t)blockIdx.x * 2 * p;
  double* wv = SH ? tri_sh + 2 * p : a.wb + (int64_t)blockIdx.x * p;
  // prologue: reflector 0 from column 0, p_0 over the columns c >= 1
  double* vcur = vb;
  for (int64_t k = 1 + threadIdx.x; k < p; k += blockDim.x) vcur[k] = A[k];
  double bcur = 0.0, alpha = 0.0;
  make_reflector(vcur, 1, p, red, bcur, alpha);
  if (lead) {
    if (threadIdx.x == 0) {
      a.d[0] = A[0];
      a.e[0] = alpha;
      a.vhead[0] = vcur[1];
      a.beta[0] = bcur;
    }
    for (int64_t k = 2 + threadIdx.x; k < p; k += blockDim.x) A[k * p] = vcur[k];  // row 0
  }
  {
    double dot = 0.0;
    if (bcur != 0.0)
      for (int64_t c = 1 + ((gw - 1) % nw + nw) % nw; c < p; c += nw) {
        const double* col = A + c * p;
        double s = 0.0;
        for (int64_t k = 1 + lane; k < p; k += 32) s = fma(col[k], vcur[k], s);
        s = warp_sum(s) * bcur;
        if (lane == 0) a.pv[c] = s;
        dot = fma(s, vcur[c], dot);
      }
    const double t = block_sum(lane == 0 ? dot : 0.0, red);
    if (threadIdx.x == 0) a.part[blockIdx.x] = t;
  }
  grid.sync();
  for (int64_t j = 0; j < a.stop; ++j) {
    const int par = (int)(j & 1), nxt = par ^ 1;
    vcur = vb + par * p;
    double* vnext = vb + nxt * p;
    const double* pj = a.pv + par * p;
    const double g = block_sum(threadIdx.x < G ? a.part[par * G + threadIdx.x] : 0.0, red);
    const double K = 0.5 * bcur * g;
    const bool upd = bcur != 0.0;
    const int64_t k1 = j + 1, k2 = j + 2;
    const double vj1 = vcur[k1], wj1 = upd ? pj[k1] - K * vj1 : 0.0;
    // column j+1 of A^{(j+1)}, rows >= j+2, and its diagonal entry
    {
      const double* colj1 = A + k1 * p;
      const int64_t bd = blockDim.x;
      int64_t k = k2 + threadIdx.x;
      for (; k + 3 * bd < p; k += 4 * bd) {
        double av[4], vv[4], qv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          av[u] = colj1[k + u * bd];
          vv[u] = vcur[k + u * bd];
          qv[u] = pj[k + u * bd];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double wk = upd ? qv[u] - K * vv[u] : 0.0;
          wv[k + u * bd] = wk;
          vnext[k + u * bd] = av[u] - (vv[u] * wj1 + wk * vj1);
        }
      }
      for (; k < p; k += bd) {
        const double vk = vcur[k], wk = upd ? pj[k] - K * vk : 0.0;
        wv[k] = wk;
        vnext[k] = colj1[k] - (vk * wj1 + wk * vj1);
      }
    }
    const double dnew = A[k1 + k1 * p] - 2.0 * vj1 * wj1;
    double bnext = 0.0;
    if (k1 + 2 < p) {
      make_reflector(vnext, k2, p, red, bnext, alpha);
      if (lead) {
        if (threadIdx.x == 0) {
          a.d[k1] = dnew;
          a.e[k1] = alpha;
          a.vhead[k1] = vnext[k2];
          a.beta[k1] = bnext;
        }
        for (int64_t k = k2 + 1 + threadIdx.x; k < p; k += blockDim.x) A[k1 + k * p] = vnext[k];
      }
    } else {  // the last 2 x 2 block: no further reflector
      __syncthreads();
      if (lead && threadIdx.x == 0) {
        a.d[k1] = dnew;
        a.e[k1] = vnext[k2];
      }
    }
    // trailing columns: update rows >= j+2 and form p_{j+1} from the new values
    double dot = 0.0;
    for (int64_t c = k2 + ((gw - k2) % nw + nw) % nw; c < p; c += nw) {
      double* col = A + c * p;
      const double vc = vcur[c], wc = wv[c];
      double s = 0.0;
      int64_t k = k2 + lane;
      if constexpr (SH) {
        // R rows per lane per step (one L2 round trip), the column's loads
        // issued before any store; the vectors come from shared memory; the
        // ragged end is one predicated step
        for (; k < p; k += 32 * R) {
          double av[R];
#pragma unroll
          for (int u = 0; u < R; ++u) av[u] = k + 32 * u < p ? col[k + 32 * u] : 0.0;
#pragma unroll
          for (int u = 0; u < R; ++u) {
            const int64_t kk = k + 32 * u;
            if (kk < p) {
              const double x = av[u] - (vcur[kk] * wc + wv[kk] * vc);
              col[kk] = x;
              s = fma(x, vnext[kk], s);
            }
          }
        }
      }
      // eight rows per lane per step, every load issued before any store
      // (the stores to col could alias the loads for all the compiler knows)
      for (; k + 224 < p; k += 256) {
        double av[8], vv[8], qv[8], nv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          av[u] = col[k + 32 * u];
          vv[u] = vcur[k + 32 * u];
          qv[u] = wv[k + 32 * u];
          nv[u] = vnext[k + 32 * u];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const double x = av[u] - (vv[u] * wc + qv[u] * vc);
          col[k + 32 * u] = x;
          s = fma(x, nv[u], s);
        }
      }
      for (; k < p; k += 32) {
        const double x = col[k] - (vcur[k] * wc + wv[k] * vc);
        col[k] = x;
        s = fma(x, vnext[k], s);
      }
      s = warp_sum(s) * bnext;
      if (lane == 0 && bnext != 0.0) a.pv[nxt * p + c] = s;
      dot = fma(s, vnext[c], dot);
    }
    const double t = block_sum(lane == 0 ? dot : 0.0, red);
    if (threadIdx.x == 0) a.part[nxt * G + blockIdx.x] = t;
    bcur = bnext;
    grid.sync();
  }
  if (lead && threadIdx.x == 0 && a.stop + 2 >= p) a.d[p - 1] = A[(p - 1) + (p - 1) * p];
}

// ------------------------------------------- resident tridiagonalisation --
// The one-barrier reduction with the trailing matrix in shared memory: the
// columns of the last n rows and columns, dealt to the CTAs in turn (14
// columns of 2 048 rows are 224 KB), stay there until they are used up.
//
// tridiag1_kernel moves every trailing element through L2 twice a column and
// waits for it in rounds: 9.3 us a column at p = 2 048, 5.2 us at 501, where
// the whole matrix is 2 MB.  Here a column costs one exchange of two vectors
// and a pass over shared memory.  A thread keeps its rows (tid, tid + NT,
// ...) of v_j, p_j, w_j and v_{j+1} in registers and walks the CTA's columns
// eight at a time.  The pivot column of the next phase travels with p_{j+1}:
// by symmetry its entry r is the pivot row's entry in column r, so each CTA
// contributes both for its own columns, 16 bytes a column (the update is
// written so that both triangles round alike).  p_j^T v_j and the reflector
// come from block sums that every CTA forms from the same values in the same
// order, so all hold the same bits.
//
// CTAs meet once a column at a counter: each adds its arrival (a release after
// its part) and one thread of each watches for the last (3 100 clocks with 148
// CTAs, data included; a flag word per CTA, watched by 148 threads of every
// CTA, took 11 900: the polls queue at the flags' lines).  The launch is
// cooperative, so all CTAs are resident; a watcher gives up after its budget,
// records a timeout and the CTA returns, and so do then the others.  One
// cluster of 16 CTAs with the exchange through distributed shared memory was
// no faster at 450 columns and below (1.71 ms against 1.65): its barrier takes
// 1 400 clocks and the scattered remote stores 2 500.
constexpr size_t RES_SMEM = 224 * 1024;  // for the columns (227 KB less the static part)
constexpr int RES_COLS = 16;             // most columns of a CTA

struct ResArgs {
  double* A;        // p x p column-major (both triangles)
  int64_t p;
  int resume;       // 0: column 0's reflector first (r0 = 1); 1: from tridiag1_kernel at
                    // phase r0 - 2, whose reflector (in row r0 - 2) and p vector are in place
  int r0;           // first row and column held in shared memory
  double* d;
  double* e;
  double* vhead;
  double* beta;
  const double* pv;    // resume: p vectors [2][p]
  double2* px;         // [2][p] (p vector, pivot column) by row
  unsigned* arrived;   // zeroed: CTAs past their part of the exchanges so far
  int* err;
  long long wait_cycles;
};

template <int NT>
__device__ __forceinline__ double res_block_sum(double v, double* red) {
  constexpr int RES_WARPS = NT / 32;
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int w = 0; w < RES_WARPS; ++w) t[w & 3] += red[w];
  return (t[0] + t[1]) + (t[2] + t[3]);
}

// Eight per-lane values summed over the warp; lane 4 q gets the sum of c[q].
__device__ __forceinline__ double warp_sum_of8(const double (&c)[8], int lane) {
  double h[4], g[2];
  const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0, hi4 = (lane & 4) != 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    h[i] = (hi16 ? c[i + 4] : c[i]) + __shfl_xor_sync(0xffffffffu, hi16 ? c[i] : c[i + 4], 16);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    g[i] = (hi8 ? h[i + 2] : h[i]) + __shfl_xor_sync(0xffffffffu, hi8 ? h[i] : h[i + 2], 8);
  double v = (hi4 ? g[1] : g[0]) + __shfl_xor_sync(0xffffffffu, hi4 ? g[0] : g[1], 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

// The reflector of a vector of squared norm norm2 and first entry x0.
__device__ __forceinline__ void res_reflector(double norm2, double x0, double& alpha, double& head,
                                              double& beta) {
  const double sig = norm2 - x0 * x0;
  alpha = head = x0;
  beta = 0.0;
  if (sig > 0.0) {
    const double nrm = sqrt(norm2);
    alpha = x0 >= 0.0 ? -nrm : nrm;
    head = x0 - alpha;
    beta = 2.0 / (sig + head * head);
  }
}

template <int RES_NT, int U>
__global__ void __launch_bounds__(RES_NT, 1) tridiag_res_kernel(const ResArgs a) {
  constexpr int RES_WARPS = RES_NT / 32;
  extern __shared__ double res_s[];  // column lc at lc * n
  __shared__ double red[2][RES_WARPS], colsum[RES_WARPS][RES_COLS];
  __shared__ double2 sc[RES_COLS];   // (v, w) at the CTA's own columns
  __shared__ double xr[RES_COLS];    // the next pivot row at them
  __shared__ double s_x0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)gridDim.x, b = (int)blockIdx.x;
  const int p = (int)a.p, r0 = a.r0, n = p - r0;
  const int C = n > b ? (n - b + G - 1) / G : 0;  // columns r0 + b + lc G
  for (int lc = 0; lc < C; ++lc) {
    const double* src = a.A + (int64_t)(r0 + b + lc * G) * p + r0;
    for (int i = tid; i < n; i += RES_NT) res_s[lc * n + i] = src[i];
  }
  int own[U];  // the CTA's column that is row tid + NT u, or -1
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int i = tid + u * RES_NT;
    own[u] = i < n && i % G == b ? i / G : -1;
  }
  double v[U];  // v_j at this thread's rows
  double bcur, head;
  unsigned epoch = 0;
  // Warp 0 sums the columns' products over the CTA (a lane a column) and
  // publishes p and the pivot row.
  auto exchange = [&](int lcs, double bn, int par) {
    __syncthreads();  // colsum and xr are complete
    ++epoch;
    if (warp != 0) return;
    const bool mine = lane >= lcs && lane < C;
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    if (mine)
#pragma unroll
      for (int w = 0; w < RES_WARPS; ++w) t[w & 3] += colsum[w][lane];
    const double pc = ((t[0] + t[1]) + (t[2] + t[3])) * bn;
    if (mine) a.px[(int64_t)par * p + r0 + b + lane * G] = make_double2(pc, xr[lane]);
    __syncwarp();
    if (lane == 0)
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.arrived) : "memory");
  };
  // Everyone's part of the last exchange; false (in every thread) on timeout.
  auto wait_all = [&]() -> bool {
    bool ok = a.wait_cycles > 0;
    if (ok && tid == 0) {
      const unsigned want = epoch * (unsigned)G;
      const long long t0 = clock64();
      for (;;) {
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.arrived) : "memory");
        if (seen >= want) break;
        if (clock64() - t0 > a.wait_cycles) {
          ok = false;
          break;
        }
      }
    }
    if (!__syncthreads_and(ok)) {
      if (tid == 0) atomicExch(a.err, DEV_ERR_TIMEOUT);
      return false;
    }
    return true;
  };
  // This thread's rows from i2 on of the columns from lcs on: A -= v w_c + w
  // v_c (upd), then the columns' products with vn into colsum.
  auto walk = [&](int i2, int lcs, bool upd, const double (&w)[U], const double (&vn)[U]) {
    for (int lc = lcs; lc < C; lc += 8) {
      double t[8] = {};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (lc + q >= C) continue;
        const double2 vw = upd ? sc[lc + q] : make_double2(0.0, 0.0);
        double* col = res_s + (lc + q) * n;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = tid + u * RES_NT;
          if (i >= i2 && i < n) {
            double x = col[i];
            if (upd) {
              x = x - (v[u] * vw.y + w[u] * vw.x);
              col[i] = x;
            }
            t[q] = fma(x, vn[u], t[q]);
            if (i == i2) xr[lc + q] = x;
          }
        }
      }
      const double ws = warp_sum_of8(t, lane);
      if ((lane & 3) == 0 && lc + (lane >> 2) < C) colsum[warp][lc + (lane >> 2)] = ws;
    }
  };

  int j = r0 - 2, turn = 0;  // turn: the CTA that writes phase j's scalars
  if (!a.resume) {
    // reflector 0 from column 0, then p_0 over the columns c >= 1
    j = 0;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = tid + u * RES_NT;
      v[u] = i < n ? a.A[r0 + i] : 0.0;
      s = fma(v[u], v[u], s);
    }
    const double norm2 = res_block_sum<RES_NT>(s, red[0]);  // (a barrier: the columns are in place)
    double alpha;
    res_reflector(norm2, a.A[r0], alpha, head, bcur);
    if (tid == 0) v[0] = head;
    if (b == 0 && tid == 0) {
      a.d[0] = a.A[0];
      a.e[0] = alpha;
      a.vhead[0] = head;
      a.beta[0] = bcur;
    }
    walk(0, 0, false, v, v);
    exchange(0, bcur, 0);
  } else {
    head = a.vhead[j];
    bcur = a.beta[j];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = tid + u * RES_NT;
      v[u] = i < n ? a.A[j + (int64_t)(r0 + i) * p] : 0.0;
    }
    __syncthreads();
  }
  for (; j + 2 < p; ++j, turn = turn + 1 == G ? 0 : turn + 1) {
    if (epoch > 0 && !wait_all()) return;
    const int par = j & 1, k1 = j + 1, k2 = j + 2, i2 = k2 - r0;
    // p_j, and column j + 1 (rows from j + 1 on) before reflector j
    double w[U], vn[U], g = 0.0;
    double2 q1;
    if (epoch > 0) {
      const double2* px = a.px + (int64_t)par * p;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = tid + u * RES_NT;
        const double2 q = i >= i2 && i < n ? __ldcg(px + r0 + i) : make_double2(0.0, 0.0);
        w[u] = q.x;
        vn[u] = q.y;
      }
      q1 = __ldcg(px + k1);
    } else {  // the first phase after tridiag1_kernel
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = tid + u * RES_NT;
        const bool on = i >= i2 && i < n;
        w[u] = on ? a.pv[(int64_t)par * p + r0 + i] : 0.0;
        vn[u] = on ? a.A[(r0 + i) + (int64_t)k1 * p] : 0.0;
      }
      q1 = make_double2(a.pv[(int64_t)par * p + k1], a.A[k1 + (int64_t)k1 * p]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = tid + u * RES_NT;
      if (i < i2 || i >= n) v[u] = 0.0;
      g = fma(w[u], v[u], g);
    }
    g = res_block_sum<RES_NT>(g, red[0]) + q1.x * head;
    if (b == turn) {  // reflector j, below the diagonal of column j
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = tid + u * RES_NT;
        if (i >= i2 && i < n) a.A[(r0 + i) + (int64_t)j * p] = v[u];
      }
    }
    const bool upd = bcur != 0.0;
    const double K = 0.5 * bcur * g;
    const double wj1 = upd ? q1.x - K * head : 0.0;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = tid + u * RES_NT;
      const bool on = i >= i2 && i < n;
      w[u] = upd && on ? w[u] - K * v[u] : 0.0;
      vn[u] = on ? vn[u] - (v[u] * wj1 + w[u] * head) : 0.0;
      s = fma(vn[u], vn[u], s);
      if (i == i2) s_x0 = vn[u];
      if (on && own[u] >= 0) sc[own[u]] = make_double2(v[u], w[u]);
    }
    const double norm2 = res_block_sum<RES_NT>(s, red[1]);  // its barrier covers s_x0 and sc
    const double dnew = q1.y - 2.0 * head * wj1;
    const bool last = k2 + 1 >= p;
    double alpha = s_x0, head_next = s_x0, bnext = 0.0;
    if (!last) {
      res_reflector(norm2, s_x0, alpha, head_next, bnext);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (tid + u * RES_NT == i2) vn[u] = head_next;
    }
    if (b == turn && tid == 0) {
      a.d[k1] = dnew;
      a.e[k1] = alpha;
      if (!last) {
        a.vhead[k1] = head_next;
        a.beta[k1] = bnext;
      }
    }
    // trailing columns c >= j + 2: rank-2 update and the next product
    const int lcs = i2 > b ? (i2 - b + G - 1) / G : 0;
    walk(i2, lcs, true, w, vn);
    if (last) {  // the only entry left
      __syncthreads();
      if (tid == 0 && lcs < C) a.d[p - 1] = xr[lcs];
      break;
    }
    exchange(lcs, bnext, par ^ 1);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = vn[u];
    head = head_next;
    bcur = bnext;
  }
}

// Rows and columns the kernel holds with `blocks` CTAs.
int64_t resident_rows(int blocks) {
  int64_t n = 1;
  while (sizeof(double) * (size_t)(n + 1) * (size_t)((n + blocks) / blocks) <= RES_SMEM &&
         (n + blocks) / blocks <= RES_COLS)
    ++n;
  return n;
}

template <int NT, int U>
shrk_status launch_resident(const ResArgs& a, int blocks, cudaStream_t s) {
  const int64_t n = a.p - a.r0;
  const size_t bytes = sizeof(double) * (size_t)n * (size_t)((n + blocks - 1) / blocks);
  const void* fn = (const void*)tridiag_res_kernel<NT, U>;
  SHRK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  SHRK_CUDA(cudaMemsetAsync(a.arrived, 0, sizeof(unsigned), s));
  ResArgs copy = a;
  void* args[] = {&copy};
  SHRK_CUDA(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(NT), args, bytes, s));
  return SHRK_OK;
}

// Threads by size (measured, ms for 256 / 512): p = 501 1.55 / 1.67, 1 000
// 3.55 / 3.82, 1 500 6.58 / 6.48, 2 048 11.57 / 10.26: fewer warps make the
// block sums short, more of them the update.
shrk_status tridiag_resident(const ResArgs& a, int blocks, cudaStream_t s) {
  const int n = (int)(a.p - a.r0);
  if (n <= 1280) {
    switch ((n + 255) / 256) {
      case 0:
      case 1: return launch_resident<256, 1>(a, blocks, s);
      case 2: return launch_resident<256, 2>(a, blocks, s);
      case 3: return launch_resident<256, 3>(a, blocks, s);
      case 4: return launch_resident<256, 4>(a, blocks, s);
      default: return launch_resident<256, 5>(a, blocks, s);
    }
  }
  switch ((n + 511) / 512) {
    case 3: return launch_resident<512, 3>(a, blocks, s);
    case 4: return launch_resident<512, 4>(a, blocks, s);
    default: return launch_resident<512, 5>(a, blocks, s);
  }
}

// ------------------------------------------------------------ bisection --
// Slot k: the kloc-th smallest eigenvalue of the unreduced block [b0, b1)
// of T, searched in the block's Gershgorin interval [lo, hi].
struct EigSlot {
  int b0, b1, kloc, pad;
  double lo, hi;
};

// Number of eigenvalues of T[b0:b1) below x: the sign changes along the
// leading minors of T - x I, n_i = (d_i - x) n_{i-1} - e_{i-1}^2 n_{i-2} (the
// ratios n_i / n_{i-1} are the pivots of its LDL^T factorisation).  A zero minor
// needs no care: its neighbours have opposite signs, so one change is counted
// whichever sign the zero carries.  te[i] = (d_i, e_{i-1}^2) of T scaled by a
// power of two to norm in (1/2, 1], so a minor grows at most threefold a row
// and, with e^2 above eps^2, two rows lose at most 2^-104: rescaling the pair
// by its exponent every eight rows keeps it in range.  Three FP64 operations,
// two integer ones and a load a row.
__device__ __forceinline__ int sturm(const double2* __restrict__ te, int b0, int b1, double x) {
  double num = te[b0].x - x, den = 1.0;
  unsigned cnt = (unsigned)__double2hiint(num) >> 31;
  auto row = [&](double2 t) {
    const double nn = fma(t.x - x, num, -(t.y * den));
    cnt += (unsigned)(__double2hiint(nn) ^ __double2hiint(num)) >> 31;
    den = num;
    num = nn;
  };
  int i = b0 + 1;
  for (; i + 8 <= b1; i += 8) {
    double2 t[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) t[u] = te[i + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) row(t[u]);
    // 2^-k of the larger magnitude's exponent, exactly
    const int hx = max(__double2hiint(num) & 0x7ff00000, __double2hiint(den) & 0x7ff00000);
    const double sc = __hiloint2double(0x7fe00000 - hx, 0);
    num *= sc;
    den *= sc;
  }
  for (; i < b1; ++i) row(te[i]);
  return (int)cnt;
}

// G-way multisection, G lanes per eigenvalue (32 / G eigenvalues a warp):
// each step probes G evenly spaced points of the bracket and keeps the
// sub-interval where the Sturm count crosses kloc (log2(G + 1) bits a step).
// A wide G takes fewer steps (each is a chain of one FMA a row), a narrow one
// fewer counts in all.  Every lane stays in the loop until its warp is done
// (the shuffles span the warp).  back = the power of two that undoes T's
// scaling.
template <int G>
__global__ void __launch_bounds__(128) bisect_kernel(const double2* __restrict__ te,
                                                     const EigSlot* __restrict__ slots, int n,
                                                     double tiny, double back,
                                                     double* __restrict__ lam) {
  const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(gt / G);
  const int wl = threadIdx.x & 31, lane = wl % G, g0 = wl - lane;
  const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << g0);
  EigSlot sl{0, 0, 0, 0, 0.0, 0.0};
  bool done = k >= n;
  if (!done) sl = slots[k];
  double lo = sl.lo, hi = sl.hi;
  const double eps = 2.220446049250313e-16;
  for (int it = 0; it < 64; ++it) {
    if (!done && hi - lo <= 2.0 * eps * fmax(fabs(lo), fabs(hi)) + tiny) done = true;
    if (__ballot_sync(0xffffffffu, !done) == 0u) break;
    const double x = lo + (hi - lo) * (double)(lane + 1) / (double)(G + 1);
    const bool above = !done && sturm(te, sl.b0, sl.b1, x) > sl.kloc;
    const unsigned m = (__ballot_sync(0xffffffffu, above) & gmask) >> g0;
    const int f = __ffs(m);  // first probe above kloc, 1-based (0: none)
    const double xl = __shfl_sync(0xffffffffu, x, g0 + (f == 0 ? G - 1 : (f >= 2 ? f - 2 : 0)));
    const double xh = __shfl_sync(0xffffffffu, x, g0 + (f == 0 ? 0 : f - 1));
    const double nlo = f == 0 ? xl : (f == 1 ? lo : xl);
    const double nhi = f == 0 ? hi : xh;
    if (!done) {
      if (!(nlo > lo || nhi < hi)) done = true;  // no representable progress
      else {
        lo = nlo;
        hi = nhi;
      }
    }
  }
  if (lane == 0 && k < n) lam[k] = 0.5 * (lo + hi) * back;
}

// ------------------------------------------------------ inverse iteration --
// Cluster c: slots [s0, s0 + ns) of the unreduced block [b0, b1).
struct Cluster {
  int s0, ns, b0, b1;
};

// Deterministic start vector entry (hash of slot and row), in [-1, 1).
__device__ __forceinline__ double start_entry(int slot, int i) {
  uint64_t h = (uint64_t)(uint32_t)slot * 0x9E3779B97F4A7C15ull ^ (uint64_t)(uint32_t)i * 0xC2B2AE3D27D4EB4Full;
  h ^= h >> 31;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 29;
  return (double)(h >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// One thread per cluster, a warp per CTA (the warp together where a cluster's
// vectors are orthogonalised).  Workspace: the factorisation of
// T - lambda I (U's off-diagonals, reciprocal pivots, multipliers, row
// swaps) and the right-hand side / solution x, rows relative to the block
// start, stored per warp as [row][array][lane].  Each eigenvalue is factored
// once and its three solves replay the elimination with multiplications only.
// Eigenvector of slot s goes to Zt[s + i p] (row s of Z^T) for i in [b0, b1).
//
// A lane's solve is one chain over the rows, a warp or less on an SM, so the
// workspace reads must be far ahead of it: each lane copies its own values
// into a ring of II_D chunks in shared memory, asynchronously.  (Chunks loaded
// into registers when their turn came waited out the memory's latency each
// time: 1.74 ms at p = 2 048, whose workspace of 200 MB does not stay in L2,
// now 1.32.)
constexpr int II_ARRAYS = 6;  // u1, u2, 1/pivot, multiplier, swap, x
constexpr int II_CH = 16;     // rows of a chunk
constexpr int II_D = 5;       // chunks in flight
constexpr int II_RING = II_D * II_CH * 4 * 32;  // doubles

__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}

constexpr int II_RS = II_ARRAYS * 32;  // doubles per workspace row of a warp
enum { II_U1 = 0, II_U2 = 1, II_RP = 2, II_MU = 3, II_SW = 4, II_X = 5 };

// One elimination step of T - lambda I with partial pivoting: rows i and
// i + 1, where row i holds (diag, sup) after the earlier steps and row i + 1
// is (sub, nd, ns).  r points at row i of this lane's workspace.  Branch
// free (the lanes of a warp pivot differently); one division.
__device__ __forceinline__ void factor_row(double* r, double sub, double nd, double ns,
                                           double small, double rsmall, double& diag,
                                           double& sup) {
  const bool swp = fabs(diag) < fabs(sub);
  const double piv = swp ? sub : diag;
  const double num = swp ? diag : sub;
  const double ap = fabs(piv);
  const double rinv = ap > 0x1p-400 && ap < 0x1p400 ? rcp_rn_signed(piv) : 1.0 / piv;
  const double m = piv != 0.0 ? num * rinv : 0.0;
  r[II_U1 * 32] = swp ? nd : sup;
  r[II_U2 * 32] = swp ? ns : 0.0;
  r[II_MU * 32] = m;
  r[II_SW * 32] = swp ? 1.0 : 0.0;
  r[II_RP * 32] = fabs(piv) < small ? (piv < 0.0 ? -rsmall : rsmall) : rinv;
  const double nd2 = swp ? fma(-m, nd, sup) : fma(-m, sup, nd);
  sup = swp ? -m * ns : ns;
  diag = nd2;
}

// The factorisation's row operation on the right-hand side: x(i) is final,
// rhs carries row i + 1 (rn is the old x(i + 1)).
__device__ __forceinline__ void forward_row(double* r, double rn, double m, double sw,
                                            double& rhs) {
  const bool swp = sw != 0.0;
  const double keep = swp ? rn : rhs;
  const double other = swp ? rhs : rn;
  r[II_X * 32] = keep;
  rhs = fma(-m, keep, other);
}

// Modified Gram-Schmidt of x (n rows II_RS apart) against q unit vectors (vector r
// at z[r], its rows p apart), then to unit length; by the warp, a row a lane.  (The
// vectors are not rescaled in between: x - (z . x) z does not depend on it.)  Two
// L2 latencies a vector bound it.  A lane of its own waited out a load for every
// row: rank 800 at p = 1 600 took 131 ms in this kernel, now 10.8; four clusters of
// 250 at p = 1 000 24 s, now 2.8.
__device__ void orthogonalise(double* x, int n, const double* z, int64_t p, int q, int lane) {
  constexpr int U = 8;  // rows in flight a lane
  __syncwarp();         // x and z as their lanes left them
  double nrm2 = 0.0;
  for (int r = 0; r < q; ++r) {
    double xv[U], zv[U], dt = 0.0;
    const auto load = [&](int i0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 32 * u + lane;
        xv[u] = i < n ? x[(int64_t)i * II_RS] : 0.0;
        zv[u] = i < n ? z[r + i * p] : 0.0;
      }
    };
    for (int i0 = 0; i0 < n; i0 += 32 * U) {
      load(i0);
#pragma unroll
      for (int u = 0; u < U; ++u) dt = fma(zv[u], xv[u], dt);
    }
    dt = warp_sum(dt);
    nrm2 = 0.0;
    for (int i0 = 0; i0 < n; i0 += 32 * U) {
      if (n > 32 * U) load(i0);  // (else they are still there)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + 32 * u + lane;
        const double xi = fma(-dt, zv[u], xv[u]);
        if (i < n) x[(int64_t)i * II_RS] = xi;
        nrm2 = fma(xi, xi, nrm2);
      }
    }
  }
  const double inv = 1.0 / sqrt(warp_sum(nrm2));
  for (int i = lane; i < n; i += 32) x[(int64_t)i * II_RS] *= inv;
  __syncwarp();
}

__global__ void __launch_bounds__(32) inverse_iteration_kernel(
    const double* __restrict__ d, const double* __restrict__ e, const double* __restrict__ lam,
    const Cluster* __restrict__ cl, int ncl, int64_t p, double tnorm, double* __restrict__ ws,
    double* __restrict__ Zt) {
  const int lane = threadIdx.x;
  const int t = blockIdx.x * 32 + lane;
  const Cluster c = t < ncl ? cl[t] : Cluster{0, 0, 0, 0};
  double* const wl = ws + (int64_t)blockIdx.x * p * II_RS + lane;  // row 0 of this lane
#define W(a, i) wl[(int64_t)(i) * II_RS + (a) * 32]
  extern __shared__ double ring[];  // [II_D][II_CH][4][32]
  const auto at = [&](int k, int u, int j) -> double* {
    return ring + ((((k % II_D) * II_CH + u) * 4 + j) * 32 + lane);
  };
  const int n = c.b1 - c.b0;
  const double small = 2.220446049250313e-16 * tnorm + 1e-300;
  const double rsmall = 1.0 / small;
  const double* db = d + c.b0;
  const double* eb = e + c.b0;
  constexpr int CH = II_CH;
  const int members = __reduce_max_sync(0xffffffffu, c.ns);  // of the warp's largest cluster
  for (int q = 0; q < members; ++q) {
    const bool on = q < c.ns;
    const int slot = c.s0 + q;
    if (on) {
      const double l = lam[slot];
      // factor T - l I once with partial pivoting (and write the start
      // vector); the three solves replay the elimination on their right-hand
      // sides
      {
        double diag = db[0] - l;
        double sup = n > 1 ? eb[0] : 0.0;
        int i0 = 0;
        for (; i0 + CH + 1 < n; i0 += CH) {  // full chunks: rows i0 + u + 2 < n
          double subv[CH], ndv[CH], nsv[CH];
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            subv[u] = eb[i0 + u];
            ndv[u] = db[i0 + u + 1] - l;
            nsv[u] = eb[i0 + u + 1];
          }
          double* r = &W(0, i0);
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            factor_row(r + u * II_RS, subv[u], ndv[u], nsv[u], small, rsmall, diag, sup);
            r[u * II_RS + II_X * 32] = start_entry(slot, i0 + u);
          }
        }
        for (int i = i0; i + 1 < n; ++i) {
          factor_row(&W(0, i), eb[i], db[i + 1] - l, i + 2 < n ? eb[i + 1] : 0.0, small, rsmall,
                     diag, sup);
          W(II_X, i) = start_entry(slot, i);
        }
        const double piv = diag;
        W(II_RP, n - 1) = fabs(piv) < small ? (piv < 0.0 ? -rsmall : rsmall) : 1.0 / piv;
        W(II_U1, n - 1) = 0.0;
        W(II_U2, n - 1) = 0.0;
        W(II_X, n - 1) = start_entry(slot, n - 1);
      }
    }
    double scale = 1.0;  // x in memory times scale is the current vector
    for (int iter = 0; iter < 3; ++iter) {
      if (on) {
        // the factorisation's row operations on the right-hand side
        __threadfence();  // the workspace before the copies of it
        double rhs = W(II_X, 0) * scale;
        {
          const int nch = (n - 1) / CH;  // full chunks: rows i0 + u + 1 < n
          const auto fetch = [&](int k) {
            if (k < nch) {
              const double* r = &W(0, k * CH);
#pragma unroll
              for (int u = 0; u < CH; ++u) {
                copy8(at(k, u, 0), r + (u + 1) * II_RS + II_X * 32);
                copy8(at(k, u, 1), r + u * II_RS + II_MU * 32);
                copy8(at(k, u, 2), r + u * II_RS + II_SW * 32);
              }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
          };
          for (int k = 0; k < II_D - 1; ++k) fetch(k);
          for (int k = 0; k < nch; ++k) {
            fetch(k + II_D - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(II_D - 1) : "memory");
            double* r = &W(0, k * CH);
            double rnv[CH], mv[CH], sv[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u) {
              rnv[u] = *at(k, u, 0) * scale;
              mv[u] = *at(k, u, 1);
              sv[u] = *at(k, u, 2);
            }
#pragma unroll
            for (int u = 0; u < CH; ++u) forward_row(r + u * II_RS, rnv[u], mv[u], sv[u], rhs);
          }
          for (int i = nch * CH; i + 1 < n; ++i) {
            const double rn = W(II_X, i + 1) * scale;
            forward_row(&W(0, i), rn, W(II_MU, i), W(II_SW, i), rhs);
          }
        }
        W(II_X, n - 1) = rhs;
        __threadfence();
        // back substitution (the last row's U entries are zero), chunks of
        // rows from the last
        double nrm2 = 0.0, x1 = 0.0, x2 = 0.0;
        {
          const int nch = n / CH;
          const auto fetch = [&](int k) {
            if (k < nch) {
              const double* r = &W(0, n - 1 - k * CH);
#pragma unroll
              for (int u = 0; u < CH; ++u) {
                copy8(at(k, u, 0), r - u * II_RS + II_RP * 32);
                copy8(at(k, u, 1), r - u * II_RS + II_U1 * 32);
                copy8(at(k, u, 2), r - u * II_RS + II_U2 * 32);
                copy8(at(k, u, 3), r - u * II_RS + II_X * 32);
              }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
          };
          for (int k = 0; k < II_D - 1; ++k) fetch(k);
          for (int k = 0; k < nch; ++k) {
            fetch(k + II_D - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(II_D - 1) : "memory");
            double* r = &W(0, n - 1 - k * CH);
#pragma unroll
            for (int u = 0; u < CH; ++u) {
              // the pivot multiplied in first: one FMA from x1 to xi
              const double r0 = *at(k, u, 0);
              const double xi = fma(-(*at(k, u, 1) * r0), x1,
                                    fma(-(*at(k, u, 2) * r0), x2, *at(k, u, 3) * r0));
              r[-u * II_RS + II_X * 32] = xi;
              nrm2 = fma(xi, xi, nrm2);
              x2 = x1;
              x1 = xi;
            }
          }
          const int i0 = n - 1 - nch * CH;
          for (int i = i0; i >= 0; --i) {
            const double r0 = W(II_RP, i);
            const double xi =
                fma(-(W(II_U1, i) * r0), x1, fma(-(W(II_U2, i) * r0), x2, W(II_X, i) * r0));
            W(II_X, i) = xi;
            nrm2 = fma(xi, xi, nrm2);
            x2 = x1;
            x1 = xi;
          }
        }
        scale = 1.0 / sqrt(nrm2);
      }
      // The cluster's earlier vectors (numerically equal eigenvalues only).
      unsigned todo = __ballot_sync(0xffffffffu, on && q > 0);
      for (; todo; todo &= todo - 1) {
        const int k = __ffs(todo) - 1;
        const int s0 = __shfl_sync(0xffffffffu, c.s0, k), b0 = __shfl_sync(0xffffffffu, c.b0, k);
        orthogonalise(&W(II_X, 0) - lane + k, __shfl_sync(0xffffffffu, n, k),
                      Zt + s0 + (int64_t)b0 * p, p, q, lane);
        if (lane == k) scale = 1.0;
      }
    }
    if (on)
      for (int i = 0; i < n; ++i) Zt[slot + (int64_t)(c.b0 + i) * p] = W(II_X, i) * scale;
    __syncwarp();  // the vector before the warp reads it
  }
#undef W
}

// M = 1.5 I - 0.5 G (Newton-Schulz step for the polar factor).
__global__ void ns_matrix_kernel(double* __restrict__ g, int64_t p) {
  // M = (3I - G)/2 from the lower triangle of G (its upper one is not
  // computed), written to both triangles
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t j = blockIdx.y;
  if (i >= p || i < j) return;
  const double v = g[i + j * p];
  const double mv = (i == j ? 1.5 : 0.0) - 0.5 * v;
  g[i + j * p] = mv;
  g[j + i * p] = mv;
}

// The reflectors in blocks of WY_NB, block t from column j0 = t WY_NB: Y_t has
// n_t = p - j0 - 1 rows (its reach) and its own leading dimension n_t; the
// blocks lie one after the other.  Everything that does not depend on Z -- Y_t,
// S_t = Y_t^T Y_t, T_t, Y_t T_t -- is formed for all blocks at once before the
// first product with Z: block by block these were four launches of a few CTAs
// each, 150 us of latency a block.
constexpr int WY_NB = 128;
__host__ __device__ inline int64_t wy_offset(int64_t p, int t) {  // entries of Y before block t
  return (int64_t)WY_NB * ((int64_t)t * (p - 1) - (int64_t)WY_NB * ((int64_t)t * (t - 1) / 2));
}

// Y_t[r, jj] = v_{j0+jj}[j0+1+r] (zero above the reflector's first entry, and a
// zero column past the last reflector or where beta = 0).  Reflector j sits
// right of the diagonal in row j (j < in_rows) or below it in column j, its
// head in vhead[j].
__global__ void build_y_kernel(const double* __restrict__ A, const double* __restrict__ vhead,
                               const double* __restrict__ beta, int64_t p, int64_t in_rows,
                               double* __restrict__ Yall) {
  const int t = blockIdx.z, jj = blockIdx.y;
  const int64_t j0 = (int64_t)t * WY_NB, n = p - j0 - 1, j = j0 + jj;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int64_t row = j0 + 1 + r;
  double v = 0.0;
  if (j >= p - 2 || beta[j] == 0.0) v = 0.0;
  else if (row == j + 1) v = vhead[j];
  else if (row > j + 1) v = j < in_rows ? A[j + row * p] : A[row + j * p];
  Yall[wy_offset(p, t) + r + (int64_t)jj * n] = v;
}

// S_t = Y_t^T Y_t, k split over gridDim.y slabs [t][slab][WY_NB][WY_NB].
__global__ void __launch_bounds__(256, 1) wy_gram_kernel(const double* __restrict__ Yall,
                                                         int64_t p, double* __restrict__ S) {
  __shared__ GemmStage st;
  const int t = blockIdx.x, n = (int)(p - (int64_t)t * WY_NB - 1);
  const int kz = ((n + (int)gridDim.y - 1) / (int)gridDim.y + GK2 - 1) / GK2 * GK2;
  const int kb = min(n, (int)blockIdx.y * kz), ke = min(n, kb + kz);
  const double* Y = Yall + wy_offset(p, t);
  double acc[4][8][2];
  gemm_tile<true, false>(st, WY_NB, WY_NB, kb, ke, 0, 0, Y, n, Y, n, acc);
  gemm_store(WY_NB, WY_NB, 0, 0, 1.0, acc, 0.0,
             S + ((int64_t)t * gridDim.y + blockIdx.y) * WY_NB * WY_NB, WY_NB);
}

// T of the compact WY form, H_{j0} ... H_{j0+nb-1} = I - Y T Y^T (forward),
// from T^{-1} = U = triu(S, 1) + diag(1 / beta), S = Y^T Y (the inverse of T
// is the strictly upper part of Y^T Y plus the reflectors' v^T v / 2 on the
// diagonal; a reflector with beta = 0 has a zero column in Y and a unit
// diagonal here).  A warp per column j of T solves U x = e_j: lane l keeps
// the running right-hand sides of rows l, l + 32, ...; from row j up, the
// owner of row i forms x_i = r_i beta_i (1 / U_ii = beta_i exactly) and
// every lane removes x_i's share from its rows above.  Each step is a
// shuffle and a few FMAs, so the 128-step chain of a column takes a few
// microseconds, all columns and blocks at once.  U lives in dynamic shared
// memory.
constexpr int WY_T_WARPS = 32;  // columns per CTA
constexpr size_t wy_t_smem() { return sizeof(double) * (WY_NB * (WY_NB + 1) + WY_NB); }

__global__ void __launch_bounds__(WY_T_WARPS * 32) wy_t_kernel(const double* __restrict__ S,
                                                              int slabs,
                                                              const double* __restrict__ beta,
                                                              int64_t p, double* __restrict__ T) {
  extern __shared__ double u[];  // u[i LD + k] = U[i][k], i < k
  constexpr int LD = WY_NB + 1, QN = WY_NB / 32, NN = WY_NB * WY_NB;
  double* rd = u + WY_NB * LD;   // 1 / U_ii
  const int t = blockIdx.y;
  const int64_t j0 = (int64_t)t * WY_NB;
  S += (int64_t)t * slabs * NN;
  T += (int64_t)t * NN;
  for (int idx = threadIdx.x; idx < NN; idx += blockDim.x) {
    const int i = idx % WY_NB, k = idx / WY_NB;
    if (i >= k) continue;
    double v = 0.0;
    for (int z = 0; z < slabs; ++z) v += S[(int64_t)z * NN + idx];
    u[i * LD + k] = v;
  }
  for (int i = threadIdx.x; i < WY_NB; i += blockDim.x) {
    const double bi = j0 + i < p - 2 ? beta[j0 + i] : 0.0;
    rd[i] = bi != 0.0 ? bi : 1.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * WY_T_WARPS + (threadIdx.x >> 5);
  if (j0 + j >= p - 2) {  // past the last reflector
    for (int i = lane; i < WY_NB; i += 32) T[i + (int64_t)j * WY_NB] = 0.0;
    return;
  }
  double r[QN];
#pragma unroll
  for (int q = 0; q < QN; ++q) r[q] = lane + 32 * q == j ? 1.0 : 0.0;
  for (int i = j; i >= 0; --i) {
    const int owner = i & 31, qi = i >> 5;
    double xi = 0.0;
#pragma unroll
    for (int q = 0; q < QN; ++q)
      if (q == qi && lane == owner) {
        xi = r[q] * rd[i];
        r[q] = xi;  // row i is final: it now holds T[i][j]
      }
    xi = __shfl_sync(0xffffffffu, xi, owner);
#pragma unroll
    for (int q = 0; q < QN; ++q) {
      const int row = lane + 32 * q;
      if (row < i) r[q] -= u[row * LD + i] * xi;
    }
  }
#pragma unroll
  for (int q = 0; q < QN; ++q) {
    const int row = lane + 32 * q;
    T[row + (int64_t)j * WY_NB] = row <= j ? r[q] : 0.0;
  }
}

// YT_t = Y_t T_t, a CTA per 128 rows of a block.
__global__ void __launch_bounds__(256, 1) wy_yt_kernel(const double* __restrict__ Yall, int64_t p,
                                                       const double* __restrict__ T,
                                                       double* __restrict__ YT) {
  __shared__ GemmStage st;
  const int t = blockIdx.y, n = (int)(p - (int64_t)t * WY_NB - 1), i0 = blockIdx.x * GT2;
  if (i0 >= n) return;
  const int64_t off = wy_offset(p, t);
  const int nb = min(WY_NB, n - 1);  // reflectors of the block
  double acc[4][8][2];
  gemm_tile<false, false>(st, n, WY_NB, 0, nb, i0, 0, Yall + off, n,
                          T + (int64_t)t * WY_NB * WY_NB, WY_NB, acc);
  gemm_store(n, WY_NB, i0, 0, 1.0, acc, 0.0, YT + off, n);
}

// out[:, k] = U[:, perm[k]]
__global__ void permute_columns_kernel(const double* __restrict__ U, int64_t p,
                                       const int* __restrict__ perm, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t k = blockIdx.y;
  if (i < p) out[i + k * p] = U[i + (int64_t)perm[k] * p];
}

// Column-major transpose: out[j + i p] = in[i + j p].
__global__ void transpose_sq_kernel(const double* __restrict__ in, int64_t p,
                                    double* __restrict__ out) {
  __shared__ double tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32;
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int64_t i = i0 + threadIdx.x, j = j0 + dy;
    if (i < p && j < p) tile[dy][threadIdx.x] = in[i + j * p];
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int64_t j = j0 + threadIdx.x, i = i0 + dy;
    if (i < p && j < p) out[j + i * p] = tile[threadIdx.x][dy];
  }
}

// A = the lower triangle mirrored (the eigensolver reads the lower triangle).
__global__ void mirror_lower_kernel(double* __restrict__ A, int64_t p) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t j = blockIdx.y;
  if (i < j && j < p) A[i + j * p] = A[j + i * p];
}

unsigned cdiv(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// Eigenvalues closer than CLUSTER_TOL ||T|| (numerically equal) share one
// thread and are orthogonalised by Gram-Schmidt during inverse iteration;
// every other pair is left to inverse iteration, whose vectors then overlap
// by about eps ||T|| / gap, and to the Newton-Schulz steps (each squares
// the overlap), as many as the smallest such gap needs.
constexpr double CLUSTER_TOL = 1e-12;

// Scratch slots 46..54 belong to this file.
constexpr int SLOT_U = 46, SLOT_Z = 47, SLOT_G = 48, SLOT_SMALL = 49, SLOT_WS = 50,
              SLOT_WY = 51, SLOT_META = 52, SLOT_VB = 53, SLOT_SPLITK = 54;

}  // namespace

template <bool TA, bool TB>
static shrk_status gemm_form(int m, int n, int k, double alpha, const double* A, int64_t lda,
                             const double* B, int64_t ldb, double beta, double* C, int64_t ldc,
                             int lower, const char* family, cudaStream_t s) {
  if (m >= GT2 && n >= GT2 && k >= 64) {
    GemmRuns g;
    g.tm = (int)cdiv(m, GT2);
    g.tn = (int)cdiv(n, GT2);
    g.lower = lower;
    g.ksteps = (int)cdiv(k, GK2);
    const int64_t tiles = lower ? (int64_t)g.tm * (g.tm + 1) / 2 : (int64_t)g.tm * g.tn;
    g.total = tiles * g.ksteps;
    // at least eight steps a CTA: a part costs a slot written and read
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(sm_count(), g.total / 8));
    g.per = g.total / grid;
    g.rem = (int)(g.total % grid);
    void* ws = nullptr;
    SHRK_TRY(scratch_get(SLOT_SPLITK, sizeof(double) * 2 * (size_t)grid * GEMM_SLOT, &ws));
    {
      LaunchScope ls(family, s);
      dgemm_big_kernel<TA, TB><<<grid, 256, 0, s>>>(g, m, n, k, alpha, A, lda, B, ldb, beta, C,
                                                    ldc, (double*)ws);
      SHRK_CUDA(cudaGetLastError());
    }
    // no tile is divided when the runs are whole tiles
    if (g.rem == 0 && g.per % g.ksteps == 0) return SHRK_OK;
    LaunchScope ls(family, s);
    dgemm_fixup_kernel<<<dim3((unsigned)tiles, GEMM_SLOT / 2048), 256, 0, s>>>(
        g, m, n, alpha, beta, C, ldc, (const double*)ws);
    SHRK_CUDA(cudaGetLastError());
    return SHRK_OK;
  }
  const int64_t tiles = (int64_t)cdiv(m, GT) * cdiv(n, GT);
  // too few output tiles to fill the GPU and a long k: split k
  const int64_t want = 2LL * sm_count();
  int splits = 1;
  if (tiles < want && k >= 512)
    splits = (int)std::min<int64_t>({(want + tiles - 1) / tiles, k / 256, 16});
  double* out = C;
  int64_t ldo = ldc;
  double b = beta;
  if (splits > 1) {
    void* ws = nullptr;
    SHRK_TRY(scratch_get(SLOT_SPLITK, sizeof(double) * (size_t)splits * (size_t)m * (size_t)n, &ws));
    out = (double*)ws;
    ldo = m;
    b = 0.0;
  }
  const int kz = (k + splits - 1) / splits;
  {
    LaunchScope ls(family, s);
    dgemm_kernel<TA, TB><<<dim3(cdiv(m, GT), cdiv(n, GT), (unsigned)splits), 256, 0, s>>>(
        m, n, k, kz, alpha, A, lda, B, ldb, b, out, ldo, lower);
    SHRK_CUDA(cudaGetLastError());
  }
  if (splits > 1) {
    LaunchScope ls(family, s);
    dgemm_reduce_kernel<<<cdiv((int64_t)m * n, 256), 256, 0, s>>>(out, splits, m, n, beta, C, ldc);
    SHRK_CUDA(cudaGetLastError());
  }
  return SHRK_OK;
}

shrk_status dgemm(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                  int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc,
                  cudaStream_t s, const char* family, bool lower) {
  if (m <= 0 || n <= 0) return SHRK_OK;
  if (lower && m != n) {
    set_error("dgemm: a lower-triangle product must be square");
    return SHRK_EINVAL;
  }
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) {
    set_error("dgemm: dimensions must be below 2^31");
    return SHRK_EINVAL;
  }
  const auto form = !ta && !tb  ? gemm_form<false, false>
                    : !ta && tb ? gemm_form<false, true>
                    : ta && !tb ? gemm_form<true, false>
                                : gemm_form<true, true>;
  return form((int)m, (int)n, (int)k, alpha, A, lda, B, ldb, beta, C, ldc, lower ? 1 : 0, family, s);
}

shrk_status eigh_device(double* A, int64_t p, std::vector<double>& w_host, cudaStream_t s) {
  w_host.assign((size_t)p, 0.0);
  if (p <= 0) return SHRK_OK;
  const int64_t P2 = p * p;
  void *small = nullptr, *zt = nullptr, *u = nullptr;
  // small: d, e, vhead, beta, pv, scal (+2), part (<= 4096), lam, perm
  SHRK_TRY(scratch_get(SLOT_SMALL, sizeof(double) * (8 * (size_t)p + 4096 + 16), &small));
  double* d = (double*)small;
  double* e = d + p;
  double* vhead = e + p;
  double* beta = vhead + p;
  double* pv = beta + p;
  double* lam = pv + p;
  int* perm = (int*)(lam + p);  // p ints in the room of p/2 doubles (8p doubles reserved)
  double* scal = lam + 2 * p;
  double* part = scal + 16;
  SHRK_TRY(scratch_get(SLOT_Z, sizeof(double) * (size_t)P2, &zt));
  SHRK_TRY(scratch_get(SLOT_U, sizeof(double) * (size_t)P2, &u));
  double* Zt = (double*)zt;
  double* U = (double*)u;

  // 0. symmetric input from its lower triangle
  {
    LaunchScope ls("eigh_tridiag", s);
    mirror_lower_kernel<<<dim3(cdiv(p, 256), (unsigned)p), 256, 0, s>>>(A, p);
    SHRK_CUDA(cudaGetLastError());
  }
  // 1. tridiagonalisation (cooperative: all CTAs resident): the last 2 048
  // rows and columns by the resident kernel, those before them by tridiag1_kernel, which
  // passes the trailing matrix through L2 once a column and leaves reflectors in
  // the upper triangle's rows.  SHRK_EIGH_TRIDIAG=2 runs the two-barrier form on
  // every column (reflectors in the lower triangle), SHRK_EIGH_TRI1_GLOBAL=1
  // tridiag1_kernel with its vectors in global memory.
  const char* tri_env = std::getenv("SHRK_EIGH_TRIDIAG");
  const bool rowstore = !(tri_env && std::strcmp(tri_env, "2") == 0);
  int64_t in_rows = 0;  // reflectors that tridiag1_kernel left in rows
  {
    int dev = 0, sms = 0, per_sm = 0;
    SHRK_CUDA(cudaGetDevice(&dev));
    SHRK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = std::min(sms, TRI_NT);  // tridiag1_kernel sums a share a thread
    const char* glob_env = std::getenv("SHRK_EIGH_TRI1_GLOBAL");
    const bool glob = glob_env && std::strcmp(glob_env, "1") == 0;
    const bool resident = rowstore && !glob && p >= 3;
    const int64_t held = resident ? resident_rows(blocks) : 0;
    // phases before the resident kernel (p - 2: all of them)
    const int64_t stop = resident ? (p - 1 <= held ? 0 : std::max<int64_t>(1, p - 2 - held)) : p - 2;
    if (rowstore) in_rows = stop;
    // p_j [2][p], (p, pivot) pairs [2][p], the partial sums [2][blocks] and the
    // counter; tridiag1_kernel's per-CTA vectors [blocks][3][p] only when they
    // are not in shared memory
    const size_t sh_bytes = sizeof(double) * 3 * (size_t)p;
    const bool sh = sh_bytes <= TRI1_SMEM_MAX && !glob;
    const size_t per_cta = sh ? 0 : (size_t)blocks * 3 * (size_t)p;
    void* vbuf = nullptr;
    SHRK_TRY(scratch_get(SLOT_VB, sizeof(double) * (6 * (size_t)p + 2 * (size_t)blocks + 2 + per_cta),
                         &vbuf));
    double2* pairs = (double2*)vbuf;
    double* pvec = (double*)(pairs + 2 * p);
    double* sums = pvec + 2 * p;
    unsigned* arrived = (unsigned*)(sums + 2 * blocks);
    double* vbd = sums + 2 * blocks + 2;
    if (!rowstore) {
      SHRK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)tridiag_kernel,
                                                              TRI_NT, 0));
      if (per_sm < 1) {
        set_error("eigensolver: the tridiagonalisation kernel cannot be resident");
        return SHRK_ECUDA;
      }
      TriArgs ta{A, p, d, e, vhead, beta, pv, part, scal};
      void* args[] = {&ta};
      LaunchScope ls("eigh_tridiag", s);
      SHRK_CUDA(cudaLaunchCooperativeKernel((const void*)tridiag_kernel, dim3(blocks),
                                            dim3(TRI_NT), args, 0, s));
    } else if (stop > 0 || !resident) {
      // rows per lane per step of the trailing update (measured: 8 best at p =
      // 2 048; 16 at 4 096; 32 slower at both)
      const void* tri1 = !sh         ? (const void*)tridiag1_kernel<false>
                         : p >= 3072 ? (const void*)tridiag1_kernel<true, 16>
                                     : (const void*)tridiag1_kernel<true, 8>;
      const size_t dyn = sh ? sh_bytes : 0;
      if (dyn > 0)
        SHRK_CUDA(cudaFuncSetAttribute(tri1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
      SHRK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tri1, TRI_NT, dyn));
      if (per_sm < 1) {
        set_error("eigensolver: the tridiagonalisation kernel cannot be resident");
        return SHRK_ECUDA;
      }
      Tri1Args ta{A,    p,    d, e, vhead, beta, pvec, sums, sh ? nullptr : vbd,
                  sh ? nullptr : vbd + (size_t)blocks * 2 * p, stop};
      void* args[] = {&ta};
      LaunchScope ls("eigh_tridiag", s);
      SHRK_CUDA(cudaLaunchCooperativeKernel(tri1, dim3(blocks), dim3(TRI_NT), args, dyn, s));
    }
    if (resident) {
      ResArgs ra;
      ra.A = A;
      ra.p = p;
      ra.resume = stop > 0;
      ra.r0 = stop > 0 ? (int)stop + 2 : 1;
      ra.d = d;
      ra.e = e;
      ra.vhead = vhead;
      ra.beta = beta;
      ra.pv = pvec;
      ra.px = pairs;
      ra.arrived = arrived;
      ra.err = device_error_word();
      ra.wait_cycles = wait_cycles();
      LaunchScope ls("eigh_tridiag", s);
      SHRK_TRY(tridiag_resident(ra, blocks, s));
    }
  }
  // 2. split T, Gershgorin bounds per block, eigenvalue slots (host; O(p))
  std::vector<double> hd(p), he(std::max<int64_t>(p - 1, 1), 0.0);
  SHRK_CUDA(cudaMemcpyAsync(hd.data(), d, sizeof(double) * p, cudaMemcpyDeviceToHost, s));
  if (p > 1)
    SHRK_CUDA(cudaMemcpyAsync(he.data(), e, sizeof(double) * (p - 1), cudaMemcpyDeviceToHost, s));
  SHRK_CUDA(cudaStreamSynchronize(s));
  // a wait of the reduction gave up (every matrix call, device-pointer ones too,
  // runs in its thread's host context)
  SHRK_TRY(poll_device_error(s));
  const double eps = 2.220446049250313e-16;
  double tnorm = 0.0;
  for (int64_t i = 0; i < p; ++i) {
    const double r = (i > 0 ? std::fabs(he[i - 1]) : 0.0) + (i + 1 < p ? std::fabs(he[i]) : 0.0);
    tnorm = std::max(tnorm, std::fabs(hd[i]) + r);
  }
  if (!(tnorm > 0.0)) tnorm = 1.0;
  if (!std::isfinite(tnorm)) {
    set_error("symmetric eigendecomposition: the matrix has non-finite entries");
    return SHRK_EINVAL;
  }
  // negligible off-diagonals split T: relative to their diagonal neighbours
  // (dstebz's criterion) or below eps ||T|| (setting them to zero moves no
  // eigenvalue by more than the tridiagonalisation's own backward error;
  // without it a block of rounding noise -- the null space of a low-rank
  // matrix -- would stay one huge cluster)
  std::vector<int> bstart{0};
  for (int64_t i = 0; i + 1 < p; ++i) {
    const double t2 = he[i] * he[i];
    if (t2 <= eps * eps * std::fabs(hd[i] * hd[i + 1]) + 1e-300 ||
        std::fabs(he[i]) <= eps * tnorm) {
      he[i] = 0.0;
      bstart.push_back((int)(i + 1));
    }
  }
  bstart.push_back((int)p);
  // T scaled exactly to norm in (1/2, 1] for the counts
  int te_exp = 0;
  (void)std::frexp(tnorm, &te_exp);
  std::vector<double2> hte(p);
  for (int64_t i = 0; i < p; ++i)
    hte[i] = make_double2(std::ldexp(hd[i], -te_exp),
                          i > 0 ? std::ldexp(he[i - 1], -te_exp) * std::ldexp(he[i - 1], -te_exp)
                                : 0.0);
  const double tiny = 1e-290;  // far below eps times any entry that is not zero
  std::vector<EigSlot> hslots(p);
  for (size_t b = 0; b + 1 < bstart.size(); ++b) {
    const int b0 = bstart[b], b1 = bstart[b + 1];
    double lo = INFINITY, hi = -INFINITY;
    for (int i = b0; i < b1; ++i) {
      const double r = (i > b0 ? std::fabs(he[i - 1]) : 0.0) + (i + 1 < b1 ? std::fabs(he[i]) : 0.0);
      lo = std::min(lo, hd[i] - r);
      hi = std::max(hi, hd[i] + r);
    }
    const double pad = 2.0 * eps;
    lo = std::ldexp(lo, -te_exp) - pad;
    hi = std::ldexp(hi, -te_exp) + pad;
    for (int i = b0; i < b1; ++i) hslots[i] = EigSlot{b0, b1, i - b0, 0, lo, hi};
  }
  void* meta = nullptr;
  SHRK_TRY(scratch_get(SLOT_META, sizeof(EigSlot) * (size_t)p + sizeof(double2) * (size_t)p +
                                      sizeof(Cluster) * (size_t)p + 256, &meta));
  double2* dte = (double2*)meta;
  EigSlot* dslots = (EigSlot*)(dte + p);
  Cluster* dcl = (Cluster*)(dslots + p);
  SHRK_CUDA(cudaMemcpyAsync(e, he.data(), sizeof(double) * std::max<int64_t>(p - 1, 0),
                            cudaMemcpyHostToDevice, s));
  SHRK_CUDA(cudaMemcpyAsync(dte, hte.data(), sizeof(double2) * p, cudaMemcpyHostToDevice, s));
  SHRK_CUDA(cudaMemcpyAsync(dslots, hslots.data(), sizeof(EigSlot) * p, cudaMemcpyHostToDevice, s));
  {
    LaunchScope ls("eigh_bisect", s);
    const double back = std::ldexp(1.0, te_exp);
    // probes per eigenvalue, measured (ms for G = 8 / 16 / 32): p = 501 0.23 /
    // 0.18 / 0.16, 1 024 0.45 / 0.36 / 0.36, 2 048 0.88 / 0.81 / 1.09, 3 100 1.58 /
    // 1.57 / 2.31
    if (p > 4096)
      bisect_kernel<8><<<cdiv(p * 8, 128), 128, 0, s>>>(dte, dslots, (int)p, tiny, back, lam);
    else if (p >= 1024)
      bisect_kernel<16><<<cdiv(p * 16, 128), 128, 0, s>>>(dte, dslots, (int)p, tiny, back, lam);
    else
      bisect_kernel<32><<<cdiv(p * 32, 128), 128, 0, s>>>(dte, dslots, (int)p, tiny, back, lam);
    SHRK_CUDA(cudaGetLastError());
  }
  // 3. clusters of close eigenvalues inside each block (host), inverse iteration
  std::vector<double> hl(p);
  SHRK_CUDA(cudaMemcpyAsync(hl.data(), lam, sizeof(double) * p, cudaMemcpyDeviceToHost, s));
  SHRK_CUDA(cudaStreamSynchronize(s));
  std::vector<Cluster> hcl;
  double min_gap = INFINITY;  // smallest gap inside a block between clusters
  for (size_t b = 0; b + 1 < bstart.size(); ++b) {
    const int b0 = bstart[b], b1 = bstart[b + 1];
    int k = b0;
    while (k < b1) {
      int g = k + 1;
      while (g < b1 && hl[g] - hl[g - 1] < CLUSTER_TOL * tnorm) ++g;
      hcl.push_back(Cluster{k, g - k, b0, b1});
      if (g < b1) min_gap = std::min(min_gap, hl[g] - hl[g - 1]);
      k = g;
    }
  }
  // expected overlap of distinct inverse-iteration vectors, and the
  // Newton-Schulz steps that take it below rounding (e -> ~1.5 e^2)
  const double overlap = min_gap < INFINITY ? 8.0 * eps * tnorm / min_gap : 0.0;
  const int ns_steps = overlap <= 1e-15 ? 0 : (overlap <= 1e-7 ? 1 : 2);
  const int ncl = (int)hcl.size();
  SHRK_CUDA(cudaMemcpyAsync(dcl, hcl.data(), sizeof(Cluster) * ncl, cudaMemcpyHostToDevice, s));
  void* ws = nullptr;
  // per warp of clusters: p rows of II_ARRAYS x 32 doubles
  SHRK_TRY(scratch_get(SLOT_WS,
                       sizeof(double) * II_ARRAYS * 32 * (size_t)cdiv(ncl, 32) * (size_t)p, &ws));
  SHRK_CUDA(cudaMemsetAsync(Zt, 0, sizeof(double) * (size_t)P2, s));
  {
    LaunchScope ls("eigh_inverse_iteration", s);
    constexpr int ring = II_RING * (int)sizeof(double);
    SHRK_CUDA(cudaFuncSetAttribute(inverse_iteration_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, ring));
    inverse_iteration_kernel<<<cdiv(ncl, 32), 32, ring, s>>>(d, e, lam, dcl, ncl, p, tnorm,
                                                            (double*)ws, Zt);
    SHRK_CUDA(cudaGetLastError());
  }
  // Newton-Schulz steps on the basis: Z <- Z (3I - Z^T Z)/2, in the
  // transposed storage Zt: G = Zt Zt^T, Zt <- M Zt
  void* gbuf = nullptr;
  SHRK_TRY(scratch_get(SLOT_G, sizeof(double) * (size_t)P2, &gbuf));
  double* G = (double*)gbuf;
  double* zcur = Zt;  // current Z^T
  double* other = U;
  for (int it = 0; it < ns_steps; ++it) {
    // G is symmetric: its lower triangle's tiles only, mirrored by the
    // kernel that forms M
    SHRK_TRY(dgemm(false, true, p, p, p, 1.0, zcur, p, zcur, p, 0.0, G, p, s, "dgemm", true));
    {
      LaunchScope ls("eigh_orthogonalise", s);
      ns_matrix_kernel<<<dim3(cdiv(p, 256), (unsigned)p), 256, 0, s>>>(G, p);
      SHRK_CUDA(cudaGetLastError());
    }
    SHRK_TRY(dgemm(false, false, p, p, p, 1.0, G, p, zcur, p, 0.0, other, p, s));  // (Z M)^T
    std::swap(zcur, other);
  }
  {
    LaunchScope ls("eigh_orthogonalise", s);
    transpose_sq_kernel<<<dim3(cdiv(p, 32), cdiv(p, 32)), dim3(32, 8), 0, s>>>(zcur, p, other);
    SHRK_CUDA(cudaGetLastError());
  }
  double* Zc = other;  // Z, column-major
  // 4. back-transformation Zc <- H_0 ... H_{p-3} Zc, blocks from the last
  const int64_t nref = std::max<int64_t>(p - 2, 0);
  if (nref > 0) {
    const int nblk = (int)((nref + WY_NB - 1) / WY_NB);
    const int slabs = (int)std::min<int64_t>(8, (p + 255) / 256);
    const int64_t y_len = wy_offset(p, nblk), NN = (int64_t)WY_NB * WY_NB;
    void* wy = nullptr;
    SHRK_TRY(scratch_get(SLOT_WY, sizeof(double) * (size_t)(2 * y_len + nblk * NN * (slabs + 1) +
                                                            (int64_t)WY_NB * p), &wy));
    double* Y = (double*)wy;
    double* YT = Y + y_len;
    double* S = YT + y_len;
    double* T = S + nblk * NN * slabs;
    double* W = T + nblk * NN;
    {
      LaunchScope ls("eigh_wy_y", s);
      build_y_kernel<<<dim3(cdiv(p - 1, 256), WY_NB, (unsigned)nblk), 256, 0, s>>>(
          A, vhead, beta, p, in_rows, Y);
      SHRK_CUDA(cudaGetLastError());
    }
    {
      LaunchScope ls("dgemm_wy_yty", s);
      wy_gram_kernel<<<dim3((unsigned)nblk, (unsigned)slabs), 256, 0, s>>>(Y, p, S);
      SHRK_CUDA(cudaGetLastError());
    }
    {
      LaunchScope ls("eigh_wy_t", s);
      SHRK_CUDA(cudaFuncSetAttribute(wy_t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)wy_t_smem()));
      wy_t_kernel<<<dim3(WY_NB / WY_T_WARPS, (unsigned)nblk), WY_T_WARPS * 32, wy_t_smem(), s>>>(
          S, slabs, beta, p, T);
      SHRK_CUDA(cudaGetLastError());
    }
    {
      LaunchScope ls("dgemm_wy_yt", s);
      wy_yt_kernel<<<dim3(cdiv(p - 1, GT2), (unsigned)nblk), 256, 0, s>>>(Y, p, T, YT);
      SHRK_CUDA(cudaGetLastError());
    }
    for (int t = nblk - 1; t >= 0; --t) {
      const int64_t j0 = (int64_t)t * WY_NB, n = p - j0 - 1, off = wy_offset(p, t);
      const int64_t nb = std::min<int64_t>(WY_NB, nref - j0);
      double* Zs = Zc + (j0 + 1);  // rows j0+1 .. p-1 of Zc (leading dimension p)
      SHRK_TRY(dgemm(true, false, nb, p, n, 1.0, Y + off, n, Zs, p, 0.0, W, WY_NB, s,
                     "dgemm_wy_ytz"));  // W = Y^T Zs
      SHRK_TRY(dgemm(false, false, n, p, nb, -1.0, YT + off, n, W, WY_NB, 1.0, Zs, p, s,
                     "dgemm_wy_update"));  // Zs -= (Y T) W
    }
  }
  // ascending eigenvalues; eigenvector columns in that order, into A
  std::vector<int> hperm(p);
  std::iota(hperm.begin(), hperm.end(), 0);
  std::stable_sort(hperm.begin(), hperm.end(), [&](int x, int y) { return hl[x] < hl[y]; });
  for (int64_t k = 0; k < p; ++k) w_host[k] = hl[hperm[k]];
  SHRK_CUDA(cudaMemcpyAsync(perm, hperm.data(), sizeof(int) * p, cudaMemcpyHostToDevice, s));
  {
    LaunchScope ls("eigh_back_transform", s);
    permute_columns_kernel<<<dim3(cdiv(p, 256), (unsigned)p), 256, 0, s>>>(Zc, p, perm, A);
    SHRK_CUDA(cudaGetLastError());
  }
  SHRK_CUDA(cudaStreamSynchronize(s));
  return SHRK_OK;
}

}  // namespace shrk
