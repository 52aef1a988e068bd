// Exact all-points sums in FP64 with every unordered pair evaluated once.
//
// The pair term 1/((x - s) - i eta) = (d + i eta)/(d^2 + eta^2), d = x - s,
// changes only the sign of its real part when x and s swap (the symmetry the
// crate's sequential route uses, symmetric_sweep, cacheblock.rs:841-954), so
// one reciprocal serves two ordered pairs: 9 FP64 operations (d, d^2 + eta^2,
// 3 for the reciprocal, two accumulations at each end) for two pairs instead
// of 14.  What bounds it is the FP64 pipe.
//
// A warp holds 32*R targets in registers.  Over a block of 32 sources, lane l
// takes source l ^ k at step k and carries that source's column sums; between
// steps the sums move with the source they belong to (a shuffle by k ^ (k+1)),
// and after 32 steps each lane holds the finished sums of its own source.  The
// columns so cost no FP64 operation beyond the accumulations themselves (a
// reduction across lanes adds one per four pairs).
//
// Measured (B200, eta = 1/sqrt(p)): p = 50 000 0.77 ms (sums of all ordered
// pairs: 1.19), 1e6 298 ms (448), 0.81 and 0.83 of the FP64 pipe; the
// other issue slots go to the reciprocal seeds, the shuffles and the loads.
#include "common.cuh"
#include "epilogue.cuh"
#include "internal.h"
#include "pairs.cuh"
#include "pairsym.cuh"

#include <algorithm>

namespace shrk {

namespace {

constexpr int NT = SYM_NT;
constexpr int NW = NT / 32;

struct SymArgs {
  SymPlan pl;
  const double* ev;
  double eta2;
  double2* rows;  // [grid + tiles][tt]: row sums (re, iv) of each (CTA, tile)
  double2* cols;  // [tiles][p]: column sums (re, iv) of each tile
  int* err;
  int use_tma;            // ev is 16-byte aligned
  long long wait_cycles;  // budget of each bulk-copy wait
};

// The source chunks of one CTA, double-buffered: a whole chunk arrives by one
// bulk copy while the chunk before is summed.
struct SymStage {
  double s[2][SYM_CH];
  uint64_t bar[2];
};

struct SymRing {
  SymStage* st;
  uint32_t phase = 0u, pending = 0u;  // bit b: parity / copy in flight of buffer b

  __device__ __forceinline__ void init() {
    if (threadIdx.x == 0) {
      mbar_init(&st->bar[0], 1);
      mbar_init(&st->bar[1], 1);
      fence_mbar_init();
    }
    __syncthreads();
  }
  // Every thread calls it; buffer b is free.
  __device__ __forceinline__ void prefetch(const double* src, int b) {
    pending |= 1u << b;
    if (threadIdx.x == 0) {
      fence_proxy_async();
      mbar_arrive_expect_tx(&st->bar[b], SYM_CH * 8);
      bulk_g2s(st->s[b], src, SYM_CH * 8, &st->bar[b]);
    }
  }
  // Makes the chunk src[0..len) visible in buffer b; false (in every thread)
  // when its copy never completed: the timeout is recorded and the copies
  // still in flight are waited for, within their own budget.
  __device__ __forceinline__ bool ready(const double* src, int len, int b, int* err,
                                        long long wait_cycles) {
    bool ok = true;
    if ((pending >> b) & 1u) {
      ok = mbar_wait(&st->bar[b], (phase >> b) & 1u, wait_cycles);
    } else {
      const int i = threadIdx.x;
      st->s[b][i] = src[i < len ? i : 0];
    }
    if (!__syncthreads_and(ok)) {
      if (threadIdx.x == 0) {
        atomicExch(err, DEV_ERR_TIMEOUT);
        for (int q = 0; q < 2; ++q)
          if ((pending >> q) & 1u) mbar_wait(&st->bar[q], (phase >> q) & 1u, 200000000LL);
      }
      return false;
    }
    if ((pending >> b) & 1u) {
      phase ^= 1u << b;
      pending &= ~(1u << b);
    }
    return true;
  }
};

// One step: the source s against the thread's R targets, its sums in cre/civ.
template <int R, bool MASK>
__device__ __forceinline__ void sym_step(const double (&x)[R], double s, double eta2, bool on,
                                         double (&re)[R], double (&iv)[R], double& cre,
                                         double& civ) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double d = x[r] - s;
    double inv = rcp_f64(fma(d, d, eta2));
    if (MASK && !on) inv = 0.0;
    re[r] = fma(d, inv, re[r]);
    iv[r] += inv;
    cre = fma(d, inv, cre);
    civ += inv;
  }
}

// Adds a chunk's row sums to the thread's totals (shared memory: in registers
// they would cost the wide tiles their second CTA).
template <int R>
__device__ __forceinline__ void sym_fold(double2* tot, const double (&re)[R],
                                         const double (&iv)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    double2 t = tot[r * NT];
    t.x += re[r];
    t.y += iv[r];
    tot[r * NT] = t;
  }
}

template <int R>
__global__ void __launch_bounds__(NT, R == 1 ? 3 : 2) sym_sums_kernel(const SymArgs a) {
  __shared__ __align__(16) SymStage stage;
  extern __shared__ double2 dyn[];
  double2(*colw)[SYM_CH] = reinterpret_cast<double2(*)[SYM_CH]>(dyn);  // [NW][SYM_CH]
  double2* tot = dyn + NW * SYM_CH + threadIdx.x;                      // [R][NT]: row totals
  const SymPlan& pl = a.pl;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double eta2 = a.eta2;
  SymRing ring{&stage};
  ring.init();
  const int64_t base0 = pl.before(pl.t0);
  int64_t u = pl.first_unit(blockIdx.x);
  const int64_t u_end = pl.first_unit(blockIdx.x + 1);
  int T = pl.tile_of(u);
  for (; u < u_end; ++T) {
    const int64_t ub = pl.before(T) - base0;
    const int64_t seg_end = min(u_end, pl.before(T + 1) - base0);
    const int64_t tile0 = (int64_t)T * pl.tt, wbase = tile0 + (int64_t)warp * (32 * R);
    const int64_t diag_end = min(pl.p, tile0 + pl.tt);
    const int64_t s0 = tile0 + (u - ub) * SYM_UB;
    const int64_t s1 = min(pl.p, tile0 + (seg_end - ub) * SYM_UB);
    double x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t idx = wbase + r * 32 + lane;
      x[r] = idx < pl.p ? a.ev[idx] : a.ev[tile0];
      tot[r * NT] = make_double2(0.0, 0.0);
    }
    // the chunk at cs: up to SYM_CH sources, all inside the tile or all after it
    auto chunk_len = [&](int64_t cs) {
      return (int)min((int64_t)SYM_CH, (cs < diag_end ? min(s1, diag_end) : s1) - cs);
    };
    auto fetch = [&](int64_t cs, int b) {
      if (a.use_tma && cs < s1 && chunk_len(cs) == SYM_CH) ring.prefetch(a.ev + cs, b);
    };
    __syncthreads();  // the last tile's readers are done with both buffers
    fetch(s0, 0);
    int len = 0, buf = 0;
    for (int64_t cs = s0; cs < s1; cs += len, buf ^= 1) {
      const bool diag = cs < diag_end;
      len = chunk_len(cs);
      if (!ring.ready(a.ev + cs, len, buf, a.err, a.wait_cycles)) return;
      fetch(cs + len, buf ^ 1);  // its readers passed the barrier in ready()
      const double* ss = stage.s[buf];
      // Rows are summed chunk by chunk: one running sum over the ~1e6 sources
      // of a large spectrum would lose a digit to rounding.
      double re[R], iv[R];
#pragma unroll
      for (int r = 0; r < R; ++r) re[r] = iv[r] = 0.0;
      if (diag) {
        // the tile against itself: full square, rows only
#pragma unroll 4
        for (int j = 0; j < len; ++j) {
          const double s = ss[j];
#pragma unroll
          for (int r = 0; r < R; ++r) pair64(x[r], s, eta2, re[r], iv[r]);
        }
        sym_fold<R>(tot, re, iv);
        continue;
      }
      // A tile with columns is full: no padded target reaches them.
      int b = 0;
      for (; b + 64 <= len; b += 64) {
        double c0 = 0.0, v0 = 0.0, c1 = 0.0, v1 = 0.0;
#pragma unroll 2
        for (int g = 0; g < 32; g += 8) {
          const int at = lane ^ g, turn = (g & 8) ? 31 : 15;  // (g + 7) ^ (g + 8)
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const double* q = &ss[b + (at ^ k)];
            sym_step<R, false>(x, q[0], eta2, true, re, iv, c0, v0);
            sym_step<R, false>(x, q[32], eta2, true, re, iv, c1, v1);
            const int m = k < 7 ? k ^ (k + 1) : turn;
            c0 = __shfl_xor_sync(0xffffffffu, c0, m);
            v0 = __shfl_xor_sync(0xffffffffu, v0, m);
            c1 = __shfl_xor_sync(0xffffffffu, c1, m);
            v1 = __shfl_xor_sync(0xffffffffu, v1, m);
          }
        }
        colw[warp][b + lane] = make_double2(c0, v0);
        colw[warp][b + 32 + lane] = make_double2(c1, v1);
      }
      for (; b < len; b += 32) {  // the spectrum's end: sources past it masked
        double c0 = 0.0, v0 = 0.0;
#pragma unroll 1
        for (int k = 0; k < 32; ++k) {
          const int j = b + (lane ^ k);
          sym_step<R, true>(x, ss[j], eta2, j < len, re, iv, c0, v0);
          c0 = __shfl_xor_sync(0xffffffffu, c0, (k ^ (k + 1)) & 31);
          v0 = __shfl_xor_sync(0xffffffffu, v0, (k ^ (k + 1)) & 31);
        }
        colw[warp][b + lane] = make_double2(c0, v0);
      }
      sym_fold<R>(tot, re, iv);
      __syncthreads();
      if (tid < len) {
        double c = 0.0, v = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          const double2 q = colw[w][tid];
          c += q.x;
          v += q.y;
        }
        a.cols[(int64_t)(T - pl.t0) * pl.p + cs + tid] = make_double2(-c, v);
      }
    }
    double2* row = a.rows + (int64_t)(blockIdx.x + T - pl.t0) * pl.tt;
#pragma unroll
    for (int r = 0; r < R; ++r)
      row[warp * (32 * R) + r * 32 + lane] = tot[r * NT];
    u = seg_end;
  }
}

struct SymReduceArgs {
  SymPlan pl;
  const double* ev;
  const double2* rows;
  const double2* cols;
  double2* acc;       // sums of the earlier phases (null: a single phase)
  bool first, last;
  double eta;
  Epilogue epi;
};

// The phase's sums of 32 targets a CTA; the last phase applies the epilogue.
__global__ void __launch_bounds__(NT) sym_reduce_kernel(const SymReduceArgs a) {
  const int64_t t0 = (int64_t)blockIdx.x * 32, t = t0 + (threadIdx.x & 31);
  const double2 q = sym_collect(a.pl, a.rows, a.cols, a.first ? nullptr : a.acc, t0);
  if (threadIdx.x >= 32 || t >= a.pl.p) return;
  if (a.last) epi_store(a.epi, t, a.ev[t], q.x, a.eta * q.y);
  else a.acc[t] = q;
}

template <int R>
shrk_status launch_sums(const SymArgs& a, cudaStream_t s) {
  constexpr int bytes = (int)sizeof(double2) * (NW * SYM_CH + R * NT);
  SHRK_CUDA(cudaFuncSetAttribute(sym_sums_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 bytes));
  sym_sums_kernel<R><<<a.pl.grid, NT, bytes, s>>>(a);
  SHRK_CUDA(cudaGetLastError());
  return SHRK_OK;
}

}  // namespace

shrk_status sym_sums(const double* d_ev, int64_t p, double eta, const Epilogue& epi,
                     cudaStream_t s) {
  // Targets per thread, measured (sums + reduction, us on the device, for
  // R = 1 / 2 / 4): p = 1024 10 / 11 / 13, 3000 19 / 18 / 18, 4096 19 / 17 /
  // 21, 7001 34 / 31 / 33, 10000 58 / 51 / 48, 50000 1034 / 820 / 770: wide
  // tiles share each rotation among more pairs, narrow ones make enough units.
  // (R = 8 in 128 registers: 790 at 50000.)
  const int R = p >= 8192 ? 4 : p >= 3072 ? 2 : 1;
  const int ctas = sm_count() * (R == 1 ? 3 : 2);
  const int tt = NT * R;
  const int n_tiles = (int)((p + tt - 1) / tt);
  // Tiles of a phase: as many column slabs as 256 MB hold, scratch that the
  // context keeps (64 MB, with a reduction more often: 3.01 ms for 2.98 at p =
  // 100 003, 48.1 for 47.4 at 400 000, 306 for 298 at 1e6).
  const int64_t per = std::max<int64_t>(1, ((int64_t)256 << 20) / ((int64_t)sizeof(double2) * p));
  const int phase = (int)std::min<int64_t>(n_tiles, per);
  const size_t row_bytes = sizeof(double2) * (size_t)(ctas + phase) * tt;
  const size_t acc_bytes = phase < n_tiles ? sizeof(double2) * (size_t)p : 0;
  void* buf = nullptr;
  SHRK_TRY(scratch_get(0, row_bytes + acc_bytes + sizeof(double2) * (size_t)phase * (size_t)p,
                       &buf));
  SymArgs a;
  a.ev = d_ev;
  a.eta2 = eta * eta;
  a.err = device_error_word();
  a.use_tma = ((uintptr_t)d_ev % 16 == 0) ? 1 : 0;
  a.wait_cycles = wait_cycles();
  a.rows = (double2*)buf;
  a.cols = (double2*)((char*)buf + row_bytes + acc_bytes);
  SymReduceArgs ra;
  ra.ev = d_ev;
  ra.rows = a.rows;
  ra.cols = a.cols;
  ra.acc = (double2*)((char*)buf + row_bytes);
  ra.eta = eta;
  ra.epi = epi;
  for (int t0 = 0; t0 < n_tiles; t0 += phase) {
    a.pl = sym_plan(p, tt, t0, std::min(n_tiles, t0 + phase), ctas);
    {
      LaunchScope ls("pair_sum_f64", s);
      if (R == 4) SHRK_TRY(launch_sums<4>(a, s));
      else if (R == 2) SHRK_TRY(launch_sums<2>(a, s));
      else SHRK_TRY(launch_sums<1>(a, s));
    }
    ra.pl = a.pl;
    ra.first = t0 == 0;
    ra.last = a.pl.t1 == n_tiles;
    LaunchScope ls("split_reduce", s);
    sym_reduce_kernel<<<(unsigned)((p + 31) / 32), NT, 0, s>>>(ra);
    SHRK_CUDA(cudaGetLastError());
  }
  return SHRK_OK;
}

}  // namespace shrk
