// The treecode's tree of a larger spectrum, built subtree by subtree (part of
// chebcode.cu, included inside its namespace).
//
// A launch per level spent its time on launches and dependent loads, not on
// work: at p = 1e6 23 split launches took 187 us and 19 M2M launches 199 us.
// Here the topology and the weights take three launches:
//   1. top_tree_kernel (one CTA): splits nodes until they hold at most S
//      sources (or are leaves); each of those roots a subtree.  The searches
//      start on every (ns/12000)-th source, kept in shared memory, and end
//      with one window of loads, so a level costs two memory round trips.
//   2. sub_topology_kernel (a CTA per subtree): splits on in shared memory,
//      local breadth-first order, and counts leaves.  The tree is full, so a
//      node after B leaves in source order, at depth D and after R right
//      turns on its path, sits at pre-order index D + 2 B - R; the counts of
//      the subtrees before give B.
//   3. sub_weights_kernel (a CTA per subtree): flat arrays, P2M, M2M level by
//      level with a barrier in between, f32 mirror; then the CTA's first warp
//      climbs: of two sibling subtrees the one to finish last (an arrival
//      count after a fence; nobody waits) merges their parent, and so on up.
// Split points, rows and the order of every accumulation are those of the
// level-by-level build (tree_split_node, bary_rows_batch), so the tree is the
// same bit for bit.  Up to three charge sets share the rows' quotients.
#pragma once

constexpr int SUB_S_MAX = 2048;    // most sources of a subtree with inner nodes
constexpr int SUB_S_MIN = 512;
constexpr int SUB_NT = 256;
constexpr int TOP_NT = 1024;
constexpr int TOP_COARSE = 12000;  // sources of the coarse search table
constexpr int TOP_FRONT = 2048;    // nodes still to split on one level: ns / S
constexpr int64_t SUB_MAX_NS = (int64_t)TOP_FRONT * SUB_S_MAX;
constexpr int SUB_REC = 512;        // node records staged in shared memory
constexpr int SUB_LEVELS = MAX_TREE_DEPTH + 2;

// Sources of a subtree: several hundred subtrees, whose uneven sizes then
// average out over the SMs (with subtrees of 4 096 at p = 1e6, 375 CTAs, the SM
// with the most work had 2.8 times the mean).
inline int sub_sources(int64_t ns) {
  int S = SUB_S_MIN;
  while (S < SUB_S_MAX && ns / S > 512) S *= 2;
  return S;
}

struct SubArrays {
  // top nodes by breadth-first slot; rc = lc + 1, lc < 0: a subtree's root; t_up:
  // parent (-1: none), t_arrive: children finished
  int *t_lo, *t_hi, *t_lc, *t_dep, *t_rt, *t_up, *t_arrive;
  double* t_rec;              // [top node][3 + NS n]: range, pre-order index, node weights
  int *s_slot, *s_lo, *s_leaves;
  uint16_t* s_lev;            // [subtree][SUB_LEVELS]: local level starts
  uint2* rec;                 // subtree at source lo: nodes from rec[2 lo], local order:
                              // x = lo | hi << 16 (offsets), y = lc | pre << 16 (lc 0: leaf)
  int* count;                 // [0] top nodes, [1] subtrees, [2] leaves
};

struct TopNode {
  double lov, hiv;  // first and last source
  int lo, hi, slot, rt;
};

constexpr size_t TOP_SMEM = sizeof(double) * TOP_COARSE + sizeof(TopNode) * 2 * TOP_FRONT;

__global__ void __launch_bounds__(TOP_NT, 1) top_tree_kernel(const double* __restrict__ sorted,
                                                             int ns, int leaf_cap, int S,
                                                             SubArrays a) {
  extern __shared__ __align__(16) unsigned char top_sm[];
  double* coarse = reinterpret_cast<double*>(top_sm);
  TopNode* front = reinterpret_cast<TopNode*>(coarse + TOP_COARSE);
  __shared__ int n_top, n_sub, n_next;
  constexpr int GL = 8;  // lanes per node
  const int tid = threadIdx.x, gl = tid % GL;
  // the first 32 nodes of a level go to 32 warps
  const int grp = (tid >> 5) + (TOP_NT / 32) * ((tid & 31) / GL);
  const unsigned gmask = 0xffu << (tid & 24);
  const int g = (ns + TOP_COARSE - 1) / TOP_COARSE, nc = (ns + g - 1) / g;
  const int most = max(S, leaf_cap);
  for (int i = tid; i < nc; i += TOP_NT) coarse[i] = sorted[(int64_t)i * g];
  // a node goes to the frontier (to be split here) or roots a subtree
  auto place = [&](int slot, int up, int lo, int hi, int depth, int rt, double lov, double hiv,
                   TopNode* next) {
    a.t_lo[slot] = lo;
    a.t_hi[slot] = hi;
    a.t_dep[slot] = depth;
    a.t_rt[slot] = rt;
    a.t_up[slot] = up;
    a.t_arrive[slot] = 0;
    if (hi - lo > most && depth < MAX_TREE_DEPTH) {
      next[atomicAdd(&n_next, 1)] = TopNode{lov, hiv, lo, hi, slot, rt};
    } else {
      const int s = atomicAdd(&n_sub, 1);
      a.t_lc[slot] = -1;
      a.s_slot[s] = slot;
      a.s_lo[s] = lo;
    }
  };
  if (tid == 0) {
    n_top = 1;
    n_sub = n_next = 0;
    place(0, -1, 0, ns, 0, 0, sorted[0], sorted[ns - 1], front);
  }
  __syncthreads();
  int depth = 0, n = n_next;
  for (; n > 0; ++depth) {
    __syncthreads();  // every thread has read n_next
    if (tid == 0) n_next = 0;
    __syncthreads();
    const TopNode* cur = front + (depth & 1) * TOP_FRONT;
    TopNode* next = front + ((depth + 1) & 1) * TOP_FRONT;
    for (int w = grp; w < n; w += TOP_NT / GL) {
      const TopNode e = cur[w];
      const double mid = e.lov + 0.5 * (e.hiv - e.lov);
      // first coarse source of the node above mid, then the window before it
      const int c0 = e.lo / g + 1, c1 = (e.hi - 1) / g + 1;
      int x = c0, y = c1;
      while (x < y) {  // a group's lanes probe 8 positions a round
        const int span = y - x, m = x + (int)(((unsigned)span * (2 * gl + 1)) >> 4);
        const unsigned up = __ballot_sync(gmask, mid < coarse[m]) >> (tid & 24) & 0xffu;
        const int f = up ? __ffs(up) - 1 : GL;  // first probe above mid
        const int below = x + (int)(((unsigned)span * (2 * f - 1)) >> 4);
        if (f < GL) y = x + (int)(((unsigned)span * (2 * f + 1)) >> 4);
        if (f > 0) x = below + 1;
      }
      const int from = x > c0 ? (x - 1) * g + 1 : e.lo, to = x < c1 ? x * g : e.hi;
      int split = to;
      for (int b = from; b < to && split == to; b += 12 * GL) {
        unsigned gt = 0;  // bit u: source b + u GL + gl is above mid
#pragma unroll
        for (int u = 0; u < 12; ++u) {
          const int i = b + u * GL + gl;
          if (i < to && mid < sorted[i]) gt |= 1u << u;
        }
        int first = gt ? b + (__ffs(gt) - 1) * GL + gl : to;
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(gmask, first, o));
        split = first;
      }
      if (split == e.lo || split == e.hi) split = (int)(((int64_t)e.lo + e.hi) / 2);
      if (gl < 2) {  // lane 0: the left child, lane 1: the right one
        const double edge = sorted[split - 1 + gl];
        int slot = 0;
        if (gl == 0) slot = atomicAdd(&n_top, 2);
        slot = __shfl_sync(3u << (tid & 24), slot, tid & 24);
        if (gl == 0) a.t_lc[e.slot] = slot;
        place(slot + gl, e.slot, gl ? split : e.lo, gl ? e.hi : split, depth + 1, e.rt + gl,
              gl ? edge : e.lov, gl ? e.hiv : edge, next);
      }
    }
    __syncthreads();
    n = n_next;
  }
  if (tid == 0) {
    a.count[0] = n_top;
    a.count[1] = n_sub;
    a.count[2] = 0;
  }
}

inline size_t sub_topo_bytes(int S) {
  return sizeof(double) * S + sizeof(uint16_t) * (3 * 2 * S + S) + 2 * S;
}

__global__ void __launch_bounds__(SUB_NT) sub_topology_kernel(const double* __restrict__ sorted,
                                                              int leaf_cap, int S, SubArrays a) {
  extern __shared__ __align__(16) unsigned char sub_sm[];
  struct {
    double* src;
    uint16_t *lo, *hi, *lc, *before;  // before: leaf starts, then leaves before each source
    uint8_t* rt;
  } t;
  t.src = reinterpret_cast<double*>(sub_sm);
  t.lo = reinterpret_cast<uint16_t*>(t.src + S);
  t.hi = t.lo + 2 * S;
  t.lc = t.hi + 2 * S;
  t.before = t.lc + 2 * S;
  t.rt = reinterpret_cast<uint8_t*>(t.before + S);
  __shared__ uint16_t lev[SUB_LEVELS];
  __shared__ int warp_sum[SUB_NT / 32], n_nodes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_sub = a.count[1];
  for (int s = blockIdx.x; s < n_sub; s += gridDim.x) {
    const int slot = a.s_slot[s], lo0 = a.t_lo[slot], cnt = a.t_hi[slot] - lo0;
    const int d0 = a.t_dep[slot];
    if (cnt <= leaf_cap || d0 >= MAX_TREE_DEPTH) {  // a single leaf, of any size
      if (tid == 0) {
        a.s_leaves[s] = 1;
        atomicAdd(&a.count[2], 1);
      }
      continue;
    }
    __syncthreads();  // the previous subtree's readers are done
    for (int i = tid; i < cnt; i += SUB_NT) {
      t.src[i] = sorted[lo0 + i];
      t.before[i] = 0;
    }
    if (tid == 0) {
      t.lo[0] = 0;
      t.hi[0] = (uint16_t)cnt;
      t.rt[0] = 0;
      n_nodes = 1;
      lev[0] = 0;
    }
    __syncthreads();
    int begin = 0, end = 1, L = 0;
    for (; begin < end; ++L) {
      for (int i = begin + tid; i < end; i += SUB_NT) {
        const int lo = t.lo[i], hi = t.hi[i];
        int lc = 0;
        if (hi - lo > leaf_cap && d0 + L < MAX_TREE_DEPTH) {
          const double lov = t.src[lo], mid = lov + 0.5 * (t.src[hi - 1] - lov);
          int x = lo, y = hi;  // upper_bound: first element > mid
          while (x < y) {
            const int m = (x + y) >> 1;
            if (mid < t.src[m]) y = m;
            else x = m + 1;
          }
          if (x == lo || x == hi) x = (int)(((int64_t)lo0 * 2 + lo + hi) / 2 - lo0);
          lc = atomicAdd(&n_nodes, 2);
          t.lo[lc] = (uint16_t)lo;
          t.hi[lc] = t.lo[lc + 1] = (uint16_t)x;
          t.hi[lc + 1] = (uint16_t)hi;
          t.rt[lc] = t.rt[i];
          t.rt[lc + 1] = t.rt[i] + 1;
        } else {
          t.before[lo] = 1;
        }
        t.lc[i] = (uint16_t)lc;
      }
      __syncthreads();
      begin = end;
      end = n_nodes;
      if (tid == 0) lev[L + 1] = (uint16_t)begin;
      __syncthreads();
    }
    // L levels; exclusive prefix of the leaf starts, a run of PER a thread
    constexpr int PER = SUB_S_MAX / SUB_NT;
    int mine[PER], sum = 0;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = tid * PER + u;
      mine[u] = sum;
      sum += i < cnt ? t.before[i] : 0;
    }
    int scan = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += v;
    }
    if (lane == 31) warp_sum[warp] = scan;
    __syncthreads();
    int base = scan - sum, total = 0;
    for (int w = 0; w < SUB_NT / 32; ++w) {
      if (w < warp) base += warp_sum[w];
      total += warp_sum[w];
    }
#pragma unroll
    for (int u = 0; u < PER; ++u)
      if (tid * PER + u < cnt) t.before[tid * PER + u] = (uint16_t)(base + mine[u]);
    __syncthreads();
    uint2* rec = a.rec + 2 * (int64_t)lo0;
    for (int l = 0; l < L; ++l)
      for (int i = lev[l] + tid; i < lev[l + 1]; i += SUB_NT) {
        const unsigned pre = l + 2 * t.before[t.lo[i]] - t.rt[i];
        rec[i] = make_uint2(t.lo[i] | (unsigned)t.hi[i] << 16, t.lc[i] | pre << 16);
      }
    for (int l = tid; l <= L; l += SUB_NT) a.s_lev[(int64_t)s * SUB_LEVELS + l] = lev[l];
    if (tid == 0) {
      if (L + 1 < SUB_LEVELS) a.s_lev[(int64_t)s * SUB_LEVELS + L + 1] = 0xffff;  // no more levels
      a.s_leaves[s] = total;
      atomicAdd(&a.count[2], total);
    }
  }
}

// Barycentric rows as bary_rows_batch, N nodes and NS masses a row: the
// quotients and the row's scale 1/sum do not depend on the mass, so they are
// shared; `on` has bit c set where the row applies to set c.  lam is +-1 or
// +-1/2, so lam * (1/d) is the rounded quotient lam / d, and with N known the
// N branch-free reciprocals of a row are in flight together.  (Both ends of a
// node's range are Chebyshev nodes, so most batches hold exact hits.)  A batch
// with a value outside their range takes the plain loop.
template <int N, int NS>
struct RowSet {
  static constexpr int ST = N | 1;  // row stride
  double q[32 * ST];
  double t[N];
  double m[NS][32];
  int code[32];  // on | (hit + 1) << 8
};

template <int N, int NS>
__device__ __forceinline__ void bary_rows_set(double x, const double (&mass)[NS], int on, int cnt,
                                              const ChebConsts& k, int lane, RowSet<N, NS>& rs,
                                              double (&w)[NS]) {
  constexpr int ST = RowSet<N, NS>::ST;
  bool plain = true;
  {
    double q[N], sum = 0.0;
    int hit = -1;
#pragma unroll
    for (int j = N - 1; j >= 0; --j) {
      const double d = x - rs.t[j];
      plain = plain && row_mid(d);
      if (((__double2hiint(d) & 0x7fffffff) | __double2loint(d)) == 0) hit = j;  // the first counts
      // lam_j = (-1)^j, halved at both ends
      double r = rcp_rn_mid(fabs(d));
      if (j == 0 || j == N - 1) r *= 0.5;
      q[j] = copysign(r, (j & 1) ? -d : d);
    }
#pragma unroll
    for (int j = 0; j < N; ++j) sum += q[j];
    const double scale = rcp_rn_signed(sum);
    // a hit's row is its mass times the hit node's unit vector
    plain = !on || hit >= 0 || (plain && row_mid(sum));
#pragma unroll
    for (int j = 0; j < N; ++j)
      rs.q[lane * ST + j] = !on ? 0.0 : hit < 0 ? q[j] : j == hit ? 1.0 : 0.0;
#pragma unroll
    for (int c = 0; c < NS; ++c)
      rs.m[c][lane] = !on ? 0.0 : hit < 0 ? mass[c] * scale : mass[c];
  }
  plain = __all_sync(0xffffffffu, plain);
  __syncwarp();
  const int j = lane < N ? lane : 0;
  if (plain) {
    // A row that does not apply has zero mass and quotients (or, in a set
    // whose mass is zero, a zero mass and finite quotients): it adds +0.
    for (int r0 = 0; r0 < cnt; r0 += 8) {
      double qq[8], mm[8][NS];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        qq[u] = rs.q[(r0 + u) * ST + j];
#pragma unroll
        for (int c = 0; c < NS; ++c) mm[u][c] = rs.m[c][r0 + u];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int c = 0; c < NS; ++c) w[c] = fma(mm[u][c], qq[u], w[c]);
    }
  } else {
    int hit = -1;
    if (on) {
      double sum = 0.0;
      for (int i = 0; i < N; ++i) {
        const double d = x - rs.t[i];
        if (d == 0.0 && hit < 0) hit = i;
        const double q = k.lam[i] / d;
        rs.q[lane * ST + i] = q;
        sum += q;
      }
#pragma unroll
      for (int c = 0; c < NS; ++c) rs.m[c][lane] = hit >= 0 ? mass[c] : mass[c] * (1.0 / sum);
    }
    rs.code[lane] = on ? on | (hit + 1) << 8 : 0;
    __syncwarp();
    for (int r = 0; r < cnt; ++r) {
      const int code = rs.code[r], at = (code >> 8) - 1;
      const double q = rs.q[r * ST + j];
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        if (!((code >> c) & 1)) continue;
        if (at < 0) w[c] = fma(rs.m[c][r], q, w[c]);
        else if (at == lane) w[c] = w[c] + rs.m[c][r];
      }
    }
  }
  __syncwarp();  // the tile is rewritten by the next batch
}

template <int NS>
struct SubCharges {
  const double* c[NS];  // per sorted source; c[0] null: unit masses
  double* w[NS];        // node weights [nn][n]
};

// P2M of the leaf over src[0..cnt) (charges from source index g0) into node idx.
template <int N, int NS>
__device__ __forceinline__ void p2m_set(const double* src, int64_t g0, int64_t cnt, double lo,
                                        double hi, int64_t idx, const SubCharges<NS>& ch,
                                        const ChebConsts& k, const double* sm1, int lane,
                                        RowSet<N, NS>& rs) {
  const double c = 0.5 * (lo + hi), l = 0.5 * (hi - lo);
  if (lane < N) rs.t[lane] = c + l * sm1[lane];
  __syncwarp();
  double w[NS] = {};
  for (int64_t q0 = 0; q0 < cnt; q0 += 32) {
    const int m = (int)min((int64_t)32, cnt - q0);
    const bool in = lane < m;
    const double x = in ? src[q0 + lane] : 0.0;
    double mass[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)
      mass[s] = in ? (ch.c[s] ? ch.c[s][g0 + q0 + lane] : 1.0) : 0.0;
    bary_rows_set<N, NS>(x, mass, in ? (1 << NS) - 1 : 0, m, k, lane, rs, w);
  }
#pragma unroll
  for (int s = 0; s < NS; ++s)
    if (lane < N) ch.w[s][idx * N + lane] = w[s];
}

// M2M of node idx over [lo, hi]: its children (flat indices kid, over
// [klo, khi], per lane: the left child for lanes below N, the right above).
template <int N, int NS>
__device__ __forceinline__ void m2m_set(double lo, double hi, int64_t idx, double klo, double khi,
                                        int64_t kid, const SubCharges<NS>& ch,
                                        const ChebConsts& k, const double* sm1, int lane,
                                        RowSet<N, NS>& rs) {
  const double c = 0.5 * (lo + hi), l = 0.5 * (hi - lo);
  if (lane < N) rs.t[lane] = c + l * sm1[lane];
  __syncwarp();
  double x = 0.0, mass[NS] = {}, w[NS] = {};
  int on = 0;
  if (lane < 2 * N) {
    const int ti = lane < N ? lane : lane - N;
    const double kc = 0.5 * (klo + khi), kl = 0.5 * (khi - klo);
    x = kc + kl * sm1[ti];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      mass[s] = ch.w[s][kid * N + ti];
      if (mass[s] != 0.0) on |= 1 << s;
    }
  }
  bary_rows_set<N, NS>(x, mass, on, 2 * N, k, lane, rs, w);
#pragma unroll
  for (int s = 0; s < NS; ++s)
    if (lane < N) ch.w[s][idx * N + lane] = w[s];
}

__device__ __forceinline__ void fill_flat(const FlatTree& f, int64_t idx, double lo, double hi,
                                          int64_t lo_idx, int64_t hi_idx, int right,
                                          double theta_sq) {
  f.lo[idx] = lo;
  f.hi[idx] = hi;
  const double hw = 0.5 * (hi - lo);
  f.accept_hw[idx] = hw * hw / theta_sq;
  f.lo_idx[idx] = lo_idx;
  f.hi_idx[idx] = hi_idx;
  f.right[idx] = right;
}

template <int N, int NS>
__global__ void __launch_bounds__(SUB_NT, 4) sub_weights_kernel(
    const double* __restrict__ sorted, int leaf_cap, int S, SubArrays a, FlatTree f,
    SubCharges<NS> ch, ChebConsts k, double theta_sq, NodeF32* nf, float* panel) {
  extern __shared__ __align__(16) unsigned char sub_sm[];
  double* src = reinterpret_cast<double*>(sub_sm);
  __shared__ uint16_t lev[SUB_LEVELS];
  __shared__ uint2 rec_s[SUB_REC];
  __shared__ double sm1[N];
  __shared__ int part[SUB_NT / 32], n_lev;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  RowSet<N, NS>& rs = reinterpret_cast<RowSet<N, NS>*>(src + S)[warp];
  const int s = blockIdx.x, n_sub = a.count[1];
  int slot = a.s_slot[s];
  const int lo0 = a.t_lo[slot], cnt = a.t_hi[slot] - lo0, d0 = a.t_dep[slot];
  // leaves before this subtree's sources
  int b = 0;
  for (int i = tid; i < n_sub; i += SUB_NT)
    if (a.s_lo[i] < lo0) b += a.s_leaves[i];
  b = __reduce_add_sync(0xffffffffu, b);
  if (lane == 0) part[warp] = b;
  if (tid < N) sm1[tid] = k.sm1[tid];
  const bool leaf = cnt <= leaf_cap || d0 >= MAX_TREE_DEPTH;
  if (!leaf) {
    for (int i = tid; i < cnt; i += SUB_NT) src[i] = sorted[lo0 + i];
    if (tid < SUB_LEVELS) lev[tid] = a.s_lev[(int64_t)s * SUB_LEVELS + tid];
  }
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int w = 0; w < SUB_NT / 32; ++w) before += part[w];
  const int64_t root = d0 + 2 * (int64_t)before - a.t_rt[slot];
  if (leaf) {
    const double lo = sorted[lo0], hi = sorted[lo0 + cnt - 1];
    if (tid == 0) fill_flat(f, root, lo, hi, lo0, (int64_t)lo0 + cnt, -1, theta_sq);
    if (tid < N) f.nodes[root * N + tid] = 0.5 * (lo + hi) + 0.5 * (hi - lo) * sm1[tid];
    if (warp == 0) {
      p2m_set<N, NS>(sorted + lo0, lo0, cnt, lo, hi, root, ch, k, sm1, lane, rs);
      __syncwarp();
      if (nf) mirror_f32(f, (int)root, N, lane, nf, panel);
    }
  } else {
    if (tid == 0) {
      int l = 1;
      while (l + 1 < SUB_LEVELS && lev[l + 1] != 0xffff) ++l;
      n_lev = l;  // levels 0 .. l - 1; lev[l] = nodes
    }
    __syncthreads();
    const int levels = n_lev, nn = lev[levels];
    // the node records, in shared memory unless there are very many
    const uint2* rec = a.rec + 2 * (int64_t)lo0;
    if (nn <= SUB_REC) {
      for (int i = tid; i < nn; i += SUB_NT) rec_s[i] = rec[i];
      __syncthreads();
      rec = rec_s;
    }
    // P2M first: the longest chains of work start at once
    for (int i = warp; i < nn; i += SUB_NT / 32) {
      const uint2 r = rec[i];
      if (r.y & 0xffff) continue;
      const int lo = r.x & 0xffff, hi = r.x >> 16;
      p2m_set<N, NS>(src + lo, (int64_t)lo0 + lo, hi - lo, src[lo], src[hi - 1],
                     root + (r.y >> 16), ch, k, sm1, lane, rs);
    }
    for (int i = tid; i < nn; i += SUB_NT) {
      const uint2 r = rec[i];
      const int lo = r.x & 0xffff, hi = r.x >> 16, lc = r.y & 0xffff;
      fill_flat(f, root + (r.y >> 16), src[lo], src[hi - 1], (int64_t)lo0 + lo,
                (int64_t)lo0 + hi, lc ? (int)(root + (rec[lc + 1].y >> 16)) : -1, theta_sq);
    }
    for (int e = tid; e < nn * N; e += SUB_NT) {
      const int i = e / N, j = e - i * N;
      const uint2 r = rec[i];
      const double lo = src[r.x & 0xffff], hi = src[(r.x >> 16) - 1];
      f.nodes[(root + (r.y >> 16)) * N + j] = 0.5 * (lo + hi) + 0.5 * (hi - lo) * sm1[j];
    }
    for (int l = levels - 2; l >= 0; --l) {
      __syncthreads();
      for (int i = lev[l] + warp; i < lev[l + 1]; i += SUB_NT / 32) {
        const uint2 r = rec[i];
        const int lc = r.y & 0xffff;
        if (!lc) continue;
        const uint2 kr = rec[lane < N ? lc : lc + 1];
        m2m_set<N, NS>(src[r.x & 0xffff], src[(r.x >> 16) - 1], root + (r.y >> 16),
                              src[kr.x & 0xffff], src[(kr.x >> 16) - 1], root + (kr.y >> 16), ch,
                              k, sm1, lane, rs);
      }
    }
    if (nf) {
      __syncthreads();
      for (int i = warp; i < nn; i += SUB_NT / 32)
        mirror_f32(f, (int)(root + (rec[i].y >> 16)), N, lane, nf, panel);
    }
  }
  if (warp != 0) return;
  // Up the top tree.  Warp 0 did (or passed a barrier after) the root's
  // weights.  In pre-order a left child follows its parent, so the parent's
  // index and range come from its children's; each finished top node leaves
  // them and its weights in one record (slot pairs are (odd, even)), so that a
  // merge waits for one load after the count.
  constexpr int TW = 3 + NS * N;
  int64_t idx = root;
  double lo = sorted[lo0], hi = sorted[lo0 + cnt - 1], w[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) w[c] = lane < N ? ch.w[c][idx * N + lane] : 0.0;
  for (int up = a.t_up[slot]; up >= 0;) {
    double* mine = a.t_rec + (int64_t)slot * TW;
    if (lane == 0) {
      mine[0] = lo;
      mine[1] = hi;
      mine[2] = (double)idx;
    }
#pragma unroll
    for (int c = 0; c < NS; ++c)
      if (lane < N) mine[3 + c * N + lane] = w[c];
    const int next_up = a.t_up[up], up_lo = a.t_lo[up], up_hi = a.t_hi[up];
    __threadfence();  // this node's record before the count
    __syncwarp();
    int seen = 0;
    if (lane == 0) seen = atomicAdd(&a.t_arrive[up], 1);
    seen = __shfl_sync(0xffffffffu, seen, 0);
    if (seen == 0) return;  // the sibling's warp merges the parent
    __threadfence();
    const bool is_left = slot & 1;
    const double* other = a.t_rec + (int64_t)(is_left ? slot + 1 : slot - 1) * TW;
    const double o_lo = __ldcg(other), o_hi = __ldcg(other + 1), o_idx = __ldcg(other + 2);
    const int ti = lane < N ? lane : lane - N;
    const bool from_left = lane < N, own = from_left == is_left;
    double mass[NS];
    int on = 0;
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      const double o = lane < 2 * N ? __ldcg(other + 3 + c * N + ti) : 0.0;
      const double m = __shfl_sync(0xffffffffu, w[c], ti & 31);
      mass[c] = lane < 2 * N ? (own ? m : o) : 0.0;
      if (mass[c] != 0.0) on |= 1 << c;
    }
    const double llo = is_left ? lo : o_lo, lhi = is_left ? hi : o_hi;
    const double rlo = is_left ? o_lo : lo, rhi = is_left ? o_hi : hi;
    const int64_t right = is_left ? (int64_t)o_idx : idx;
    idx = (is_left ? idx : (int64_t)o_idx) - 1;
    lo = llo;
    hi = rhi;
    const double pc = 0.5 * (lo + hi), pl = 0.5 * (hi - lo);
    if (lane == 0) fill_flat(f, idx, lo, hi, up_lo, up_hi, (int)right, theta_sq);
    if (lane < N) {
      rs.t[lane] = pc + pl * sm1[lane];
      f.nodes[idx * N + lane] = rs.t[lane];
    }
    __syncwarp();
    const double klo = from_left ? llo : rlo, khi = from_left ? lhi : rhi;
    const double x = lane < 2 * N ? 0.5 * (klo + khi) + 0.5 * (khi - klo) * sm1[ti] : 0.0;
#pragma unroll
    for (int c = 0; c < NS; ++c) w[c] = 0.0;
    bary_rows_set<N, NS>(x, mass, on, 2 * N, k, lane, rs, w);
#pragma unroll
    for (int c = 0; c < NS; ++c)
      if (lane < N) ch.w[c][idx * N + lane] = w[c];
    __syncwarp();
    if (nf) mirror_f32(f, (int)idx, N, lane, nf, panel);
    slot = up;
    up = next_up;
  }
}
