// The preconditioner's clusters and their inverses (solver.cu describes it).
#pragma once

#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "abd_common.cuh"
#include "abd_merge.cuh"

namespace abd {
namespace precond {

constexpr int BP = 3;  // most bodies of a preconditioner cluster that one CTA inverts alone

struct SolverArgs {
  const double *diag, *offdiag;
  const int *row_ptr, *adj_col, *adj_pair, *pair_active, *fixed;
  const int* ncl_dev; // clusters (formed on the device)
  const int* dstat;
  const int* resume;  // device loop: set when the iteration's solve is done (or null)
  const int *cl_ptr, *cl_body, *body_cl;
  const long long* cl_off;
  double* cl_inv;
  const int* big;     // [0, ncl_dev[1]) the clusters of 2 .. BP bodies, [n - ncl_dev[2], n) the larger
  int n;
};

// ---- preconditioner setup: assemble and invert each cluster's dense block system ----
// Clusters of one body (in a resting pile nearly every cluster: most bodies touch only the
// fixed ground) are inverted by one warp each, in registers: lane j + 12 h (j < 12, h < 2)
// holds rows 6h .. 6h + 5 of column j, and the pivot values and multipliers travel by
// shuffles, so no shared memory and no barrier.  The arithmetic of every entry is the CTA
// kernel's, in the same order: at pivot k row k becomes (j == k ? 1 : K[k][j]) times the
// reciprocal of K[k][k], then every other row i with f = K[i][k] != 0 becomes
// (j == k ? 0 : K[i][j]) - f K[k][j] (f == 0: only K[i][k] = 0).
__device__ inline void warp_inverse1(const SolverArgs& a, int c, int b, int lane) {
  const int j = lane % 12, h = lane / 12;  // lanes 24..31 (h = 2) carry values that no one reads
  double col[6];
  const double* B = a.diag + (size_t)b * 144;
#pragma unroll
  for (int t = 0; t < 6; ++t) col[t] = h < 2 ? B[(6 * h + t) * 12 + j] : 0.0;
  // The pivot loop stays rolled (the code stays small); the rows are unrolled so that they
  // live in registers, and the updates are branch-free so that the rows' shuffles overlap.
#pragma unroll 1
  for (int k = 0; k < 12; ++k) {
    const int hk = k / 6, tk = k % 6;
    double ck = 0.0;  // this lane's entry of row k (meaningful in half hk)
#pragma unroll
    for (int t = 0; t < 6; ++t)
      if (t == tk) ck = col[t];
    const double ip = 1.0 / __shfl_sync(0xffffffffu, ck, k + 12 * hk);
    const double rk = __shfl_sync(0xffffffffu, ck, j + 12 * hk);  // K[k][j]
    const double pk = (j == k ? 1.0 : rk) * ip;                     // row k scaled
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const double f = __shfl_sync(0xffffffffu, col[t], k + 12 * h);  // K[6h + t][k]
      const double base = j == k ? 0.0 : col[t];
      const double upd = base - f * pk;
      col[t] = (h == hk && t == tk) ? pk : (f != 0.0 ? upd : base);
    }
  }
  if (h < 2) {
    double* out = a.cl_inv + a.cl_off[c];
#pragma unroll
    for (int t = 0; t < 6; ++t) out[12 * j + 6 * h + t] = col[t];
  }
}

// Clusters of two bodies or more: one CTA each up to BP bodies, above that a thread-block cluster
// of four CTAs; the system's columns are dealt to the CTAs a body (12 columns, a panel) at a time,
// in shared memory.
//
// The arithmetic is the oracle's in-place Gauss-Jordan inverse (SPD: no pivoting): at pivot k, row
// k is scaled by 1 / K[k][k] (its diagonal becoming that reciprocal), then every other row i with
// f = K[i][k] != 0 becomes (j == k ? 0 : K[i][j]) - f K[k][j] (f == 0: only K[i][k] = 0).  A column
// needs from the others only the multipliers f and the reciprocals, so the pivots go a panel at a
// time, every entry seeing its operations in the same order:
//   factor: the panel's CTA takes its 12 columns through its 12 pivots, a thread per row with the
//     row's 12 entries in registers, and keeps the multipliers F [12][D] and the reciprocals;
//   apply: every CTA takes them (from that CTA's shared memory) through its other columns: first
//     the panel's 12 rows of a column, a thread per column, which gives the scaled pivot entries
//     P [12]; then all other rows, K[i][j] - f_0 P_0 - ... - f_11 P_11 in order.
// The CTA of the next panel brings that panel up to date and factors it before the rest of its
// columns.  One cluster barrier a panel.
//
// What bounds it: the chain of 12 s pivots (a divide, a broadcast and a barrier each, 0.13 us) and
// FP64 throughput (a 12-body system is 6 MFLOP, 47 us on one SM).  One CTA per cluster with a
// barrier and a pass over the whole system per pivot took 160 us for 12 bodies and 19 us for two;
// this took 96 us for a pass over clusters of up to 8 bodies that it made in 146.
constexpr int BC = 4;                          // CTAs of a cluster
static_assert(BP * BC >= kMaxCluster, "panels per CTA");
constexpr int kMaxD = 12 * kMaxCluster;
struct BigShared {
  double K[BP * 12 * kMaxD];  // the CTA's columns: entry (i, j) of its local column j at [j D + i]
  double F[12 * kMaxD];       // its last factored panel's multipliers: f_ik at [12-pivot k][row i]
  double ip[12];              // and reciprocals
  double R[12 * 24];          // the applied panel's multipliers of its own 12 rows, twice side by side
  double rip[12];
  double P[BP * 12][12];      // scaled pivot entries per local column
  double row[2][12];          // factor: the scaled pivot row, two in turn
  int member[kMaxCluster];
  int nblk;
  int2 blk[BP * kMaxCluster];  // coupling blocks: (row body, local panel) and the block's index
  int bid[BP * kMaxCluster];
};

// the panel's 12 pivots on the CTA's local panel lp (its pivots are rows 12 q ..)
static __device__ __noinline__ void big_factor(BigShared& S, int D, int q, int lp) {
  const int i = (int)threadIdx.x, k0 = 12 * q;
  double r[12];  // row i: column (k + t) % 12 of the panel at place t before pivot k
  if (i < D) {
#pragma unroll
    for (int j = 0; j < 12; ++j) r[j] = S.K[(12 * lp + j) * D + i];
  }
  auto publish = [&](int k) {  // row i is the pivot row: its scaled entries, from column k on
    const double ip = 1.0 / r[0];
    S.ip[k] = ip;
    S.row[k & 1][0] = 1.0 * ip;
#pragma unroll
    for (int t = 1; t < 12; ++t) S.row[k & 1][t] = r[t] * ip;
  };
  if (i == k0) publish(0);
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < 12; ++k) {
    if (i < D) {
      const double* P = S.row[k & 1];
      double last;
      if (i == k0 + k) {
        last = P[0];
#pragma unroll
        for (int t = 1; t < 12; ++t) r[t] = P[t];
        S.F[k * D + i] = 0.0;
      } else {
        const double f = r[0];
        S.F[k * D + i] = f;
        last = f != 0.0 ? 0.0 - f * P[0] : 0.0;
#pragma unroll
        for (int t = 1; t < 12; ++t) {
          const double u = r[t] - f * P[t];
          r[t] = f != 0.0 ? u : r[t];
        }
      }
#pragma unroll
      for (int t = 0; t < 11; ++t) r[t] = r[t + 1];
      r[11] = last;
      if (k < 11 && i == k0 + k + 1) publish(k + 1);
    }
    __syncthreads();
  }
  if (i < D) {
#pragma unroll
    for (int j = 0; j < 12; ++j) S.K[(12 * lp + j) * D + i] = r[j];
  }
  __syncthreads();
}

// the applied panel's multipliers f [12] of the thread's row through local columns [j0, j1), each
// thread group taking every G-th, three at a time (an entry is a chain of 12 multiply-subtracts)
__device__ inline void big_apply(BigShared& S, int D, int i, int g, int G, const double f[12], int j0, int j1) {
  for (int j = j0 + g; j < j1; j += 3 * G) {
    double x[3];
    int c[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      c[m] = j + m * G < j1 ? j + m * G : j;
      x[m] = S.K[c[m] * D + i];
    }
#pragma unroll
    for (int k = 0; k < 12; ++k)
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double u = x[m] - f[k] * S.P[c[m]][k];
        x[m] = f[k] != 0.0 ? u : x[m];
      }
#pragma unroll
    for (int m = 0; m < 3; ++m)
      if (m == 0 || c[m] != j) S.K[c[m] * D + i] = x[m];
  }
}

// Cluster c by nc CTAs of BT threads, this one the rank-th (nc 1: the CTA alone, at most BP bodies)
template <int BT>
__device__ void big_inverse(const SolverArgs& a, BigShared& S, int c, int rank, int nc) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int base = a.cl_ptr[c], s = a.cl_ptr[c + 1] - base, D = 12 * s;
  const int np = rank < s ? (s - rank + nc - 1) / nc : 0;  // panels rank, rank + nc, ...
  if (tid < s) S.member[tid] = a.cl_body[base + tid];
  if (tid == 0) S.nblk = 0;
  for (int e = tid; e < 12 * np * D; e += BT) S.K[e] = 0.0;
  __syncthreads();
  // the coupling blocks of the CTA's column bodies: a warp per panel finds the active pairs whose
  // other body is a member
  for (int lp = warp; lp < np; lp += BT / 32) {
    const int b = S.member[rank + nc * lp];
    const int k1 = a.fixed[b] ? a.row_ptr[b] : a.row_ptr[b + 1];
    for (int k = a.row_ptr[b] + lane; k < k1; k += 32) {
      const int J = a.adj_col[k], pr = a.adj_pair[k];
      if (a.body_cl[J] != c || a.fixed[J] || a.pair_active[pr] <= 0) continue;
      int li = 0;
      while (S.member[li] != J) ++li;
      const int e = atomicAdd(&S.nblk, 1);
      S.blk[e] = make_int2(li, lp);
      S.bid[e] = 2 * pr + (J < b ? 0 : 1);  // the block with J's rows
    }
  }
  for (int e = tid; e < np * 144; e += BT) {
    const int lp = e / 144, q = rank + nc * lp, r = e % 12, col = (e / 12) % 12;
    S.K[(12 * lp + col) * D + 12 * q + r] = a.diag[(size_t)S.member[q] * 144 + 12 * r + col];
  }
  __syncthreads();
  for (int e = tid; e < S.nblk * 144; e += BT) {
    const int2 m = S.blk[e / 144];
    const int r = (e / 12) % 12, col = e % 12;
    S.K[(12 * m.y + col) * D + 12 * m.x + r] = a.offdiag[(size_t)S.bid[e / 144] * 144 + 12 * r + col];
  }
  __syncthreads();
  const int i = tid % D, g = tid / D, G = BT / D;
  if (rank == 0) big_factor(S, D, 0, 0);
  for (int q = 0; q < s; ++q) {
    if (nc > 1) cl.sync();  // panel q is factored
    else __syncthreads();
    const int owner = q % nc, own = rank == owner ? q / nc : -1;  // (its own columns are done)
    const double* F = nc > 1 ? cl.map_shared_rank(S.F, owner) : S.F;
    const double* ip = nc > 1 ? cl.map_shared_rank(S.ip, owner) : S.ip;
    double f[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) f[k] = F[k * D + i];
    for (int e = tid; e < 144; e += BT) {
      const double v = F[(e / 12) * D + 12 * q + e % 12];
      S.R[(e / 12) * 24 + e % 12] = v;
      S.R[(e / 12) * 24 + 12 + e % 12] = v;
    }
    if (tid < 12) S.rip[tid] = ip[tid];
    __syncthreads();
    // the panel's rows of every column: row (k + t) % 12 at place t before pivot k
    for (int j = tid; j < 12 * np; j += BT) {
      if (j / 12 == own) continue;
      double u[12];
      double* col = &S.K[j * D + 12 * q];
#pragma unroll
      for (int k = 0; k < 12; ++k) u[k] = col[k];
#pragma unroll 1
      for (int k = 0; k < 12; ++k) {
        const double pk = u[0] * S.rip[k];
        S.P[j][k] = pk;
        const double* m = &S.R[k * 24 + k];
#pragma unroll
        for (int t = 1; t < 12; ++t) {
          const double v = u[t] - m[t] * pk;
          u[t - 1] = m[t] != 0.0 ? v : u[t];
        }
        u[11] = pk;
      }
#pragma unroll
      for (int k = 0; k < 12; ++k) col[k] = u[k];
    }
    __syncthreads();
    // the other rows; the next panel's columns first, and its factors
    const bool row = g < G && (i < 12 * q || i >= 12 * q + 12);
    const int next = q + 1 < s && (q + 1) % nc == rank ? (q + 1) / nc : -1;
    if (next >= 0) {
      if (row) big_apply(S, D, i, g, G, f, 12 * next, 12 * next + 12);
      __syncthreads();
      big_factor(S, D, q + 1, next);
    }
    for (int lp = 0; lp < np; ++lp)
      if (lp != next && lp != own && row) big_apply(S, D, i, g, G, f, 12 * lp, 12 * lp + 12);
    __syncthreads();
  }
  double* out = a.cl_inv + a.cl_off[c];  // (transposed: column j contiguous)
  for (int e = tid; e < 12 * np * D; e += BT) {
    const int j = e / D, q = rank + nc * (j / 12);
    out[(size_t)(12 * q + j % 12) * D + e % D] = S.K[e];
  }
  if (nc > 1) cl.sync();  // (another CTA may still read this one's factors)
  else __syncthreads();
}

// Exclusive prefix sum over the threads of a CTA (one value per thread); *total gets the
// sum.  Every thread must call it.
__device__ inline long long block_scan_excl(long long v, long long* total) {
  __shared__ long long wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    long long w = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;  // inclusive prefix of the warp totals
  }
  __syncthreads();
  const long long before = (warp > 0 ? wsum[warp - 1] : 0) + x - v;
  *total = wsum[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before;
}

// a CTA of KT threads, for merge_rounds
template <int KT>
struct CtaTeam {
  __device__ __forceinline__ int id() const { return (int)threadIdx.x; }
  __device__ __forceinline__ int size() const { return KT; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ bool any(bool p) const { return __syncthreads_or(p) != 0; }
  __device__ __forceinline__ void best(unsigned long long* p, unsigned long long key) const { atomicMax(p, key); }
};

// The preconditioner's clusters, formed on the device by one CTA from the active-pair list
// the pair assembly appended (pair, I, J, FP32 weight bits; in any order).  Rounds: every
// cluster picks its strongest admissible pair to another cluster (weight, then the lower pair
// index, as one 64-bit key; admissible: both clusters together within cap bodies) and two
// clusters that pick the same pair merge under the lower label.  Every decision of a round
// uses the labels and sizes from its start, so the result does not depend on the order in
// which threads see the pairs.  Then the tables: clusters ordered by their first body (the
// label), members in increasing order, the offsets of the dense inverses. 
// By the CTA's KT threads.
template <int KT>
__device__ void make_clusters(int n, int cap, const int4* act, int cap_act, const int* dstat, const ClusterTables& t,
                              const ClusterWork& w) {
  const int tid = threadIdx.x;
  const int m = min(dstat[DS_NACTP], cap_act);
  for (int b = tid; b < n; b += KT) {
    w.label[b] = b;
    w.size[b] = 1;
  }
  __shared__ int nsolo, nmulti;
  if (tid == 0) nsolo = nmulti = 0;
  __syncthreads();
  merge_rounds(CtaTeam<KT>{}, n, cap, 4 * kMaxCluster, act, m, w);
  // cluster index of every label, cluster offsets and inverse offsets, in label order
  long long ccarry = 0, pcarry = 0, ocarry = 0;
  for (int b0 = 0; b0 < n; b0 += KT) {
    const int b = b0 + tid;
    const bool root = b < n && w.label[b] == b;
    const int sz = root ? w.size[b] : 0;
    long long tc, tp, to_;
    const long long c = block_scan_excl(root ? 1 : 0, &tc) + ccarry;
    const long long p = block_scan_excl(sz, &tp) + pcarry;
    const long long o = block_scan_excl(root ? 144LL * sz * sz : 0, &to_) + ocarry;
    if (root) {
      w.cidx[b] = (int)c;
      t.cl_ptr[c] = (int)p;
      t.cl_off[c] = o;
      w.fill[c] = 0;
    }
    ccarry += tc;
    pcarry += tp;
    ocarry += to_;
  }
  const int ncl = (int)ccarry;
  __syncthreads();
  // the clusters of 2 .. BP bodies from the front, the larger ones from the back, in any order
  for (int b = tid; b < n; b += KT)
    if (w.label[b] == b && w.size[b] > 1)
      w.to[w.size[b] <= BP ? atomicAdd(&nsolo, 1) : n - 1 - atomicAdd(&nmulti, 1)] = w.cidx[b];
  __syncthreads();
  if (tid == 0) {
    *t.ncl = ncl;
    t.ncl[1] = nsolo;
    t.ncl[2] = nmulti;
    t.cl_ptr[ncl] = n;
    t.cl_off[ncl] = ocarry;
  }
  __syncthreads();
  for (int b = tid; b < n; b += KT) {
    const int c = w.cidx[w.label[b]];
    t.body_cl[b] = c;
    t.cl_body[t.cl_ptr[c] + atomicAdd(&w.fill[c], 1)] = b;
  }
  __syncthreads();
  for (int c = tid; c < ncl; c += KT) {  // members in increasing order (at most cap of them)
    int* mb = t.cl_body + t.cl_ptr[c];
    const int k1 = t.cl_ptr[c + 1] - t.cl_ptr[c];
    for (int i = 1; i < k1; ++i) {
      const int v = mb[i];
      int j = i - 1;
      for (; j >= 0 && mb[j] > v; --j) mb[j + 1] = mb[j];
      mb[j + 1] = v;
    }
  }
}

}  // namespace precond

precond::SolverArgs solver_args(Sim& s);   // solver.cu
int cluster_cap(const Sim& s);             // most bodies of a preconditioner cluster

}  // namespace abd
