// The Krylov solve of the Newton system (krylov.cu describes it): one thread-block cluster, its
// kernel's body.
#pragma once

#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "abd_common.cuh"
#include "abd_warpsum.cuh"

namespace abd {
namespace krylov {

namespace cg = cooperative_groups;

constexpr int KC = 16;         // most CTAs of the cluster
constexpr int kMaxDots = 4;    // dot products of one reduction
// dstat slots of the solve's outcome
enum { DS_R_DONE = 10, DS_S_DONE = 11 };

// a body position of a CTA's rows: its place in its preconditioner cluster and its neighbours
struct PosInfo {
  int body, lbase, D, ncnt;  // body; first local row and rows of its cluster; active neighbours
  long long koff, noff;      // its cluster's inverse; its neighbour list
};

struct KrylovArgs {
  int n, maxit;
  const double *diag, *offdiag, *g;
  const int *row_ptr, *adj_col, *adj_pair, *pair_active, *fixed;
  int2* nb;                 // [adjacency capacity] active neighbours per row: (body, 2 pair + side)
  const int *cl_ptr, *cl_body, *body_cl;
  const long long* cl_off;
  const double* cl_inv;     // the clusters' inverses, transposed
  double tol2;
  double* x;                // in: the warm start, out: the solution
  double *pub0, *pub1, *pub2;  // published vectors (read by other rows): PCG p, p, z; BiCGSTAB y, z
  int rows_max, pos_max;    // shared memory's rows and positions
  int* dstat;
  Mailbox* tally;           // device loop: the outcome goes to the step's counters, with
                            // x.g and g.g in its dots (else null)
};

// row vectors in shared memory: PCG x, r, p, Ap; BiCGSTAB x, r (then s), p, rh, v, t

struct RedShared {  // of two reductions in turn
  int sum[2][kMaxDots][kDSlots];      // the CTA's digits (abd_warpsum.cuh); zero between reductions
  int cta[2][kMaxDots][KC][kDSlots];  // every CTA's digits, pushed by it
  double out[2][kMaxDots];
};

// The solve's shared state in each thread: the cluster, the row range, the reductions
struct Ctx {
  int T, tid, lane, warp, nw, rank, C;
  int nrow;       // local rows
  int turn;       // reductions done (their buffers alternate)
  RedShared* red;
};

__device__ inline void all_sync(const Ctx& c) {
  if (c.C == 1) __syncthreads();
  else cg::this_cluster().sync();
}

// x into dot product k of the next reduction
__device__ inline void add(Ctx& c, int k, double x) { ds_add(c.red->sum[c.turn & 1][k], x); }

// The exact dot products of the terms added since the last reduction, rounded.  Also a barrier of
// the whole cluster: what was written before it is visible after it.  (Not inlined, like the row
// products: a solve runs once through its code, and instructions that are fetched for a single
// use cost more than the calls.)
static __device__ __noinline__ const double* reduce(Ctx& c, int nd) {
  RedShared& R = *c.red;
  const int b = c.turn & 1;
  ++c.turn;
  __syncthreads();
  if (c.C > 1) {
    // each warp pushes the CTA's digits to one CTA of the cluster (in turn when there are more
    // CTAs than warps)
    for (int r = c.warp; r < c.C; r += c.nw)
      for (int k = 0; k < nd; ++k)
        *cg::this_cluster().map_shared_rank(&R.cta[b][k][c.rank][c.lane], r) = R.sum[b][k][c.lane];
    cg::this_cluster().sync();
  }
  for (int k = c.warp; k < nd; k += c.nw) {  // a warp per dot product
    long long v = 0;
    if (c.C == 1) {
      v = R.sum[b][k][c.lane];
    } else {
#pragma unroll
      for (int r = 0; r < KC; ++r) {
        const long long x = r < c.C ? R.cta[b][k][r][c.lane] : 0;
        v = c.lane == kDFlags ? v | x : v + x;
      }
    }
    R.sum[b][k][c.lane] = 0;  // (every warp has read it)
    const double t = ds_round(v);
    if (c.lane == 0) R.out[b][k] = t;
  }
  __syncthreads();
  return R.out[b];
}

// A value of the system: through the read-only path (NC) unless the kernel that runs the solve also
// wrote it
template <bool NC, class T>
__device__ inline T fixed_value(const T* p) {
  return NC ? __ldg(p) : *p;
}

// 12 values at p (16-byte aligned: the library's own buffers); FIXED: of the system, else they come
// from L2, where the other CTAs' published values are
template <bool FIXED, bool NC>
__device__ inline void load12(const double* p, double out[12]) {
  const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double2 v = FIXED ? fixed_value<NC>(q + k) : __ldcg(q + k);
    out[2 * k] = v.x;
    out[2 * k + 1] = v.y;
  }
}

// row i of A u for the body position P, u = v or (z given) z + beta v, entry for entry
template <bool NC>
static __device__ __noinline__ double row_product(const KrylovArgs& a, const PosInfo& P, int i, const double* v,
                                                  const double* z, double beta) {
  double lo = 0.0, hi = 0.0;
  const double* row = a.diag + (size_t)P.body * 144 + 12 * i;
  int J = P.body;
  for (int e = 0;; ++e) {
    double B[12], u[12];
    load12<true, NC>(row, B);
    load12<false, NC>(v + (size_t)J * 12, u);
    if (z) {
      double w[12];
      load12<false, NC>(z + (size_t)J * 12, w);
#pragma unroll
      for (int k = 0; k < 12; ++k) u[k] = w[k] + beta * u[k];
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      lo += B[k] * u[k];
      hi += B[6 + k] * u[6 + k];
    }
    if (e == P.ncnt) return lo + hi;
    const int2 q = a.nb[P.noff + e];
    J = q.x;
    row = a.offdiag + (size_t)q.y * 144 + 12 * i;
  }
}

// row l of M^-1 v (and of M^-1 w): the transposed inverse's column, v and w local rows
template <bool NC>
static __device__ __noinline__ double2 apply_rows(const KrylovArgs& a, const PosInfo& P, int l, const double* v,
                                           const double* w) {
  const int D = P.D;
  const double* K = a.cl_inv + P.koff + (l - P.lbase);
  v += P.lbase;
  w += P.lbase;
  double2 acc = make_double2(0.0, 0.0);
  for (int j0 = 0; j0 < D; j0 += 12) {
    double k[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) k[j] = fixed_value<NC>(K + (size_t)(j0 + j) * D);
#pragma unroll
    for (int j = 0; j < 12; ++j) acc.x += k[j] * v[j0 + j];
    if (w != v) {
#pragma unroll
      for (int j = 0; j < 12; ++j) acc.y += k[j] * w[j0 + j];
    }
  }
  return acc;
}
template <bool NC>
__device__ inline double apply_row(const KrylovArgs& a, const PosInfo& P, int l, const double* v) {
  return apply_rows<NC>(a, P, l, v, v).x;
}

// After a block of rows, when more follow: the counters' carries to the counters above, which
// makes room for the next block's terms
constexpr int kRowBlock = 2048;
static_assert(kRowBlock + 64 < kDTerms, "a block's terms fit the counters");
static __device__ __noinline__ void fold(Ctx& c) {
  __syncthreads();
  for (int k = c.warp; k < kMaxDots; k += c.nw) ds_fold(c.red->sum[c.turn & 1][k]);
  __syncthreads();
}
__device__ inline int next_block(Ctx& c, int b) {
  if (b + kRowBlock < c.nrow) fold(c);
  return b + kRowBlock;
}

// rows of the CTA, a thread each, in blocks
#define FOR_ROWS(l)                                                  \
  for (int l##b = 0; l##b < c.nrow; l##b = next_block(c, l##b))      \
    for (int l = l##b + c.tid; l < min(c.nrow, l##b + kRowBlock); l += c.T)

// The solve by a cluster of C CTAs, this one the rank-th.  dyn: the CTA's dynamic shared memory;
// red: in shared memory.  NC: the kernel is the solve alone; then no barrier has told yet that every
// CTA of the cluster runs, which the first store to another CTA's shared memory needs: each
// arrives here and waits just before its first dot products, when the others have long arrived.
// (Without NC the caller has passed a cluster barrier.)
template <bool PCG, bool NC>
__device__ __forceinline__ void solve(const KrylovArgs& a, double* dyn, RedShared& red, int C, int rank) {
  __shared__ int sh_p[2];
  if (NC && C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  Ctx c;
  c.T = (int)blockDim.x;
  c.tid = (int)threadIdx.x;
  c.lane = c.tid & 31;
  c.warp = c.tid >> 5;
  c.nw = c.T >> 5;
  c.C = C;
  c.rank = rank;
  c.turn = 0;
  c.red = &red;
  for (int i = c.tid; i < 2 * kMaxDots * kDSlots; i += c.T) (&red.sum[0][0][0])[i] = 0;
  const int n = a.n;
  // The CTA's body positions (bodies in cluster order): an equal share, moved up to whole
  // preconditioner clusters, whose rows need each other's vector entries
  if (c.tid < 2) {
    const long long t = (long long)(c.rank + c.tid) * n / c.C;
    int p = n;
    if (t < n) {
      const int k = a.body_cl[a.cl_body[t]];
      p = a.cl_ptr[k] == (int)t ? (int)t : a.cl_ptr[k + 1];
    }
    sh_p[c.tid] = p;
  }
  __syncthreads();
  const int P0 = sh_p[0], np = sh_p[1] - P0;
  c.nrow = 12 * np;
  auto vec = [&](int k) { return dyn + (size_t)k * a.rows_max; };
  double *const S_x = vec(0), *const S_r = vec(1), *const S_p = vec(2), *const S_a = vec(3);
  double *const S_v = PCG ? nullptr : vec(4), *const S_t = PCG ? nullptr : vec(5);
  PosInfo* const pos = reinterpret_cast<PosInfo*>(dyn + (size_t)(PCG ? 4 : 6) * a.rows_max);
  // positions (a thread each)
  for (int q = c.tid; q < np; q += c.T) {
    const int b = a.cl_body[P0 + q], k = a.body_cl[b], base = a.cl_ptr[k];
    PosInfo P;
    P.body = b;
    P.lbase = 12 * (base - P0);
    P.D = 12 * (a.cl_ptr[k + 1] - base);
    P.noff = a.row_ptr[b];
    P.ncnt = a.fixed[b] ? 0 : a.row_ptr[b + 1] - (int)P.noff;
    P.koff = a.cl_off[k];
    pos[q] = P;
  }
  __syncthreads();
  // each body's active neighbours in increasing order (eight lanes a body)
  for (int q0 = 4 * c.warp; q0 < np; q0 += 4 * c.nw) {
    const int q = q0 + c.lane / 8, sub = c.lane % 8;
    const int deg = q < np ? pos[q].ncnt : 0, r0 = q < np ? (int)pos[q].noff : 0, b = q < np ? pos[q].body : 0;
    int cnt = 0;
    for (int k0 = 0; __any_sync(0xffffffffu, k0 < deg); k0 += 8) {
      const int k = r0 + k0 + sub;
      bool on = false;
      int2 e = make_int2(0, 0);
      if (k0 + sub < deg) {
        const int pr = a.adj_pair[k], J = a.adj_col[k];
        on = a.pair_active[pr] > 0 && !a.fixed[J];
        e = make_int2(J, 2 * pr + (b < J ? 0 : 1));
      }
      const unsigned m = (__ballot_sync(0xffffffffu, on) >> (c.lane & 24)) & 0xffu;
      if (on) a.nb[r0 + cnt + __popc(m & ((1u << sub) - 1u))] = e;
      cnt += __popc(m);
    }
    __syncwarp();
    if (sub == 0 && q < np) pos[q].ncnt = cnt;
  }
  __syncthreads();
  auto gi = [&](int l) { return (size_t)pos[l / 12].body * 12 + l % 12; };  // global entry of local row l

  // ---- set-up: r = b - A x, M^-1 r, M^-1 b and their dot products ----
  FOR_ROWS(l) {
    const size_t i = gi(l);
    const double bi = a.g[i];
    S_x[l] = a.x[i];
    S_r[l] = bi - row_product<NC>(a, pos[l / 12], l % 12, a.x, nullptr, 0.0);
    S_a[l] = bi;
  }
  __syncthreads();
  if (NC && C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  FOR_ROWS(l) {
    const double2 m = apply_rows<NC>(a, pos[l / 12], l, S_r, S_a);
    add(c, 0, S_r[l] * m.x);
    add(c, 1, S_a[l] * m.y);
    if (a.tally) add(c, 2, S_a[l] * S_a[l]);
    if (PCG) {
      S_p[l] = m.x;
      a.pub0[gi(l)] = m.x;
    } else {
      add(c, 3, S_r[l] * S_r[l]);
    }
  }
  const double* o = reduce(c, PCG ? 3 : 4);
  const double bz = o[1], gg = o[2];
  double rz = o[0];
  const double thr2 = a.tol2 * bz;
  int r_done = 0, s_done = 0, iters = 0;
  if (!(bz > 0.0)) {  // the solution is 0
    r_done = 1;
    FOR_ROWS(l) S_x[l] = 0.0;
  } else if constexpr (PCG) {
    double *po = a.pub0, *pn = a.pub1, beta = 0.0;
    for (int it = 1; it <= a.maxit; ++it) {
      if (!(rz > thr2)) {
        r_done = it;
        iters = it - 1;
        break;
      }
      // p = z + beta p and Ap with p.Ap; a neighbour's p from its z and old p
      FOR_ROWS(l) {
        const size_t i = gi(l);
        const double pi = it == 1 ? S_p[l] : __ldcg(&a.pub2[i]) + beta * S_p[l];
        const double y = row_product<NC>(a, pos[l / 12], l % 12, po, it > 1 ? a.pub2 : nullptr, beta);
        S_p[l] = pi;
        if (it > 1) pn[i] = pi;
        S_a[l] = y;
        add(c, 0, pi * y);
      }
      const double pap = *reduce(c, 1);
      if (it > 1) {
        double* const t = po;
        po = pn;
        pn = t;
      }
      if (!(pap > 0.0)) {  // no positive curvature
        r_done = it;
        iters = it - 1;
        break;
      }
      const double alpha = rz / pap;
      FOR_ROWS(l) {
        S_x[l] += alpha * S_p[l];
        S_r[l] -= alpha * S_a[l];
      }
      __syncthreads();
      FOR_ROWS(l) {
        const double z = apply_row<NC>(a, pos[l / 12], l, S_r);
        a.pub2[gi(l)] = z;
        add(c, 0, S_r[l] * z);
      }
      const double rzn = *reduce(c, 1);
      iters = it;
      if (it + 1 > a.maxit) break;
      if (!(rzn > thr2)) {
        r_done = it + 1;
        break;
      }
      beta = rzn / rz;
      rz = rzn;
    }
  } else {
    // right-preconditioned BiCGSTAB; rh keeps its place in S_a, s takes r's
    double *const S_rh = S_a, *const S_s = S_r;
    double rho = o[3], rho_old = 1.0, alpha = 1.0, omega = 1.0;
    FOR_ROWS(l) S_rh[l] = S_r[l];
    for (int it = 1; it <= a.maxit; ++it) {
      if (!(rz > thr2) || rho == 0.0 || !isfinite(rho)) {
        r_done = it;
        iters = it - 1;
        break;
      }
      const double beta = (rho / rho_old) * (alpha / omega);
      FOR_ROWS(l) S_p[l] = it == 1 ? S_r[l] : S_r[l] + beta * (S_p[l] - omega * S_v[l]);
      __syncthreads();
      FOR_ROWS(l) a.pub0[gi(l)] = apply_row<NC>(a, pos[l / 12], l, S_p);
      all_sync(c);
      FOR_ROWS(l) {
        const double v = row_product<NC>(a, pos[l / 12], l % 12, a.pub0, nullptr, 0.0);
        S_v[l] = v;
        add(c, 0, S_rh[l] * v);
      }
      alpha = rho / *reduce(c, 1);
      FOR_ROWS(l) S_s[l] = S_r[l] - alpha * S_v[l];
      __syncthreads();
      FOR_ROWS(l) {
        const double z = apply_row<NC>(a, pos[l / 12], l, S_s);
        a.pub1[gi(l)] = z;
        add(c, 0, S_s[l] * z);
      }
      if (!(*reduce(c, 1) > thr2)) {
        FOR_ROWS(l) S_x[l] += alpha * __ldcg(&a.pub0[gi(l)]);
        s_done = it;
        iters = it;
        break;
      }
      FOR_ROWS(l) {
        const double t = row_product<NC>(a, pos[l / 12], l % 12, a.pub1, nullptr, 0.0);
        S_t[l] = t;
        add(c, 0, S_s[l] * t);
        add(c, 1, t * t);
      }
      const double* ts = reduce(c, 2);
      omega = ts[0] / ts[1];
      FOR_ROWS(l) {
        const size_t i = gi(l);
        S_x[l] += alpha * __ldcg(&a.pub0[i]) + omega * __ldcg(&a.pub1[i]);
        S_r[l] = S_s[l] - omega * S_t[l];
      }
      __syncthreads();
      FOR_ROWS(l) {
        add(c, 0, S_r[l] * apply_row<NC>(a, pos[l / 12], l, S_r));
        add(c, 1, S_rh[l] * S_r[l]);
      }
      const double* rr = reduce(c, 2);
      iters = it;
      rz = rr[0];
      rho_old = rho;
      rho = rr[1];
      if (it + 1 > a.maxit) break;
      if (!(rz > thr2) || rho == 0.0 || !isfinite(rho)) {
        r_done = it + 1;
        break;
      }
    }
  }
  // the solution, and x.g for the device loop's line search
  FOR_ROWS(l) {
    const size_t i = gi(l);
    const double xi = S_x[l];
    a.x[i] = xi;
    if (a.tally) add(c, 0, xi * a.g[i]);
  }
  double xg = 0.0;
  if (a.tally) xg = *reduce(c, 1);
  if (c.rank == 0 && c.tid == 0) {
    a.dstat[DS_R_DONE] = r_done;
    a.dstat[DS_S_DONE] = s_done;
    a.dstat[DS_SOLVER_ITERS] = iters;
    if (a.tally) {
      a.tally->dots[0] = xg;
      a.tally->dots[1] = gg;
      a.tally->step.lin += iters;
      if (!(r_done || s_done)) atomicOr(&a.dstat[DS_STATUS], ST_SOLVER_NOCONV);
    }
  }
}

#undef FOR_ROWS

}  // namespace krylov

// krylov.cu
krylov::KrylovArgs krylov_args(Sim& s, double* x, bool tally, int C, size_t* smem);

}  // namespace abd
