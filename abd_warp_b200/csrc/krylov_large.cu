// The Krylov solve of large systems: short kernels over the whole GPU inside a WHILE node of the graph.
//
// krylov.cu's kernel holds a solve in one thread-block cluster, whose 16 SMs bound it once the system
// is large.  Here an iteration is three (PCG) or six (BiCGSTAB) kernels, a warp per block row (24 lanes
// = 12 rows x 2 half-rows) or per preconditioner cluster; the kernel that completes an iteration's
// last dot product also ends it: it advances the iteration counter, makes the convergence test
// that the next iteration would make, and sets the loop's condition.  The arithmetic is krylov.cu's,
// entry for entry, and dot products are exact (per-CTA partials summed in fixed point), so both give
// the same bits.
// (krylov_is_large, krylov.cu, says which systems come here, with the figures of both.)
#include <cuda_runtime.h>

#include <algorithm>

#include "abd_common.cuh"
#include "abd_graph.cuh"
#include "abd_krylov.cuh"
#include "abd_precond.cuh"

namespace abd {

namespace {

using krylov::DS_R_DONE;
using krylov::DS_S_DONE;

constexpr int WPB = 8;          // warps (body rows) per CTA of the row kernels
constexpr int AT = 128;         // threads of the cluster kernels

// slots of Sim::partials
enum { SL_RZ0 = 0, SL_RZ1 = 1, SL_PAP = 2, SL_BZ = 3, SL_RHR = 4, SL_RHV = 5, SL_SZ = 6, SL_TS = 7, SL_TT = 8 };
// Sim::kry_scal layout: scalars, then the totals
enum { SC_RHO0 = 0, SC_RHO1 = 1, SC_ALPHA = 2, SC_OMEGA = 3, SC_THR2 = 4 };
// Sim::kry_int: the current iteration (1 at the first), the loop body's runs (a watchdog)
enum { KI_IT = 0, KI_RUNS = 1 };

struct LargeArgs {
  int n;
  const double *diag, *offdiag;
  const int *row_ptr, *adj_col, *adj_pair, *pair_active, *fixed;
  const int2* ij;
  const int* ncl_dev;
  int maxit;
  const int *cl_ptr, *cl_body;
  const long long* cl_off;
  const double* cl_inv;  // the clusters' inverses, transposed
  XSum* part;            // [kRedSlots][kRedBlocks] exact per-CTA partials
  int* red_count;        // [kRedSlots] CTAs that delivered their partial
  double* scal;
  int* ki;
  int* dstat;
  Mailbox* tally;        // device loop: the solve's outcome goes to the step's counters (else null)
  cudaGraphConditionalHandle loop;  // the iteration loop's WHILE node
};

constexpr int SC_RED = 16;  // scal[SC_RED + slot]: the rounded total of reduction `slot`

// scalars produced by the previous kernel's reductions
__device__ inline void cta_scalars(const LargeArgs& a, const int* slots, int ns, double* out) {
  for (int k = 0; k < ns; ++k) out[k] = a.scal[SC_RED + slots[k]];
}

// The CTA's exact partial of a dot product into part[slot] (every thread passes its accumulator)
__device__ inline void cta_partial(const LargeArgs& a, XSum& x, int slot, XSum* sh) {
  xs_block_sum(x, sh);
  if (threadIdx.x == 0) a.part[slot * kRedBlocks + blockIdx.x] = x;
}

// After a CTA's partials: true in the last CTA to deliver (the launch's single counter cslot,
// reset here for the next launch), which then sees every CTA's partials
__device__ inline bool cta_last(const LargeArgs& a, int cslot) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&a.red_count[cslot], 1) == (int)gridDim.x - 1;
    if (last) a.red_count[cslot] = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// In the last CTA: the sum of every CTA's partial of `slot`, rounded into scal[SC_RED + slot]
__device__ inline void total_of(const LargeArgs& a, int slot, XSum* sh) {
  XSum t;
  xs_zero(t);
  const XSum* P = a.part + slot * kRedBlocks;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
    const long long* q = reinterpret_cast<const long long*>(P + i);
#pragma unroll
    for (int j = 0; j < kXD; ++j) t.d[j] += __ldcg(q + j);
    t.flags |= __ldcg(q + kXD);
  }
  xs_block_sum(t, sh);
  if (threadIdx.x == 0) a.scal[SC_RED + slot] = xs_round(t);
}

// Exact per-CTA partials of up to two dot products (every thread passes its accumulators);
// the last CTA to deliver sums the partials of all CTAs and stores the rounded totals in
// scal[SC_RED + slot] (a single counter per launch: slot0 if >= 0, else slot1).
// Returns true in the last CTA, whose thread 0 wrote the totals.
__device__ inline bool cta_partials(const LargeArgs& a, XSum& x0, XSum& x1, int slot0, int slot1) {
  __shared__ XSum sh[8];
  if (slot0 >= 0) cta_partial(a, x0, slot0, sh);
  if (slot1 >= 0) cta_partial(a, x1, slot1, sh);
  if (!cta_last(a, slot0 >= 0 ? slot0 : slot1)) return false;
  if (slot0 >= 0) total_of(a, slot0, sh);
  if (slot1 >= 0) total_of(a, slot1, sh);
  return true;
}

// y_b (lanes 0..11 hold row lane) = (A x)_b for block row b
__device__ inline double row_product(const LargeArgs& a, int b, const double* x) {
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  if (lane < 24) {
    const int r = lane % 12, h = lane / 12;
    const double* B = a.diag + (size_t)b * 144 + r * 12 + 6 * h;
    const double* xb = x + (size_t)b * 12 + 6 * h;
#pragma unroll
    for (int c = 0; c < 6; ++c) acc += B[c] * xb[c];
    if (!a.fixed[b]) {
      for (int k = a.row_ptr[b]; k < a.row_ptr[b + 1]; ++k) {
        const int pr = a.adj_pair[k];
        if (a.pair_active[pr] <= 0) continue;
        const int J = a.adj_col[k];
        if (a.fixed[J]) continue;
        const int side = a.ij[pr].x == b ? 0 : 1;
        const double* O = a.offdiag + (size_t)pr * 288 + side * 144 + r * 12 + 6 * h;
        const double* xj = x + (size_t)J * 12 + 6 * h;
#pragma unroll
        for (int c = 0; c < 6; ++c) acc += O[c] * xj[c];
      }
    }
  }
  acc += __shfl_down_sync(0xffffffffu, acc, 12);
  return acc;  // valid on lanes 0..11
}

#define FOR_BODIES(b) for (int b = blockIdx.x * WPB + (int)(threadIdx.x >> 5); b < a.n; b += (int)gridDim.x * WPB)

__device__ inline bool solver_done(const int* dstat) {
  return ((volatile const int*)dstat)[DS_R_DONE] != 0 || ((volatile const int*)dstat)[DS_S_DONE] != 0;
}

// the current Krylov iteration (device counter, 1 at the first iteration, advanced by
// loop_end); iterations beyond the limit do nothing
__device__ inline int iteration(const LargeArgs& a) { return a.ki[KI_IT]; }

// The outcome of a finished solve into the device loop's step counters (a.tally): its
// iterations, and the non-convergence bit when it stopped at cg_max_iter (one thread)
__device__ inline void tally_solve(const LargeArgs& a) {
  if (!a.tally) return;
  a.tally->step.lin += a.dstat[DS_SOLVER_ITERS];
  if (!(a.dstat[DS_R_DONE] || a.dstat[DS_S_DONE])) atomicOr(&a.dstat[DS_STATUS], ST_SOLVER_NOCONV);
}

// The end of a loop iteration (one thread, in the iteration's last kernel once its last
// reduction is final): advances the iteration counter, makes the convergence test of the next
// iteration's first kernel (PCG: r.z against the threshold; BiCGSTAB: r.M^-1 r and
// rho = rh.r), records a stop as that kernel would, and sets the WHILE node's condition.  The
// loop ends at convergence or after maxit iterations (and the solve's outcome is tallied); a
// body that ran more than maxit times also ends it.
__device__ inline void loop_end(const LargeArgs& a, int pcg) {
  const int it = a.ki[KI_IT];
  bool stop = solver_done(a.dstat) || it + 1 > a.maxit || a.ki[KI_RUNS] > a.maxit;
  if (!stop) {
    const double thr2 = a.scal[SC_THR2];
    if (pcg) {
      stop = !(a.scal[SC_RED + ((it & 1) ? SL_RZ1 : SL_RZ0)] > thr2);
    } else {
      const double rho = a.scal[SC_RED + SL_RHR];
      stop = !(a.scal[SC_RED + SL_RZ0] > thr2) || rho == 0.0 || !isfinite(rho);
    }
    if (stop) {
      a.dstat[DS_R_DONE] = it + 1;
      a.dstat[DS_SOLVER_ITERS] = it;
    }
  }
  a.ki[KI_IT] = it + 1;
  if (stop) tally_solve(a);
  cudaGraphSetConditional(a.loop, stop ? 0u : 1u);
}

// The first kernel of an iteration counts the loop body's runs (thread 0 of CTA 0); a body
// that runs more than maxit times ends the loop (a safeguard: loop_end ends it at maxit)
__device__ inline void count_run(const LargeArgs& a) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && ++a.ki[KI_RUNS] > a.maxit)
    cudaGraphSetConditional(a.loop, 0u);
}

// One warp per cluster: the input's entries of the cluster's body rows, in = row_in(i) for the
// entry i of a member body (lanes 0..11: the row's 12 entries; row_in may also update the
// body's own entries of other vectors), then out = M^-1 in over the cluster -- lane i
// computes rows i, i + 32, ... of the cluster's dense inverse (stored transposed) times the gathered input,
// summing over the columns in order -- with the partial in.out added to *dot (if not null);
// out null: the product only feeds the dot.
template <class RowIn>
__device__ inline void cluster_apply(const LargeArgs& a, double* out, XSum* dot, RowIn&& row_in) {
  constexpr int NWA = AT / 32;
  __shared__ double vs[NWA][12 * kMaxCluster];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ncl = *a.ncl_dev;
  for (int c = blockIdx.x * NWA + warp; c < ncl; c += gridDim.x * NWA) {
    const int base = a.cl_ptr[c], sz = a.cl_ptr[c + 1] - base, D = 12 * sz;
    if (lane < 12)
      for (int m = 0; m < sz; ++m) vs[warp][12 * m + lane] = row_in((size_t)a.cl_body[base + m] * 12 + lane);
    __syncwarp();
    const double* Kc = a.cl_inv + a.cl_off[c];
    for (int i = lane; i < D; i += 32) {
      double acc = 0.0;
      for (int j = 0; j < D; ++j) acc += Kc[(size_t)j * D + i] * vs[warp][j];
      if (out) out[(size_t)a.cl_body[base + i / 12] * 12 + i % 12] = acc;
      if (dot) xs_add(*dot, vs[warp][i] * acc);
    }
    __syncwarp();
  }
}

// ---- the solve's set-up ----
// One launch, one warp per cluster (every body is in exactly one): the residual r = b - A x of
// the cluster's bodies (BiCGSTAB: also rh = r, p = v = 0), z = M^-1 r (PCG: also p = z) and
// M^-1 b, with the exact partials of b.M^-1 b, r.r and r.z -- the arithmetic of the row
// kernels and of cluster_apply, entry for entry.  The last CTA rounds the three totals and
// starts the solve: the threshold tol^2 b.M^-1 b, the scalars, the iteration counter, the outcome
// flags and the WHILE node's condition (set at every solve: the loop's node may sit inside
// another conditional node, whose launches do not reset it).  With b.M^-1 b <= 0 the solution
// is 0 (x is cleared) and no iteration runs; a solve without iterations is tallied here.
__global__ void __launch_bounds__(AT) k_krylov_setup(LargeArgs a, const double* bvec, double* x, double* r,
                                                     double* z, double* pz, double* rh, double* p0, double* v0,
                                                     double tol2, cudaGraphConditionalHandle h) {
  // a pass that is made again, or an iteration whose solve is done (its list was made again)
  if ((a.dstat[DS_STATUS] & kRerunMask) || (a.tally && a.tally->step.resume)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
    return;
  }
  constexpr int NWA = AT / 32;
  __shared__ double vr[NWA][12 * kMaxCluster], vb[NWA][12 * kMaxCluster];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  XSum bz, rr, rz;
  xs_zero(bz);
  xs_zero(rr);
  xs_zero(rz);
  const int ncl = *a.ncl_dev;
  for (int c = blockIdx.x * NWA + warp; c < ncl; c += gridDim.x * NWA) {
    const int base = a.cl_ptr[c], sz = a.cl_ptr[c + 1] - base, D = 12 * sz;
    for (int m = 0; m < sz; ++m) {
      const int b = a.cl_body[base + m];
      const double ax = row_product(a, b, x);
      if (lane < 12) {
        const size_t i = (size_t)b * 12 + lane;
        const double bi = bvec[i], ri = bi - ax;
        r[i] = ri;
        if (rh) rh[i] = ri;
        if (p0) p0[i] = 0.0;
        if (v0) v0[i] = 0.0;
        xs_add(rr, ri * ri);
        vr[warp][12 * m + lane] = ri;
        vb[warp][12 * m + lane] = bi;
      }
    }
    __syncwarp();
    const double* Kc = a.cl_inv + a.cl_off[c];
    for (int i = lane; i < D; i += 32) {
      double ar = 0.0, ab = 0.0;
      for (int j = 0; j < D; ++j) {
        const double k = Kc[(size_t)j * D + i];
        ar += k * vr[warp][j];
        ab += k * vb[warp][j];
      }
      const size_t gi = (size_t)a.cl_body[base + i / 12] * 12 + i % 12;
      z[gi] = ar;
      if (pz) pz[gi] = ar;
      xs_add(rz, vr[warp][i] * ar);
      xs_add(bz, vb[warp][i] * ab);
    }
    __syncwarp();
  }
  __shared__ XSum sh[NWA];
  cta_partial(a, bz, SL_BZ, sh);
  cta_partial(a, rr, SL_RHR, sh);
  cta_partial(a, rz, SL_RZ0, sh);
  if (!cta_last(a, SL_BZ)) return;
  total_of(a, SL_BZ, sh);
  total_of(a, SL_RHR, sh);
  total_of(a, SL_RZ0, sh);
  __syncthreads();  // the totals, stored by thread 0
  const double b = a.scal[SC_RED + SL_BZ];
  if (!(b > 0.0))
    for (int i = threadIdx.x; i < 12 * a.n; i += AT) x[i] = 0.0;
  if (threadIdx.x == 0) {
    a.scal[SC_RHO0] = a.scal[SC_RHO1] = a.scal[SC_ALPHA] = a.scal[SC_OMEGA] = 1.0;
    a.scal[SC_THR2] = tol2 * b;
    a.ki[KI_IT] = 1;
    a.ki[KI_RUNS] = 0;
    // the solve's outcome flags start clear (the iterations that follow set and read them)
    a.dstat[DS_R_DONE] = b > 0.0 ? 0 : 1;
    a.dstat[DS_S_DONE] = 0;
    a.dstat[DS_SOLVER_ITERS] = 0;
    const bool loop = b > 0.0 && a.maxit >= 1;
    if (!loop) tally_solve(a);
    cudaGraphSetConditional(h, loop ? 1u : 0u);
  }
}

// ---- PCG ----
// K1: converged if r.z <= thr^2; else Ap = A p with partial p.Ap
__global__ void __launch_bounds__(256) k_pcg_1(LargeArgs a, const double* pv, double* Ap) {
  count_run(a);
  const int it = iteration(a);
  if (solver_done(a.dstat) || it > a.maxit) return;
  const int rz = (it & 1) ? SL_RZ0 : SL_RZ1;
  const int slots[1] = {rz};
  double sc[1];
  cta_scalars(a, slots, 1, sc);
  if (!(sc[0] > a.scal[SC_THR2])) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.dstat[DS_R_DONE] = it;
      a.dstat[DS_SOLVER_ITERS] = it - 1;
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  XSum d0, d1;
  xs_zero(d0);
  xs_zero(d1);
  FOR_BODIES(b) {
    const double yi = row_product(a, b, pv);
    if (lane < 12) {
      const size_t i = (size_t)b * 12 + lane;
      Ap[i] = yi;
      xs_add(d0, pv[i] * yi);
    }
  }
  cta_partials(a, d0, d1, SL_PAP, -1);
}

// K2: alpha = rz / p.Ap; x += alpha p; r -= alpha Ap (stops on a non-positive curvature); then
// z = M^-1 r with the partial r.z into the new slot, one warp per cluster (cluster_apply: the
// update of the cluster's bodies, then the product over the updated r).  The iteration's end
// (loop_end): by the last CTA, or by CTA 0 when the solve stops here or has stopped.
__global__ void __launch_bounds__(AT) k_pcg_2(LargeArgs a, const double* pv, const double* Ap, double* x, double* r,
                                              double* z) {
  const int it = iteration(a);
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  if (solver_done(a.dstat) || it > a.maxit) {
    if (lead) loop_end(a, 1);
    return;
  }
  const int rz = (it & 1) ? SL_RZ0 : SL_RZ1;
  const int slots[2] = {rz, SL_PAP};
  double sc[2];
  cta_scalars(a, slots, 2, sc);
  if (!(sc[1] > 0.0)) {
    if (lead) {
      a.dstat[DS_R_DONE] = it;
      a.dstat[DS_SOLVER_ITERS] = it - 1;
      loop_end(a, 1);
    }
    return;
  }
  const double alpha = sc[0] / sc[1];
  XSum d0, d1;
  xs_zero(d0);
  xs_zero(d1);
  cluster_apply(a, z, &d0, [&](size_t i) {
    x[i] += alpha * pv[i];
    const double ri = r[i] - alpha * Ap[i];
    r[i] = ri;
    return ri;
  });
  if (cta_partials(a, d0, d1, (it & 1) ? SL_RZ1 : SL_RZ0, -1) && threadIdx.x == 0) {
    a.dstat[DS_SOLVER_ITERS] = it;
    loop_end(a, 1);  // (the new r.z is final)
  }
}

// K3 (after K2's z = M^-1 r and r.z in the new slot): beta = rz_new / rz_old; p = z + beta p
__global__ void __launch_bounds__(256) k_pcg_3(LargeArgs a, const double* z, double* pv) {
  const int it = iteration(a) - 1;  // (K2 ended the iteration: the counter is one ahead)
  if (solver_done(a.dstat) || it > a.maxit) return;
  const int rz_old = (it & 1) ? SL_RZ0 : SL_RZ1, rz_new = (it & 1) ? SL_RZ1 : SL_RZ0;
  const int slots[2] = {rz_new, rz_old};
  double sc[2];
  cta_scalars(a, slots, 2, sc);
  if (!(sc[0] > a.scal[SC_THR2])) return;  // converged: K1 of the next iteration stops
  const double beta = sc[0] / sc[1];
  const int lane = threadIdx.x & 31;
  FOR_BODIES(b) {
    if (lane < 12) {
      const size_t i = (size_t)b * 12 + lane;
      pv[i] = z[i] + beta * pv[i];
    }
  }
}

// ---- BiCGSTAB (right preconditioned) ----
// K1: converged if r.M^-1 r small; rho = rh.r; p = r + beta (p - omega v); then y = M^-1 p,
// one warp per cluster (cluster_apply)
__global__ void __launch_bounds__(AT) k_bicg_1(LargeArgs a, const double* r, double* pv, const double* v,
                                               double* y) {
  count_run(a);
  const int it = iteration(a);
  if (solver_done(a.dstat) || it > a.maxit) return;
  const int slots[2] = {SL_RZ0, SL_RHR};
  double sc[2];
  cta_scalars(a, slots, 2, sc);
  if (!(sc[0] > a.scal[SC_THR2]) || sc[1] == 0.0 || !isfinite(sc[1])) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      a.dstat[DS_R_DONE] = it;
      a.dstat[DS_SOLVER_ITERS] = it - 1;
    }
    return;
  }
  const double rho = sc[1];
  const double rho_old = a.scal[(it + 1) & 1];
  const double alpha = a.scal[SC_ALPHA], omega = a.scal[SC_OMEGA];
  const double beta = (rho / rho_old) * (alpha / omega);
  cluster_apply(a, y, nullptr, [&](size_t i) {
    const double pi = it == 1 ? r[i] : r[i] + beta * (pv[i] - omega * v[i]);
    pv[i] = pi;
    return pi;
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) a.scal[it & 1] = rho;
}

// out = A in; partials w0.out (slot0), w1.out (slot1)
__global__ void __launch_bounds__(256) k_spmv(LargeArgs a, const double* in, double* out, const double* w0, int slot0,
                                              const double* w1, int slot1) {
  if (solver_done(a.dstat) || iteration(a) > a.maxit) return;
  const int lane = threadIdx.x & 31;
  XSum d0, d1;
  xs_zero(d0);
  xs_zero(d1);
  FOR_BODIES(b) {
    const double yi = row_product(a, b, in);
    if (lane < 12) {
      const size_t i = (size_t)b * 12 + lane;
      out[i] = yi;
      if (w0) xs_add(d0, w0[i] * yi);
      if (w1) xs_add(d1, w1[i] * yi);
    }
  }
  cta_partials(a, d0, d1, slot0, slot1);
}

// K3: alpha = rho / rh.v; s = r - alpha v; then z = M^-1 s with the partial s.z, one warp per
// cluster (cluster_apply)
__global__ void __launch_bounds__(AT) k_bicg_3(LargeArgs a, const double* r, const double* v, double* s,
                                               double* z) {
  const int it = iteration(a);
  if (solver_done(a.dstat) || it > a.maxit) return;
  const int slots[1] = {SL_RHV};
  double sc[1];
  cta_scalars(a, slots, 1, sc);
  const double alpha = a.scal[it & 1] / sc[0];
  XSum d0, d1;
  xs_zero(d0);
  xs_zero(d1);
  cluster_apply(a, z, &d0, [&](size_t i) {
    const double si = r[i] - alpha * v[i];
    s[i] = si;
    return si;
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) a.scal[SC_ALPHA] = alpha;
  cta_partials(a, d0, d1, SL_SZ, -1);
}

// K4 (after K3's z = M^-1 s and s.z): if small, x += alpha y and stop
__global__ void __launch_bounds__(256) k_bicg_4(LargeArgs a, const double* y, double* x) {
  const int it = iteration(a);
  const volatile int* ds = a.dstat;
  if (ds[DS_R_DONE] != 0 || (ds[DS_S_DONE] != 0 && ds[DS_S_DONE] != it) || it > a.maxit) return;
  const int slots[1] = {SL_SZ};
  double sc[1];
  cta_scalars(a, slots, 1, sc);
  if (sc[0] > a.scal[SC_THR2]) return;
  const double alpha = a.scal[SC_ALPHA];
  const int lane = threadIdx.x & 31;
  FOR_BODIES(b) {
    if (lane < 12) {
      const size_t i = (size_t)b * 12 + lane;
      x[i] += alpha * y[i];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.dstat[DS_S_DONE] = it;
    a.dstat[DS_SOLVER_ITERS] = it;
  }
}

// K6: omega = t.s / t.t; x += alpha y + omega z; r = s - omega t; partial rh.r; then the
// partial r.M^-1 r, one warp per cluster (cluster_apply; the product itself is not kept).  The
// iteration's end (loop_end): by the last CTA, or by CTA 0 when the solve has stopped.
__global__ void __launch_bounds__(AT) k_bicg_6(LargeArgs a, const double* y, const double* z, const double* s,
                                               const double* t, const double* rh, double* x, double* r) {
  const int it = iteration(a);
  if (solver_done(a.dstat) || it > a.maxit) {
    if (blockIdx.x == 0 && threadIdx.x == 0) loop_end(a, 0);
    return;
  }
  const int slots[2] = {SL_TS, SL_TT};
  double sc[2];
  cta_scalars(a, slots, 2, sc);
  const double omega = sc[0] / sc[1];
  const double alpha = a.scal[SC_ALPHA];
  XSum rz, rhr;
  xs_zero(rz);
  xs_zero(rhr);
  cluster_apply(a, nullptr, &rz, [&](size_t i) {
    x[i] += alpha * y[i] + omega * z[i];
    const double ri = s[i] - omega * t[i];
    r[i] = ri;
    xs_add(rhr, rh[i] * ri);
    return ri;
  });
  if (cta_partials(a, rz, rhr, SL_RZ0, SL_RHR) && threadIdx.x == 0) {
    a.scal[SC_OMEGA] = omega;
    a.dstat[DS_SOLVER_ITERS] = it;
    loop_end(a, 0);  // (r.M^-1 r and rh.r are final)
  }
}

}  // namespace

int krylov_large_kernels(const Sim& s) { return s.prm.solver == 1 ? 3 : 6; }

// Enqueues a solve on s.stream, which must be capturing: the set-up kernel, then a WHILE node whose
// body is one iteration, captured on cap_stream5
int krylov_large_issue(Sim& s, double* x, bool tally) {
  const bool pcg = s.prm.solver == 1;
  const size_t m = 12 * (size_t)s.n;
  double *const r = s.kry_vec, *const rh = r + m, *const pv = r + 2 * m, *const v = r + 3 * m, *const y = r + 4 * m,
         *const sv = r + 5 * m, *const z = r + 6 * m, *const t = r + 7 * m;
  LargeArgs a;
  a.n = s.n;
  a.diag = s.diag;
  a.offdiag = s.offdiag;
  a.row_ptr = s.row_ptr;
  a.adj_col = s.adj_col;
  a.adj_pair = s.adj_pair;
  a.pair_active = s.pair_active;
  a.fixed = s.fixed;
  a.ij = s.ij;
  a.ncl_dev = s.ncl_dev;
  a.maxit = s.prm.cg_max_iter;
  a.cl_ptr = s.cl_ptr;
  a.cl_body = s.cl_body;
  a.cl_off = s.cl_off;
  a.cl_inv = s.cl_inv;
  a.part = s.partials;
  a.red_count = s.red_count;
  a.scal = s.kry_scal;
  a.ki = s.kry_int;
  a.dstat = s.dstat;
  a.tally = tally ? s.box : nullptr;
  if (int q = make_handle(s.stream, &a.loop)) return q;
  const int rows = std::min(kRedBlocks, (s.n + WPB - 1) / WPB), cls = std::min(kRedBlocks, (s.n + 3) / 4);
  k_krylov_setup<<<cls, AT, 0, s.stream>>>(a, s.g, x, r, z, pcg ? pv : nullptr, pcg ? nullptr : rh, pcg ? nullptr : pv,
                                           pcg ? nullptr : v, s.prm.cg_tol * s.prm.cg_tol, a.loop);
  ++s.launches;
  if (ABD_NOTE(cudaGetLastError()) != cudaSuccess) return ABD_ERR_CUDA;
  cudaGraph_t body = nullptr;
  if (int q = add_conditional(s.stream, a.loop, cudaGraphCondTypeWhile, &body)) return q;
  return capture_body(s, body, s.cap_stream5, [&]() -> int {
    const cudaStream_t bs = s.stream;
    if (pcg) {
      k_pcg_1<<<rows, 256, 0, bs>>>(a, pv, v);
      k_pcg_2<<<cls, AT, 0, bs>>>(a, pv, v, x, r, z);
      k_pcg_3<<<rows, 256, 0, bs>>>(a, z, pv);
    } else {
      k_bicg_1<<<cls, AT, 0, bs>>>(a, r, pv, v, y);
      k_spmv<<<rows, 256, 0, bs>>>(a, y, v, rh, SL_RHV, nullptr, -1);
      k_bicg_3<<<cls, AT, 0, bs>>>(a, r, v, sv, z);
      k_bicg_4<<<rows, 256, 0, bs>>>(a, y, x);
      k_spmv<<<rows, 256, 0, bs>>>(a, z, t, sv, SL_TS, t, SL_TT);
      k_bicg_6<<<cls, AT, 0, bs>>>(a, y, z, sv, t, rh, x, r);
    }
    return ABD_NOTE(cudaGetLastError()) == cudaSuccess ? ABD_OK : ABD_ERR_CUDA;
  });
}

}  // namespace abd
