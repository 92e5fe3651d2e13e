// The preconditioner of the Newton linear solve H dq = g (krylov.cu), which the reference's
// bicgstab call (abd/abd.py:244) does not have: contact-cluster block Jacobi.  Barrier stiffness between touching bodies is
// 1e8-1e10 times their mass, so a per-body block Jacobi leaves the Krylov method facing that
// condition number.  Bodies coupled by active contacts are grouped on the device (mutual
// strongest couplings merge in rounds, at most cluster_max bodies: k_clusters); each
// cluster's dense system is assembled and inverted (Gauss-Jordan, SPD, no pivoting) by one
// warp in registers (one body) or four CTAs in shared memory (more), and applied as a dense
// product.  Clusters of one body reduce to the per-body 12x12 block.
// The inverses are stored transposed: the solve's threads hold a row each, so a column of the
// transposed inverse is a coalesced load.
#include <cuda_runtime.h>

#include <algorithm>

#include "abd_precond.cuh"

namespace abd {

using namespace precond;

SolverArgs solver_args(Sim& s) {
  SolverArgs a;
  a.diag = s.diag;
  a.offdiag = s.offdiag;
  a.row_ptr = s.row_ptr;
  a.adj_col = s.adj_col;
  a.adj_pair = s.adj_pair;
  a.pair_active = s.pair_active;
  a.fixed = s.fixed;
  a.ncl_dev = s.ncl_dev;
  a.dstat = s.dstat;
  a.resume = s.in_device_loop ? &s.box->step.resume : nullptr;
  a.cl_ptr = s.cl_ptr;
  a.cl_body = s.cl_body;
  a.body_cl = s.body_cl;
  a.big = s.cl_work.to;
  a.n = s.n;
  a.cl_off = s.cl_off;
  a.cl_inv = s.cl_inv;
  return a;
}

int cluster_cap(const Sim& s) { return s.prm.precond == 1 ? std::max(1, std::min(kMaxCluster, s.prm.cluster_max)) : 1; }

namespace {

constexpr int BT = 288;                        // threads of the inverse: two per row of the largest system
constexpr int kBigCtas = 2 * 148;              // most CTAs for the larger clusters: two per SM
constexpr int kSmallCtas = 148;                // and for one-body clusters, a warp each
constexpr int KT = 1024;                       // threads of the clustering CTA

__global__ void __cluster_dims__(BC, 1, 1) __launch_bounds__(BT, 2) k_cluster_inverse(const __grid_constant__ SolverArgs a,
                                                                                   int big_ctas) {
  extern __shared__ double dyn[];
  if ((a.dstat[DS_STATUS] & kRerunMask) || (a.resume && *a.resume)) return;  // (no tables, or no solve)
  const int bx = (int)blockIdx.x;
  if (bx < big_ctas) {
    BigShared& S = *reinterpret_cast<BigShared*>(dyn);
    const int solo = a.ncl_dev[1], multi = a.ncl_dev[2];
    for (int e = bx / BC; e < multi; e += big_ctas / BC) big_inverse<BT>(a, S, a.big[a.n - 1 - e], bx % BC, BC);
    for (int e = bx; e < solo; e += big_ctas) big_inverse<BT>(a, S, a.big[e], 0, 1);
    return;
  }
  const int ncl = *a.ncl_dev, lane = (int)(threadIdx.x & 31);
  const int nw = ((int)gridDim.x - big_ctas) * (BT / 32);
  for (int c = (int)(((bx - big_ctas) * BT + threadIdx.x) >> 5); c < ncl; c += nw) {
    const int base = a.cl_ptr[c];
    if (a.cl_ptr[c + 1] - base == 1) warp_inverse1(a, c, a.cl_body[base], lane);
  }
}

// (skipped when the list overflowed: the pass is made again)
__global__ void __launch_bounds__(KT) k_clusters(int n, int cap, const int4* act, int cap_act, const int* dstat,
                                                 ClusterTables t, ClusterWork w) {
  if (dstat[DS_STATUS] & (ST_ACT_OVERFLOW | ST_PAIR_OVERFLOW | ST_CONTACT_OVERFLOW)) return;
  make_clusters<KT>(n, cap, act, cap_act, dstat, t, w);
}

}  // namespace

// Clusters of the preconditioner from the active-pair list of the last GH pass, on the device
// (k_clusters); enqueued on stream st (the pass's stream when null).
cudaError_t cluster_tables(Sim& s, cudaStream_t st) {
  k_clusters<<<1, KT, 0, st ? st : s.stream>>>(s.n, cluster_cap(s), s.act_pairs, s.cap_act, s.dstat,
                                               cluster_tables_at(s.cl_tab, s.n), s.cl_work);
  ++s.launches;
  return cudaGetLastError();
}

// Inverts every cluster's dense system (the tables k_clusters made; their counts are read on the
// device), in one launch of a fixed grid.
int cluster_inverse(Sim& s) {
  // (whole clusters of CTAs; a larger cluster takes at least two bodies)
  const int big = std::min(kBigCtas, BC * std::max(1, s.n / 2));
  const int small = std::min(kSmallCtas, BC * ((s.n + BC * (BT / 32) - 1) / (BC * (BT / 32))));
  static_assert(kBigCtas % BC == 0 && kSmallCtas % BC == 0, "whole clusters");
  k_cluster_inverse<<<big + small, BT, sizeof(BigShared), s.stream>>>(solver_args(s), big);
  ++s.launches;
  return ABD_NOTE(cudaGetLastError()) == cudaSuccess ? ABD_OK : ABD_ERR_CUDA;
}

// Opts the inverse kernel in to its shared memory (once, at creation: the passes that launch it may
// be under stream capture)
int prepare_solver(Sim& s) {
  (void)s;
  return cudaFuncSetAttribute(k_cluster_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BigShared)) ==
                 cudaSuccess
             ? ABD_OK
             : ABD_ERR_CUDA;
}

int build_preconditioner(Sim& s) {
  if (cluster_tables(s, nullptr) != cudaSuccess) return ABD_ERR_CUDA;
  return cluster_inverse(s);
}

}  // namespace abd
