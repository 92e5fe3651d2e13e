// Krylov solve of the Newton system H dq = g: preconditioned CG or BiCGSTAB in one kernel.
//
// Replaces warp.optim.linear.bicgstab(hess, g, dq, 1e-4) and warp.sparse's BSR product
// (abd/abd.py:243-244).  The arithmetic is the row-wise one of the block-sparse system: a row
// of A x is two half-row sums (columns 0-5, 6-11) over the diagonal block, then the active
// neighbours in increasing order; a row of M^-1 r is the dense inverse's row summed in column
// order; dot products are exact (abd_exact.cuh).  Convergence is measured in the
// preconditioned norm, r^T M^-1 r <= tol^2 b^T M^-1 b, which stays resolvable in FP64 although
// the plain residual of such stiff systems has a rounding floor near eps * cond.
//
// What bounds it: a solve is a chain of two (BiCGSTAB: six) short phases per iteration, each
// ended by a dot product that every row needs.  The system is small (2.4 MB for 1024 bodies),
// so the chain's latency counts, not the bandwidth: as one kernel per phase inside a WHILE node
// of the step's graph an iteration of the 1024-body pile took 25.7 us and the set-up 25.4 us (72
// us a solve of 1.8 iterations; 8 bodies: 50 us), nearly all of it launches, the loop node and
// partials summed through global memory; this kernel takes 37 us (8 bodies: 16 us).  Here one
// thread-block cluster (at most 16 CTAs) holds the whole solve: a thread per row, the rows'
// vectors in shared memory, the phases separated by the hardware cluster barrier, and the
// partial sums of a dot product pushed into every CTA's shared memory (distributed shared
// memory) before that barrier.  p (PCG) is not published after its update: a neighbour's p is
// formed from the published z and the p of the iteration before, so an iteration has two
// cluster barriers.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "abd_graph.cuh"
#include "abd_krylov.cuh"

namespace abd {

using krylov::KC;
using krylov::KrylovArgs;
using krylov::PosInfo;
using krylov::RedShared;

// The arguments of a solve by a cluster of C CTAs, and the dynamic shared memory it takes
KrylovArgs krylov_args(Sim& s, double* x, bool tally, int C, size_t* smem_out) {
  const bool pcg = s.prm.solver == 1;
  KrylovArgs a;
  a.n = s.n;
  a.maxit = s.prm.cg_max_iter;
  a.diag = s.diag;
  a.offdiag = s.offdiag;
  a.g = s.g;
  a.row_ptr = s.row_ptr;
  a.adj_col = s.adj_col;
  a.adj_pair = s.adj_pair;
  a.pair_active = s.pair_active;
  a.fixed = s.fixed;
  a.nb = s.nb_act;
  a.cl_ptr = s.cl_ptr;
  a.cl_body = s.cl_body;
  a.body_cl = s.body_cl;
  a.cl_off = s.cl_off;
  a.cl_inv = s.cl_inv;
  a.tol2 = s.prm.cg_tol * s.prm.cg_tol;
  a.x = x;
  a.pub0 = s.kry_pub;
  a.pub1 = s.kry_pub + 12 * (size_t)s.n;
  a.pub2 = s.kry_pub + 24 * (size_t)s.n;
  a.dstat = s.dstat;
  a.tally = tally ? s.box : nullptr;
  // a CTA's share, plus the members its last cluster may reach over it
  a.pos_max = std::min(s.n, (s.n + C - 1) / C + kMaxCluster);
  a.rows_max = 12 * a.pos_max;
  *smem_out = (size_t)a.rows_max * (pcg ? 4 : 6) * sizeof(double) + (size_t)a.pos_max * sizeof(PosInfo);
  return a;
}

namespace {

constexpr int KT = 512;        // most threads of a CTA

template <bool PCG>
__global__ void __launch_bounds__(KT) k_krylov(const __grid_constant__ KrylovArgs a) {
  extern __shared__ double2 dyn2[];
  // a pass that is made again, or an iteration whose solve is done (its list was made again)
  if ((a.dstat[DS_STATUS] & kRerunMask) || (a.tally && a.tally->step.resume)) return;
  __shared__ RedShared red;
  krylov::solve<PCG, true>(a, reinterpret_cast<double*>(dyn2), red, (int)gridDim.x, (int)blockIdx.x);
}

// CTAs of the cluster: about 192 rows each, at most the largest cluster the device can hold
int cluster_ctas(const Sim& s) {
  int c = 1;
  while (c < s.max_cluster && 192 * c < 12 * s.n) c *= 2;
  return c;
}

cudaError_t enqueue(Sim& s, double* x, bool tally) {
  const bool pcg = s.prm.solver == 1;
  const int C = cluster_ctas(s);
  size_t smem = 0;
  const KrylovArgs a = krylov_args(s, x, tally, C, &smem);
  // threads: the rows in as few rounds as KT allows, spread evenly
  const int rows = 12 * ((s.n + C - 1) / C), rounds = (rows + KT - 1) / KT;
  const int T = std::max(64, ((rows + rounds - 1) / rounds + 31) / 32 * 32);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ++s.launches;
  return pcg ? cudaLaunchKernelEx(&cfg, k_krylov<true>, a) : cudaLaunchKernelEx(&cfg, k_krylov<false>, a);
}

// the largest cluster (16, 8, ... CTAs) of the kernel at its largest shared memory
template <class K>
cudaError_t fit_cluster(K kernel, int* best) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kKrylovSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  for (; *best > 1; *best /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(*best);
    cfg.blockDim = dim3(KT);
    cfg.dynamicSmemBytes = kKrylovSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = *best;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int k = 0;
    e = cudaOccupancyMaxActiveClusters(&k, kernel, &cfg);
    if (e == cudaSuccess && k > 0) return e;
    (void)cudaGetLastError();
  }
  return cudaSuccess;
}

}  // namespace

// Which solves are made by krylov_large.cu's kernels: more than kLargeBodies bodies (or, where the device
// holds smaller clusters, vectors that do not fit them).  Below, this file's cluster is the faster one
// for the few iterations that a step's solves take and for many: with 2,117 bodies a solve of two CG
// iterations takes 128 us and each further one 20 us (377 and 29 us there, in round figures the cost of its
// launches); with 4,097 bodies 178 and 193 us; 5,001 205 and 209; 8,101 300 (67 us an iteration) and 267 (50);
// 16,385 566 (130) and 424 (73).  BiCGSTAB the same: 8,101 bodies 341 (157 us an iteration) and 282 (114).
constexpr int kLargeBodies = 4096;
bool krylov_is_large(const Sim& s) {
  if (s.n > kLargeBodies) return true;
  const int C = cluster_ctas(s);
  const size_t pos = std::min(s.n, (s.n + C - 1) / C + kMaxCluster);
  return pos * (12 * 6 * sizeof(double) + sizeof(PosInfo)) > (size_t)kKrylovSmem;  // (BiCGSTAB's)
}

cudaError_t prepare_krylov(Sim& s) {
  // the kernels' attributes and the largest cluster are the device's: found once per device (the
  // queries take milliseconds)
  static std::mutex m;
  static std::map<int, int> known;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(m);
  int& best = known[dev];
  if (best == 0) {
    int c = KC;
    e = fit_cluster(k_krylov<true>, &c);
    if (e == cudaSuccess) e = fit_cluster(k_krylov<false>, &c);
    if (e != cudaSuccess) return e;
    best = c;
  }
  s.max_cluster = best;
  if (!krylov_is_large(s)) return cudaSuccess;
  e = cudaMalloc(&s.kry_vec, sizeof(double) * 96 * (size_t)s.n);
  if (e == cudaSuccess) e = cudaMalloc(&s.kry_scal, sizeof(double) * 32);
  if (e == cudaSuccess) e = cudaMalloc(&s.kry_int, sizeof(int) * 4);
  return e;
}

int krylov_solve(Sim& s, double* x, int* iters_out) {
  const bool large = krylov_is_large(s);
  // (the kernel loads x in 16-byte pieces; a large solve's graph is kept for its own vectors)
  double* const y = x == s.dq || (!large && reinterpret_cast<uintptr_t>(x) % 16 == 0) ? x : s.adj_x;
  const size_t bytes = sizeof(double) * 12 * (size_t)s.n;
  if (y != x && ABD_NOTE(cudaMemcpyAsync(y, x, bytes, cudaMemcpyDeviceToDevice, s.stream)) != cudaSuccess)
    return ABD_ERR_CUDA;
  if (large) {
    KeyHash k;
    k.add(y).add(s.prm_version).add(s.prm.solver).add(s.cap_gen);
    if (int r = run_graph(s, y == s.dq ? s.g_solve_dq : s.g_solve, k.h, [&]() { return krylov_large_issue(s, y, false); }))
      return r;
  } else if (ABD_NOTE(enqueue(s, y, false)) != cudaSuccess) {
    return ABD_ERR_CUDA;
  }
  if (y != x && ABD_NOTE(cudaMemcpyAsync(x, y, bytes, cudaMemcpyDeviceToDevice, s.stream)) != cudaSuccess)
    return ABD_ERR_CUDA;
  if (!iters_out) return ABD_OK;
  if (cudaMemcpyAsync(s.hbox, s.box, sizeof(Mailbox), cudaMemcpyDeviceToHost, s.stream) ||
      cudaStreamSynchronize(s.stream) != cudaSuccess)
    return ABD_ERR_CUDA;
  *iters_out = krylov_outcome(s);
  return ABD_OK;
}

int krylov_issue(Sim& s, double* x) {
  if (!krylov_is_large(s)) return ABD_NOTE(enqueue(s, x, true)) == cudaSuccess ? ABD_OK : ABD_ERR_CUDA;
  if (int r = krylov_large_issue(s, x, true)) return r;
  s.loop.solve = krylov_large_kernels(s);
  return ABD_NOTE(dots(s, x, s.g, s.g, s.g, s.box->dots, s.stream)) == cudaSuccess ? ABD_OK : ABD_ERR_CUDA;
}

int krylov_outcome(Sim& s) {
  const int* ds = s.hbox->dstat;
  if (!(ds[krylov::DS_R_DONE] || ds[krylov::DS_S_DONE])) s.host_status |= ST_SOLVER_NOCONV;
  if (krylov_is_large(s)) s.launches += (long long)krylov_large_kernels(s) * ds[DS_SOLVER_ITERS];
  return ds[DS_SOLVER_ITERS];
}

}  // namespace abd
