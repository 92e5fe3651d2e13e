// The Newton iterations of many small scenes in one kernel.
//
// A scene's step is a graph (newton.cu) whose iterations are ten kernels in a WHILE node, and a
// batch of scenes was a graph with such a branch per scene.  But a graph's branches share eight
// hardware queues: of 48 scenes about eight ran at a time, 9 to 12 ms a step in which each scene
// took about 1 ms.  Here one launch holds every scene's iterations: a thread-block cluster
// per scene goes through the phases of its loop (the headers that the kernels are made of),
// separated by the hardware cluster barrier.  Every sum is exact and every list's order is
// immaterial, so the results are the kernels', bit for bit.
//
// The rule (batch_loop_takes): scenes with the reference's contact model, no friction and the CG
// solver, when the batch has kBatchLeast of them; a scene of at most kLoopBodies bodies, and of vertices
// and edges at most kLoopPrims or, if that is more, kLoopShare for each scene of the batch.  A larger
// scene's phases want more SMs than a cluster has, and get them while few scenes share the GPU; with
// fewer scenes than the eight queues each has one.  Measured, a step as branches -> in this kernel:
//   scenes   9 of 4 to 14 bodies 2.5 -> 1.7 ms, 48 11.6 -> 4.0, 512 198 -> 28 (6: 1.9 -> 1.5, 4: 1.3 -> 1.4);
//   bodies   12 scenes of 127 3.9 -> 2.6 ms, of 176 3.9 -> 3.1;
//   vertices and edges a scene   41,000: 9 scenes 4.2 -> 3.6 ms, 48 21.5 -> 13.5;  82,000: 9 scenes
//            5.3 -> 6.7, 24 11.3 -> 9.9;  164,000: 12 scenes 9.8 -> 13.6, 24 18.2 -> 18.1, 48 36.6 -> 32.9.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>

#include "abd_assemble.cuh"
#include "abd_ghpass.cuh"
#include "abd_krylov.cuh"
#include "abd_listccd.cuh"
#include "abd_lsterms.cuh"
#include "abd_precond.cuh"

namespace abd {

namespace {

namespace cg = cooperative_groups;

constexpr int LT = assemble::PT_THREADS;  // threads of a CTA
constexpr int kLoopCtas = 16;             // most CTAs of a cluster
constexpr int kLoopBodies = 192, kLoopPrims = 1 << 16, kLoopShare = 1 << 12;
constexpr int kLoopSlots = 2 * 148;       // CTAs resident at a time: two per SM (128 registers)
static_assert(LT >= 160, "a body's pass");
// four CTAs at least, so that a preconditioner cluster's panels fit (abd_precond.cuh)
constexpr int kLoopLeast = precond::BC;

struct LoopArgs {
  NarrowArgs gh;
  BodyArgs body;
  precond::SolverArgs pre;
  krylov::KrylovArgs kry;
  ccd::CcdArgs ccd;
  ls::LsArgs ls;
  ClusterTables tables;
  ClusterWork work;
  int cap_cluster;  // most bodies of a preconditioner cluster
  int cap_pairs;
  Mailbox* box;
  int* bad;
  double *Ak, *pk;
};
static_assert(sizeof(LoopArgs) % 8 == 0, "copied in 8-byte words");

struct LoopShared {
  unsigned long long args[sizeof(LoopArgs) / 8];
  krylov::RedShared red;
  BodyShared body;
  int acc[kLsMax][kDSlots];  // the CTA's terms of the line search's trials
  double al[kLsMax];         // their step lengths
  int first, count;
  double e1;
};

// The CCD pass's step bound and candidates, as k_list_ccd (listpass.cu)
__device__ __noinline__ void ccd_phase(const ccd::CcdArgs& a, bool ground, int rank, int C) {
  const int tid = (int)threadIdx.x, m = min(a.box->dstat[DS_NLIST], a.cap_list);
  // (the bodies go to the last CTA's threads, the candidates start at the first's)
  for (int b = (C - 1 - rank) * LT + tid; b < a.n; b += C * LT) ccd::body(a, b);
  for (int i = rank * LT + tid; i < m; i += C * LT) ccd::candidate<true>(a, i);
  if (!ground) return;
  for (int b = rank; b < a.n; b += C) {
    ccd::ground(a, b);
    __syncthreads();
  }
}

// Trials [k0, k0 + g) of the line search, m terms each: their energies into a.energy
__device__ __noinline__ void trials_phase(const ls::LsArgs& a, LoopShared& S, int k0, int g, int cnt, int m, int rank,
                                          int C) {
  const int tid = (int)threadIdx.x;
  for (int e = tid; e < g * kDSlots; e += LT) (&S.acc[0][0])[e] = 0;
  __syncthreads();
  constexpr int kRounds = 256;  // rounds of LT terms between folds
  static_assert(LT * kRounds + 64 < kDTerms, "the terms between two folds fit the counters");
  const int nv = m - cnt - a.n;
  int r = 0;
  for (long long q0 = (long long)rank * LT; q0 < (long long)g * m; q0 += C * LT) {
    if (++r == kRounds) {
      r = 0;
      __syncthreads();
      for (int k = tid >> 5; k < g; k += LT / 32) ds_fold(S.acc[k]);
      __syncthreads();
    }
    const long long q = q0 + tid;
    if (q >= (long long)g * m) continue;
    const int k = (int)(q / m), i = (int)(q % m);
    const double al = S.al[k0 + k];
    double e = 0.0;
    if (i < cnt) e = ls::candidate<true>(a, al, i);
    else if (i < cnt + nv) e = ls::vertex(a, al, i - cnt);
    else if (!a.fixed[i - cnt - nv]) e = ls::inertia(a, al, i - cnt - nv);
    if (e != 0.0) ds_add(S.acc[k], e);
  }
  __syncthreads();
  for (int e = tid; e < g * kDSlots; e += LT) ds_to_limbs(S.acc[e / kDSlots], e % kDSlots, &a.energy[k0 + e / kDSlots]);
}

// Newton iterations of scene blockIdx.x / C until its loop's end (k_newton_end's rules, newton.cu), by
// its cluster.  Whatever decides where a CTA goes next (status bits, the list's state, the trials'
// energies) is read between two barriers between which nothing writes it, so the cluster's CTAs
// take the same way.
// What bounds it: the chain of an iteration's phases, each a few dependent loads and FP64 divides
// deep, and the fetching of their code; so two CTAs share an SM (the second at 128 registers costs
// a scene alone 25% and lets twice as many scenes run).
__global__ void __launch_bounds__(LT, 2) k_newton_batch(const LoopArgs* scenes, int C) {
  extern __shared__ double2 dyn2[];
  __shared__ LoopShared S;
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)blockIdx.x % C, tid = (int)threadIdx.x;
  {
    const unsigned long long* from = reinterpret_cast<const unsigned long long*>(scenes + blockIdx.x / C);
    for (int k = tid; k < (int)(sizeof(LoopArgs) / 8); k += LT) S.args[k] = from[k];
  }
  __syncthreads();
  const LoopArgs& a = *reinterpret_cast<const LoopArgs*>(S.args);
  const int n = a.kry.n;
  Mailbox* const box = a.box;
  StepDev& D = box->step;
  int* const ds = box->dstat;
  const abd_params& P = a.gh.prm;
  const bool ground = P.ground_enabled && P.enable_vg, lead = rank == 0 && tid == 0;
  if (!D.run) return;  // (its step is done: written before this launch, or by the cluster's end below)
  int it = D.it;
  bool resume = D.resume != 0;  // (its list was made again: the solve is done)
  const bool unmade = *a.bad != 0;  // (no list: never, unless a capacity was short)
  bool stop = unmade || (ds[DS_STATUS] & kRerunMask) != 0;
  cl.sync();
  while (!stop) {
    list_gh_pass<true>(a.gh, rank, C);
    cl.sync();
    stop = (ds[DS_STATUS] & kRerunMask) != 0;
    if (rank == 0 && !stop)
      contact_scan(a.cap_pairs, a.gh.pair_cand, ds, a.gh.cap_contacts, a.gh.contacts, a.gh.contacts_by_pair,
                   a.gh.pair_active);
    cl.sync();
    if (stop) break;
    assemble::assemble_pairs<assemble::kAsmRef>(a.gh, rank, C, reinterpret_cast<XSum*>(dyn2));
    cl.sync();
    stop = (ds[DS_STATUS] & kRerunMask) != 0;
    if (stop) break;
    // the bodies' blocks; the last CTA makes the preconditioner's clusters beside them
    if (rank == C - 1) {
      precond::make_clusters<LT>(n, a.cap_cluster, a.gh.act_pairs, a.gh.cap_act, ds, a.tables, a.work);
    } else {
      for (int b = rank; b < n; b += C - 1) {
        body_gh_pass(a.body, b, S.body);
        __syncthreads();
      }
    }
    cl.sync();
    if (!resume) {
      precond::BigShared& B = *reinterpret_cast<precond::BigShared*>(dyn2);
      const int ncl = a.pre.ncl_dev[0], solo = a.pre.ncl_dev[1], multi = a.pre.ncl_dev[2];
      for (int e = 0; e < multi; ++e) precond::big_inverse<LT>(a.pre, B, a.pre.big[n - 1 - e], rank, C);
      for (int e = rank; e < solo; e += C) precond::big_inverse<LT>(a.pre, B, a.pre.big[e], 0, 1);
      for (int c = (C - 1 - rank) + C * (tid >> 5); c < ncl; c += C * (LT / 32)) {
        const int base = a.pre.cl_ptr[c];
        if (a.pre.cl_ptr[c + 1] - base == 1) precond::warp_inverse1(a.pre, c, a.pre.cl_body[base], tid & 31);
      }
      cl.sync();
      krylov::solve<true, false>(a.kry, reinterpret_cast<double*>(dyn2), S.red, C, rank);
    }
    ccd_phase(a.ccd, ground, rank, C);
    cl.sync();
    stop = (ds[DS_STATUS] & kRerunMask) != 0;
    if (stop) break;
    if (*a.bad) {  // the iteration left the list's region: the list is made again first
      if (lead) D.resume = D.again = 1;
      return;  // (D.run stays)
    }
    // the line search: as many trials at a time as the threads take in one round
    const unsigned long long key = *a.ls.toi_key;
    int K;
    const double al = ls::trial_from_toi(key, P.alpha_min, tid < kLsMax ? tid : 0, &K);
    if (tid < K) S.al[tid] = al;
    const int cnt = min(ds[DS_NECAND], a.ls.cap_ecand), m = cnt + (ground ? a.ls.V : 0) + n;
    const int G = min(K, max(1, C * LT / m));
    const double E0 = D.E0;
    for (int k0 = 0;; k0 += G) {
      const int g = min(G, K - k0);
      trials_phase(a.ls, S, k0, g, cnt, m, rank, C);
      cl.sync();
      if (tid < 32) {
        bool ok = false;
        double E1 = 0.0;
        if (tid < g) {
          E1 = xs_round(box->ls_energy[k0 + tid]);
          ok = ls::accepts(P, E0, E1, S.al[k0 + tid], box->dots[0]);
        }
        const unsigned found = __ballot_sync(0xffffffffu, ok);
        const int f = found ? __ffs((int)found) - 1 : g - 1;
        if (tid == f) S.e1 = E1;
        if (tid == 0) {
          S.first = k0 + f;
          S.count = found ? k0 + f + 1 : -(k0 + g);
        }
      }
      __syncthreads();
      if (S.count > 0 || k0 + g >= K) break;
    }
    const int count = S.count;
    const double alpha = S.al[S.first];
    if (count > 0)
      for (int b = rank * LT + tid; b < n; b += C * LT)
        update_body_dofs(b, a.ccd.A, a.ccd.p, a.ccd.dq, alpha, const_cast<double*>(a.ccd.A),
                         const_cast<double*>(a.ccd.p), a.Ak, a.pk);
    const bool done = count < 0 || box->dots[1] < P.tol || it + 1 >= P.max_iter;
    clear_gh(ds, a.gh.pair_cand, a.cap_pairs, rank * LT + tid, C * LT);
    if (lead) {
      D.ls += count > 0 ? count : -count;
      D.E1 = S.e1;
      D.alpha = alpha;
      D.toi = key ? __longlong_as_double((long long)~key) : 1.0;
      D.resume = 0;
      D.it = it + 1;
      if (done) D.run = 0;
      if (count < 0) atomicOr(&ds[DS_STATUS], ST_LS_MORE);
    }
    ++it;
    resume = false;
    if (done) return;
    cl.sync();
  }
  if (lead) {  // a list was short: the step is made again
    D.it = it + 1;
    D.run = 0;
    if (unmade && !(ds[DS_STATUS] & kRerunMask)) atomicOr(&ds[DS_STATUS], ST_LS_MORE);
  }
}

// A round's end: another one while a scene's iteration left its list's region (and one can be due, as
// in k_round_end)
__global__ void __launch_bounds__(128) k_batch_end(const LoopArgs* scenes, int n, cudaGraphConditionalHandle h) {
  int more = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    Mailbox* const box = scenes[i].box;
    if (!box->step.run) continue;
    if (another_round(box->step.rounds, scenes[i].gh.prm.max_iter)) {
      more = 1;
    } else {
      box->step.run = 0;
      box->dstat[DS_STATUS] |= ST_LS_MORE;
    }
  }
  more = __syncthreads_or(more);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, more ? 1u : 0u);
}

constexpr size_t kLoopSmem = std::max(sizeof(precond::BigShared), (size_t)assemble::kRefSmem);
// a CTA's share of at most kLoopBodies bodies, plus its last cluster's members
static_assert((4 * 8 * 12 + sizeof(krylov::PosInfo)) * (kLoopBodies / kLoopLeast + kMaxCluster) <= kLoopSmem,
              "the solve's vectors fit");

cudaError_t loop_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int scenes, int C, cudaStream_t st) {
  cfg.gridDim = dim3(scenes * C);
  cfg.blockDim = dim3(LT);
  cfg.dynamicSmemBytes = kLoopSmem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaSuccess;
}

}  // namespace

// The kernel's attributes, and the most CTAs of its clusters (0: none fits): found once per device
cudaError_t prepare_newton_batch(Sim& s) {
  static std::mutex m;
  static std::map<int, int> known;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(m);
  const auto at = known.find(dev);
  if (at == known.end()) {
    e = cudaFuncSetAttribute(k_newton_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLoopSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_newton_batch, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    int c = kLoopCtas;
    for (; c >= kLoopLeast; c /= 2) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute la[1];
      loop_config(cfg, la, 1, c, 0);
      int k = 0;
      if (cudaOccupancyMaxActiveClusters(&k, k_newton_batch, &cfg) == cudaSuccess && k > 0) break;
      (void)cudaGetLastError();
    }
    known[dev] = c < kLoopLeast ? 0 : c;
  }
  s.max_loop_ctas = known[dev];
  return cudaSuccess;
}

bool batch_loop_takes(const Sim& s, int scenes) {
  return s.prm.solver == 1 && !s.prm.ipc_full && !(s.prm.friction_mu > 0.0) && s.max_loop_ctas > 0 &&
         s.n <= kLoopBodies && (long long)s.V + s.E <= std::max((long long)kLoopPrims, (long long)kLoopShare * scenes);
}

// As many CTAs for a scene as make up to twice what the GPU holds at a time: the largest scenes come
// first and take the longest, and the small ones that wait run as others end.  Five steps of 48
// scenes: 28.6 ms with 4 CTAs each (all resident), 20.8 with 8, 24.2 with 16.
int batch_loop_ctas(const Sim& s, int scenes) {
  int c = kLoopLeast;
  while (2 * c <= s.max_loop_ctas && 2 * c * scenes <= 2 * kLoopSlots) c *= 2;
  return c;
}

size_t batch_loop_bytes() { return sizeof(LoopArgs); }

void batch_loop_args(Sim& s, const abd_states& st, int C, void* host) {
  LoopArgs a;
  size_t smem = 0;
  a.gh = narrow_args(s, NARROW_GH, st.A, st.p, nullptr, nullptr, nullptr, nullptr, nullptr);
  a.body = body_args(s, &st, st.A, st.p, nullptr, nullptr);
  a.pre = solver_args(s);
  a.kry = krylov_args(s, s.dq, true, C, &smem);
  a.ccd = ccd_args(s, st);
  a.ls = ls_args(s, st, st.A, st.p, true);
  a.tables = cluster_tables_at(s.cl_tab, s.n);
  a.work = s.cl_work;
  a.cap_cluster = cluster_cap(s);
  a.cap_pairs = s.cap_pairs;
  a.box = s.box;
  a.bad = s.dint + kListBad;
  a.Ak = st.Ak;
  a.pk = st.pk;
  std::memcpy(host, &a, sizeof(a));
}

cudaError_t batch_newton(cudaStream_t st, const void* args, int scenes, int C) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  loop_config(cfg, at, scenes, C, st);
  return cudaLaunchKernelEx(&cfg, k_newton_batch, static_cast<const LoopArgs*>(args), C);
}

cudaError_t batch_round_end(cudaStream_t st, const void* args, int scenes, cudaGraphConditionalHandle h_round) {
  k_batch_end<<<1, 128, 0, st>>>(static_cast<const LoopArgs*>(args), scenes, h_round);
  return cudaGetLastError();
}

}  // namespace abd
