// The step's Newton iterations as a device loop (abd_step with newton_loop = 0).
//
// AffineBodySimulator.step (abd/abd.py:212-276) iterates gradient / Hessian, linear solve, CCD
// bound and backtracking line search until g.g < tol or max_iter iterations.  Run from the host,
// every iteration waits for the device twice: to read the line search's energies and to check
// the passes' list capacities.  Here one CUDA graph holds the whole step: a WHILE node over
// rounds, each making the kept candidate list when it has to be made (an IF node; listpass.cu)
// and then running Newton iterations in a nested WHILE node: the GH pass, the preconditioner, the
// Krylov solve, the CCD pass, the line search's trials, and the end, which accepts a trial,
// updates the DOFs and makes the convergence test.  A conditional node costs 4 to 6 us even when
// its body does not run, so an iteration holds none: after a capacity shortfall its kernels
// return at once, and the loop ends.  The host launches the graph once per step and reads the
// step's counters with one copy.  When a list overflowed, the states are left as they were, and
// the host grows the list and runs the step again from its start (the warm start dq is restored
// from the copy the graph made).
//
// The kernels here keep the host loop's arithmetic, so both loops give the same bits: the
// energies are the exact sums rounded once on the device (the host rounds the same sums with
// the same rule), the Armijo test is evaluated in the same order, and the iteration counts
// follow the same rules.
#include <cuda_runtime.h>

#include "abd_ghpass.cuh"
#include "abd_lsterms.cuh"

namespace abd {

static_assert(PF_N == 7 && kProfBytes[0] == 24.0 && kProfBytes[1] == 36.0 && kProfBytes[2] == 140.0 &&
                  kProfBytes[3] == 36.0 && kProfBytes[4] == 36.0 && kProfBytes[5] == 36.0 && kProfBytes[6] == 16.0,
              "k_list_made's copy of the profiling weights");

namespace {

// The step's start, one thread per body: q <- q0 and the line-search origin (Ak, pk) <- q0
// (abd.py:124-128), the warm start dq kept for a rerun, and whether q0 and the prediction q~ stay
// in the kept list's region; thread 0 clears the step's counters and enters the round loop.
__global__ void k_step_begin(Mailbox* box, cudaGraphConditionalHandle h, int n, abd_states st, const double* dq,
                             double* dq_save, abd_params P, const int* fixed, const double* reg, const Box* body_rest,
                             const double* dpar, int* bad) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  const double skin = dpar[kParSkin];
  if (b < n) {
    for (int k = 0; k < 9; ++k) st.A[9 * b + k] = st.Ak[9 * b + k] = st.A0[9 * b + k];
    for (int k = 0; k < 3; ++k) st.p[3 * b + k] = st.pk[3 * b + k] = st.p0[3 * b + k];
    for (int k = 0; k < 12; ++k) dq_save[12 * b + k] = dq[12 * b + k];
    double M[12];
    load_dofs(st.A0, st.p0, b, M);
    const Box R = load_box(&body_rest[b]);
    const double* g = reg + 24 * (size_t)b;
    bool in = in_region(g, M, R, skin);
    if (in && !fixed[b]) {
      tilde_of(P, st, b, M, M + 9);
      in = in_region(g, M, R, skin);
    }
    if (!in) *bad = 1;
  }
  if (b != 0) return;
  if (dpar[kParSkinNext] < skin) *bad = 1;  // (the list was long)
  xs_zero(box->energy);
  StepDev& S = box->step;
  S.it = S.lin = S.ls = 0;
  S.n_pt = S.n_ee = S.n_vg = S.n_ij = S.n_active = 0;
  S.resume = S.again = S.lists = S.rounds = S.shrunk = 0;
  S.run = 1;
  S.E0 = S.E1 = S.alpha = 0.0;
  S.toi = 1.0;
  S.t0 = ~0ULL;
  S.t1 = 0ULL;
  S.prof_ns = S.prof_n = 0ULL;
  S.prof_bytes = 0.0;
  cudaGraphSetConditional(h, 1u);
}

// A round's start: the kept list is made when it has to be (for an iteration that left the region of a
// short one, with twice the displacement: listpass.cu), then Newton iterations run.
// shared: the scene's iterations are in its batch's kernel (newton_batch.cu), if it still runs.
__global__ void k_round_begin(Mailbox* box, const int* bad, double* dpar, int* cand, int cap_pairs,
                              cudaGraphConditionalHandle h_list, cudaGraphConditionalHandle h_newton, int shared) {
  int* const ds = box->dstat;
  const bool run = !shared || box->step.run;
  if (threadIdx.x == 0) {
    box->step.again = 0;
    if (run) ++box->step.rounds;
    if (run && *bad && box->step.resume && ds[DS_NLIST] <= kListShort)
      dpar[kParSkinNext] = fmin(2.0 * dpar[kParSkinNext], dpar[kParSkinMost]);
    cudaGraphSetConditional(h_list, run && *bad ? 1u : 0u);
    if (!shared) cudaGraphSetConditional(h_newton, 1u);
  }
  if (run) clear_gh(ds, cand, cap_pairs, threadIdx.x, blockDim.x);
}

// A round's end: another one when an iteration left the list's region (and one can be due).
__global__ void k_round_end(Mailbox* box, int max_iter, cudaGraphConditionalHandle h) {
  bool more = box->step.again && !(box->dstat[DS_STATUS] & kRerunMask);
  if (more && !another_round(box->step.rounds, max_iter)) {
    box->dstat[DS_STATUS] |= ST_LS_MORE;  // (never; the host finishes the step)
    more = false;
  }
  cudaGraphSetConditional(h, more ? 1u : 0u);
}

// A Newton iteration's end.  Every CTA makes the backtracking line search's decision (abd.py:146-160)
// over the trials of the batch (k_ls_eval's step lengths alpha, alpha / 2, ... to the first below
// alpha_min): the first trial that passes the Armijo test, or the first below alpha_min, is taken,
// as the sequential search takes it; its first warp rounds the trials' exact energies, a lane
// each.  Then one thread per body: the accepted step q <- q - alpha dq, also into the line-search
// origin (Ak, pk) (update_qk, abd.py:154-157); thread 0: the step's counters and the convergence
// test (abd.py:259-271: g.g < tol on the gradient the iteration solved with, or max_iter
// iterations); and the counters of the next GH pass.
// An iteration that left the kept list's region ends the loop without all that: its list is made
// again (listpass.cu) and the iteration goes on after its solve.  A list overflow, or a batch whose
// trials all fail while none is below alpha_min (ST_LS_MORE), also ends it (the step is then
// made again from its start).
__global__ void k_newton_end(Mailbox* box, const double* dpar, const int* bad, abd_params P,
                             cudaGraphConditionalHandle h, int n, abd_states st, const double* dq, int* cand,
                             int cap_pairs) {
  StepDev& S = box->step;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (box->dstat[DS_STATUS] & kRerunMask) {
    if (b == 0) {
      ++S.it;
      cudaGraphSetConditional(h, 0u);
    }
    return;
  }
  if (*bad) {
    if (b == 0) {
      S.resume = S.again = 1;
      cudaGraphSetConditional(h, 0u);
    }
    return;
  }
  __shared__ int first, count;
  __shared__ double e1;
  if (threadIdx.x < 32) {
    const int K = (int)dpar[kParK], k = (int)threadIdx.x;
    bool ok = false;
    double E1 = 0.0;
    if (k < K) {
      const double al = dpar[kParAlpha + k], E0 = S.E0;
      E1 = xs_round(box->ls_energy[k]);
      ok = ls::accepts(P, E0, E1, al, box->dots[0]);
    }
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    const int f = m ? __ffs((int)m) - 1 : K - 1;
    if (k == f) e1 = E1;
    if (k == 0) {
      first = f;
      count = m ? f + 1 : -K;
    }
  }
  __syncthreads();
  const double alpha = dpar[kParAlpha + first];
  if (b < n && count > 0) update_body_dofs(b, st.A, st.p, dq, alpha, st.A, st.p, st.Ak, st.pk);
  clear_gh(box->dstat, cand, cap_pairs, b, gridDim.x * blockDim.x);
  if (b != 0) return;
  S.ls += count > 0 ? count : -count;
  S.E1 = e1;
  S.alpha = alpha;
  double toi = 1.0;
  if (const unsigned long long key = box->toi_key) toi = __longlong_as_double((long long)~key);
  S.toi = toi;
  S.resume = 0;
  ++S.it;
  if (count < 0) atomicOr(&box->dstat[DS_STATUS], ST_LS_MORE);
  cudaGraphSetConditional(h, count > 0 && !(box->dots[1] < P.tol) && S.it < P.max_iter ? 1u : 0u);
}

// The adjoint step's right-hand side a = qb + qdb / dt (fixed bodies: 0), into g
__global__ void k_adjoint_rhs(int n, const double* qb, const double* qdb, double dt, const int* fixed, double* g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 12 * n) return;
  g[i] = fixed[i / 12] ? 0.0 : qb[i] + qdb[i] / dt;
}

// From lambda = H^-1 a: t = M lambda, qb_t = t - qdb / dt, qdb_t = dt t (fixed bodies: 0);
// M = mass on p, I0 on the rows of A
__global__ void k_adjoint_out(int n, const double* lam, const double* mass, const double* I0, const double* qdb,
                              double dt, const int* fixed, double* qb_out, double* qdb_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 12 * n) return;
  const int b = i / 12;
  if (fixed[b]) {
    qb_out[i] = 0.0;
    qdb_out[i] = 0.0;
    return;
  }
  const double t = ((i % 12) < 3 ? mass[b] : I0[b]) * lam[i];
  const double d = qdb[i];
  qb_out[i] = t - d / dt;
  qdb_out[i] = dt * t;
}

}  // namespace

cudaError_t adjoint_rhs(Sim& s, const double* qb, const double* qdb) {
  k_adjoint_rhs<<<(12 * s.n + 255) / 256, 256, 0, s.stream>>>(s.n, qb, qdb, s.prm.dt, s.fixed, s.g);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t adjoint_out(Sim& s, const double* lam, const double* qdb, double* qb_out, double* qdb_out) {
  k_adjoint_out<<<(12 * s.n + 255) / 256, 256, 0, s.stream>>>(s.n, lam, s.mass, s.I0, qdb, s.prm.dt, s.fixed,
                                                             qb_out, qdb_out);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t step_begin(Sim& s, const abd_states& st, cudaGraphConditionalHandle h) {
  k_step_begin<<<(s.n + 127) / 128, 128, 0, s.stream>>>(s.box, h, s.n, st, s.dq, s.dq_save, s.prm, s.fixed, s.reg,
                                                        s.body_rest, s.dpar, s.dint + kListBad);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t round_begin(Sim& s, cudaGraphConditionalHandle h_list, cudaGraphConditionalHandle h_newton, bool shared) {
  k_round_begin<<<1, shared ? 128 : 1024, 0, s.stream>>>(s.box, s.dint + kListBad, s.dpar, s.pair_cand, s.cap_pairs,
                                                        h_list, h_newton, shared ? 1 : 0);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t round_end(Sim& s, cudaGraphConditionalHandle h_round) {
  k_round_end<<<1, 1, 0, s.stream>>>(s.box, s.prm.max_iter, h_round);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t newton_end(Sim& s, const abd_states& st, cudaGraphConditionalHandle h) {
  k_newton_end<<<(s.n + 127) / 128, 128, 0, s.stream>>>(s.box, s.dpar, s.dint + kListBad, s.prm, h, s.n, st, s.dq,
                                                        s.pair_cand, s.cap_pairs);
  ++s.launches;
  return cudaGetLastError();
}

}  // namespace abd
