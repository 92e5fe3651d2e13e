// Parts of the GH pass: its candidates, the contacts by pair, the bodies' blocks.
#pragma once

#include <cuda_runtime.h>

#include "abd_narrow.cuh"
#include "abd_warpsum.cuh"

namespace abd {

// The counters of a GH pass, cleared before it (by threads t of stride s).  Not the coupled pairs
// (DS_NACTP): a solve after the step forms its clusters from the last pass's.
__device__ inline void clear_gh(int* ds, int* pair_cand, int cap_pairs, int t, int s) {
  const int np = min(ds[DS_NPAIRS], cap_pairs);
  for (int p = t; p < np; p += s) pair_cand[4 * p + 1] = 0;
  if (t == 0) ds[DS_PT_COUNT] = ds[DS_EE_COUNT] = ds[DS_VG_COUNT] = ds[DS_ACTIVE] = ds[DS_NCONTACT] = 0;
}

// contacts into their pair's segment, thread k taking contacts k, k + stride, ... (the order
// inside a segment does not matter: the assembly sums exactly)
__device__ inline void scatter_contacts(int k, int stride, int cap_contacts, const int4* in,
                                        int* pair_cand, int4* out, const int* dstat) {
  for (const int m = min(dstat[DS_NCONTACT], cap_contacts); k < m; k += stride) {
    const int4 c = in[k];
    out[pair_cand[4 * c.x] + atomicAdd(&pair_cand[4 * c.x + 2], 1)] = c;
  }
}

// Lists of at most this many contacts are scattered by the scan's CTA itself
constexpr int kScanScatter = 16384;

// One CTA: per-pair offsets of the contact lists (pair_cand[4p] = offset, [4p+1] = count,
// [4p+2] = fill cursor), the pairs' active counts, and the pairs that have contacts (in any order:
// pair_cand[4k+3], k < DS_NASM), which the assembly takes; with `in` (a list of at most kScanScatter), then the contacts into
// their segments.
__device__ inline void contact_scan(int cap_pairs, int* pair_cand, int* dstat, int cap_contacts, const int4* in, int4* out,
                                    int* pair_active) {
  const int np = min(dstat[DS_NPAIRS], cap_pairs);
  __shared__ int sh[33];
  __shared__ int carry, nasm;
  if (threadIdx.x == 0) carry = nasm = 0;
  const int T = (int)blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c0 = 0; c0 < np; c0 += T) {
    const int p = c0 + (int)threadIdx.x;
    const int v = p < np ? pair_cand[4 * p + 1] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
      int acc = carry;
      for (int w = 0; w < T / 32; ++w) {
        const int t = sh[w];
        sh[w] = acc;
        acc += t;
      }
      sh[32] = acc;
    }
    __syncthreads();
    if (p < np) {
      pair_cand[4 * p] = sh[warp] + x - v;
      pair_cand[4 * p + 2] = 0;
      pair_active[p] = v;
      if (v) pair_cand[4 * atomicAdd(&nasm, 1) + 3] = p;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = sh[32];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    dstat[DS_NASM] = nasm;
    dstat[DS_ACTIVE] += carry;  // (less the friction contacts: k_fric_pairs)
  }
  // (the barrier above makes the CTA's offsets and cleared cursors visible to all its threads)
  if (in) scatter_contacts(threadIdx.x, T, cap_contacts, in, pair_cand, out, dstat);
}

// does vertex v take part in the vertex-ground terms (culling.py:64-82)?  bb: its body box
__device__ inline bool vg_candidate_of(const abd_params& P, const Box& bb, const double* y0, const double* y1, int v) {
  return vg_box_test(P, bb, point_box(y0, y1, v, (float)P.dhat));
}

// One candidate's barrier energy at positions xs: the reference's model (ipcsk/energy.py:9-48)
// or, with ipc_full, the full model (its rest positions scale the edge-edge mollifier)
template <bool REF = false>
__device__ inline double candidate_energy(const NarrowArgs& a, int type, const int ids[4], const d3 xs[4]) {
  if constexpr (!REF) {
    if (a.prm.ipc_full) {
      double r[12];
#pragma unroll
      for (int k = 0; k < 12; ++k) r[k] = __ldg(&a.x0[3 * ids[k / 3] + k % 3]);
      return full_contact_energy(type, xs, r, a.prm);
    }
  }
  return contact_energy(type, xs, a.prm);
}

// Lagged friction (friction_mu > 0, with the full model; Li et al. 2020, section 5): at the
// step's first GH pass every contact within dhat fixes its lagged quantities (the header's
// friction_lag at the step-start positions xs) and its body pair joins the step's pair lists;
// returns the contact's friction potential there (mu lambda eps / 3: no displacement yet).
__device__ inline double friction_lag_contact(const NarrowArgs& a, int kind, const int ids[4], const d3 xs[4]) {
  double x12[12], r12[12];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    x12[3 * k] = xs[k].x, x12[3 * k + 1] = xs[k].y, x12[3 * k + 2] = xs[k].z;
    for (int m = 0; m < 3; ++m) r12[3 * k + m] = __ldg(&a.x0[3 * ids[k] + m]);
  }
  ipc::FrictionLag L;
  if (!ipc::friction_lag(kind, x12, r12, a.prm.d2hat, a.prm.kappa, SharedLog(), &L)) return 0.0;
  const int I = __ldg(&a.vbody[ids[0]]), J = __ldg(&a.vbody[ids[kind == 0 ? 1 : 2]]);
  const int pos = atomicAdd(&a.dstat[DS_NFRIC], 1);
  if (pos < a.cap_fric) {
    FricRec& f = a.fric[pos];
    for (int k = 0; k < 4; ++k) f.w[k] = L.w[k];
    for (int k = 0; k < 6; ++k) f.P[k] = L.P[k];
    f.lam = L.lambda;
    for (int k = 0; k < 12; ++k) f.xt[k] = x12[k];
    for (int k = 0; k < 4; ++k) f.ids[k] = ids[k];
    f.I = I;
    f.J = J;
    f.kind = kind;
  } else {
    atomicOr(&a.dstat[DS_STATUS], ST_FRIC_OVERFLOW);
  }
  if (I != J) {
    atomicOr(&a.fric_mask[(size_t)I * a.W + (J >> 5)], 1u << (J & 31));
    atomicOr(&a.fric_mask[(size_t)J * a.W + (I >> 5)], 1u << (I & 31));
  }
  return ipc::friction_d(L, x12, x12, a.prm.friction_mu, a.prm.friction_epsv * a.prm.dt);
}

// is a candidate an active contact?
template <bool REF = false>
__device__ inline bool gh_active(const NarrowArgs& a, int type, const d3 xs[4]) {
  Geo G;
  double d2;
  int fty;
  return !REF && a.prm.ipc_full ? full_d2(type, xs, &fty) < a.prm.d2hat : contact_active(type, xs, a.prm, &G, &d2);
}

// One candidate of the GH pass, c = (pair, type | swap << 1, primitive a, primitive b), its
// vertices ids at xs: counted
// by kind; when active (pt_ipc.py:13-22, 114; ee_ipc.py:13-23, 382) appended for the per-pair
// assembly and counted for its pair, and at the step's first GH pass (lag) its lagged friction
// is fixed.  With gh_energy its barrier energy joins the pass's exact energy (k_body_gh adds
// the bodies' terms: the GH pass then also gives the energy at its DOFs, the same sum as an
// energy pass there).
template <bool REF = false>
__device__ inline void gh_candidate(const NarrowArgs& a, const int4 c, const int ids[4], const d3 xs[4],
                                    bool with_energy, bool lag, int& cpt, int& cee, XSum& en) {
  const int type = c.y & 1;
  if (type == 0) ++cpt;
  else ++cee;
  if (with_energy) {
    const double e = candidate_energy<REF>(a, type, ids, xs);
    if (e != 0.0) xs_add(en, e);
  }
  if (gh_active<REF>(a, type, xs)) {
    const int pos = append_slot(&a.dstat[DS_NCONTACT]);
    if (pos < a.cap_contacts) a.contacts[pos] = c;
    else atomicOr(&a.dstat[DS_STATUS], ST_CONTACT_OVERFLOW);
    atomicAdd(&a.pair_cand[4 * c.x + 1], 1);
    if (!REF && lag) {
      const double e = friction_lag_contact(a, type, ids, xs);
      if (with_energy && e != 0.0) xs_add(en, e);
    }
  }
}

// the per-kind counts and the energy of a CTA's candidates into the pass's totals (every thread)
__device__ inline void gh_flush(const NarrowArgs& a, int cpt, int cee, XSum& en, bool with_energy) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cpt += __shfl_xor_sync(0xffffffffu, cpt, o);
    cee += __shfl_xor_sync(0xffffffffu, cee, o);
  }
  if (with_energy) xs_warp_sum(en);
  if ((threadIdx.x & 31) == 0) {
    if (cpt) atomicAdd(&a.dstat[DS_PT_COUNT], cpt);
    if (cee) atomicAdd(&a.dstat[DS_EE_COUNT], cee);
    long long* d = reinterpret_cast<long long*>(a.energy);
#pragma unroll
    for (int i = 0; i < kXD; ++i)
      if (en.d[i]) atomicAdd((unsigned long long*)&d[i], (unsigned long long)en.d[i]);
    if (en.flags) atomicOr((unsigned long long*)&d[kXD], (unsigned long long)en.flags);
  }
}

// the energy and the friction lag ride on the step's first GH pass
__device__ inline bool gh_with_energy(const NarrowArgs& a) {
  return a.gh_energy && (!a.energy_gate || *a.energy_gate == 0);
}
__device__ inline bool gh_lag(const NarrowArgs& a) { return a.fric_lag && (!a.energy_gate || *a.energy_gate == 0); }

// The GH pass of the device loop: the kept list's candidates at the DOFs (A, p), one thread per
// candidate.  The list holds every pair its culling can produce, so the pass needs no boxes, pairs
// or vertex positions of its own: a thread computes its four positions and applies the culling
// predicate (culling2.py:32-79, 213-227) as k_ls_eval does (linesearch.cu: the primitives' boxes;
// the body boxes only where a tie at the rounding boundary leaves them to decide).  CTA 0 also
// clears what the iteration's assembly, CCD pass and line search add to.
// Bound by its chain of dependent loads (candidate, vertices, bodies, DOFs): 8.7 us for the 71k
// candidates of the 1024-body pile, in place of 43 us (broad phase, pairs, and the scan of the
// candidates kept from the CCD pass).
// By CTA bx of nb.
template <bool REF = false>
__device__ __forceinline__ void list_gh_pass(const NarrowArgs& a, int bx, int nb) {
  const int T = (int)blockDim.x;
  if (bx == 0) {
    for (int i = threadIdx.x; i < kLsMax * (kXD + 1); i += T) reinterpret_cast<long long*>(a.ls_energy)[i] = 0;
    if (threadIdx.x == 0) {
      a.dstat[DS_NECAND] = 0;
      a.dstat[DS_NACTP] = 0;  // (the assembly appends them)
      *a.toi_key = 0;
    }
  }
  if (a.dstat[DS_STATUS] & kRerunMask) return;
  const int n = min(a.dstat[DS_NLIST], a.cap_list);
  const float dhf = (float)a.prm.dhat;
  const double dhh = 0.5 * a.prm.dhat;
  int cpt = 0, cee = 0;
  XSum en;
  xs_zero(en);
  const bool with_energy = gh_with_energy(a), lag = !REF && gh_lag(a);
  for (int k = bx * T + (int)threadIdx.x; k < n; k += nb * T) {
    const int4 c = a.list[k];
    const int type = c.x;
    int ids[4];
    cand_vertices(a, type, c.y, c.z, ids);
    const int I = __ldg(&a.vbody[ids[0]]), J = __ldg(&a.vbody[ids[type == 0 ? 1 : 2]]);
    double MI[12], MJ[12];
    load_dofs(a.A, a.p, I, MI);
    load_dofs(a.A, a.p, J, MJ);
    d3 xs[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) xs[q] = position_of((q == 0 || (type == 1 && q == 1)) ? MI : MJ, a.x0, ids[q]);
    if (type == 0) {
      if (!overlap(point_box_at(xs[0], dhf), tri_box_at(xs[1], xs[2], xs[3]))) continue;
      if (!overlap(edge_box_at(xs[0], xs[0], dhh), tri_box_dilated(xs[1], xs[2], xs[3], dhh))) {
        // the body boxes decide; only the step's first pass needs to know of an inactive pair
        if (!with_energy && !gh_active<REF>(a, type, xs)) continue;
        if (!overlap(body_box_under(a.voff, a.x0, I, MI, nullptr, dhh), body_box_under(a.voff, a.x0, J, MJ, nullptr, dhh)))
          continue;
      }
    } else if (!overlap(edge_box_at(xs[0], xs[1], dhh), edge_box_at(xs[2], xs[3], dhh))) {
      continue;
    }
    const int swap = (type == 0 && I > J) ? 1 : 0;
    gh_candidate<REF>(a, make_int4(c.w, type | (swap << 1), c.y, c.z), ids, xs, with_energy, lag, cpt, cee, en);
  }
  gh_flush(a, cpt, cee, en, with_energy);
}

struct BodyArgs {
  abd_params prm;
  int n;
  const int* voff;
  const double *x0, *mass, *I0;
  const int* fixed;
  abd_states st;
  const double *A, *p, *y, *y1;  // (y null: the positions at (A, p))
  const Box* body_box;
  const int *row_ptr, *adj_pair, *pair_active;
  const int2* ij;
  const double *pdiag, *pgrad;
  double *diag, *g;
  int* dstat;
  int* vg_list;
  int cap_vg;
  XSum* energy;  // or null; the pass's exact energy (GH: inertia + vertex-ground terms, added here)
  const int* energy_gate;  // device loop: the energy is summed only while this counter is 0
  int exact;     // the adjoint's system: the vertex-ground Hessian with its 2 B' term
  int* highlight;  // [n] or null: the body takes part in an active PT / EE / vertex-ground contact
};

__device__ inline void tilde(const BodyArgs& a, int b, double At[9], double pt[3]) {
  tilde_of(a.prm, a.st, b, At, pt);
}
__device__ inline bool vg_candidate(const BodyArgs& a, const Box& bb, const double* y0, const double* y1, int v) {
  return vg_candidate_of(a.prm, bb, y0, y1, v);
}

// Shared memory of a body's pass: the digits of its exact sums (abd_warpsum.cuh) -- the
// vertex-ground gradient (4 y-components) and Hessian (4x4 yy-components), [20] its energy
// (vertex-ground barriers of every body, inertia + orthogonality of a free one)
constexpr int kBodySums = 21;
struct BodyShared {
  int sum[kBodySums][kDSlots];
  unsigned long long ymin;  // without boxes: the body's lowest vertex (as a max key)
  int vg_hit;               // an active vertex-ground contact (d^2 < dhat^2)
};
constexpr int kBodyRoom = 1 << 15;  // vertices (two terms of a sum each) between folds
static_assert(2 * (kBodyRoom + 1024) + 64 < kDTerms, "the terms between two folds fit the counters");

// Body b by a CTA of at least 160 threads: its diagonal block, gradient, vertex-ground terms,
// energy and contact flag.
// What bounds it: a chain of short phases over a body's vertices and pairs.  The vertex-ground sums
// were 64-bit shared atomics (compare-and-swap loops; 20 entries a vertex, all vertices on the
// same ones): 27 bodies on the ground plane took 19.1 us, with 32-bit digit counters 15.9 us.
__device__ __forceinline__ void body_gh_pass(const BodyArgs& a, int b, BodyShared& S) {
  const int t = threadIdx.x, T = (int)blockDim.x;
  XSum* const energy = (a.energy && (!a.energy_gate || *a.energy_gate == 0)) ? a.energy : nullptr;
  const bool fixed = a.fixed[b] != 0;
  const double dt = a.prm.dt, ks = a.prm.stiffness;
  const double* A = a.A + 9 * b;
  double val = 0.0;
  const bool vg_any = a.prm.ground_enabled && a.prm.enable_vg, vg_on = vg_any && !fixed;
  for (int e = t; e < kBodySums * kDSlots; e += T) (&S.sum[0][0])[e] = 0;
  if (t == 0) {
    S.vg_hit = 0;
    S.ymin = 0;
  }
  __syncthreads();
  if (energy && t == 128 && !fixed)
    ds_add(S.sum[20], inertia_energy(a.prm, a.st, a.mass, a.I0, b, a.A + 9 * b, a.p + 3 * b));
  const int v1 = a.voff[b + 1];
  double MB[12];
  if (vg_any && !a.y) {
    load_dofs(a.A, a.p, b, MB);
    unsigned long long k = 0;
    for (int v = a.voff[b] + t; v < v1; v += T) {
      const unsigned long long q = max_key(-position_of(MB, a.x0, v).y);
      k = q > k ? q : k;
    }
    if (k) atomicMax(&S.ymin, k);
    __syncthreads();
  }
  if (vg_any) {
    Box bb;
    if (a.y) bb = load_box(&a.body_box[b]);
    else bb.lo[1] = (float)(-key_value(S.ymin) - 0.5 * a.prm.dhat);  // (the only face the test reads)
    const bool low = (double)bb.lo[1] < 0.5 * a.prm.dhat + a.prm.ground;
    int cnt = 0;  // the culling's vertex-ground pairs, fixed bodies included (culling.py:54-82)
    for (int v0 = a.voff[b], seen = 0; low && v0 < v1; v0 += T, seen += T) {
      if (seen >= kBodyRoom) {
        __syncthreads();
        for (int k = t >> 5; k < kBodySums; k += T >> 5) ds_fold(S.sum[k]);
        __syncthreads();
        seen = 0;
      }
      const int v = v0 + t;
      if (v >= v1) continue;
      const d3 x = a.y ? mk(a.y[3 * v], a.y[3 * v + 1], a.y[3 * v + 2]) : position_of(MB, a.x0, v);
      if (!vg_box_test(a.prm, bb, point_box_at(x, (float)a.prm.dhat))) continue;
      ++cnt;
      const double d = x.y - a.prm.ground;
      if (d * d < a.prm.d2hat) S.vg_hit = 1;
      if (energy) {
        const double e = barrier(d * d, a.prm);
        if (e != 0.0) ds_add(S.sum[20], e);
      }
      if (!vg_on) continue;
      const double d2b = barrier_d2(d * d, a.prm), db = barrier_d1(d * d, a.prm);
#pragma unroll 1
      for (int e = 0; e < 16; ++e) {
        const int ii = e / 4, jj = e % 4;
        const double ti = ii ? a.x0[3 * v + ii - 1] : 1.0, tj = jj ? a.x0[3 * v + jj - 1] : 1.0;
        if (jj == 0) ds_add(S.sum[ii], ((d * 2.0) * ti) * db);
        ds_add(S.sum[4 + e], (((ti * tj) * d2b) * 4.0) * d * d);
        if (a.exact) ds_add(S.sum[4 + e], (ti * tj) * (2.0 * db));
      }
    }
    if (cnt) atomicAdd(&a.dstat[DS_VG_COUNT], cnt);
  }
  __syncthreads();
  if (energy && t < kDSlots) ds_to_limbs(S.sum[20], t, energy);
  // contact flags (abd.py:238): any active contact of the body's pairs, or vertex-ground
  if (a.highlight && t == 156) {
    int on = S.vg_hit;
    const int k1 = (a.dstat[DS_STATUS] & ST_PAIR_OVERFLOW) ? a.row_ptr[b] : a.row_ptr[b + 1];
    for (int k = a.row_ptr[b]; k < k1 && !on; ++k) on = a.pair_active[a.adj_pair[k]] > 0;
    a.highlight[b] = on;
  }
  if (t < 156) {
    if (!fixed) {
      double At[9], pt[3];
      tilde(a, b, At, pt);
      if (t < 144) {
        const int r = t / 12, c = t % 12, ii = r / 3, jj = c / 3, rr = r % 3, cc = c % 3;
        const double m = (ii != jj) ? 0.0 : (ii == 0 ? a.mass[b] : a.I0[b]);
        double dh = rr == cc ? m : 0.0;
        if (ii > 0 && jj > 0) {
          const int i = ii - 1, j = jj - 1;
          double h;
          if (i == j) {
            h = 0.0;
            for (int k = 0; k < 3; ++k) h += A[3 * k + rr] * A[3 * k + cc];
            const double ti = (A[3 * i] * A[3 * i] + A[3 * i + 1] * A[3 * i + 1] + A[3 * i + 2] * A[3 * i + 2]) - 1.0;
            h += (A[3 * i + rr] * A[3 * i + cc] + (rr == cc ? ti : 0.0));
          } else {
            const double tj = A[3 * j] * A[3 * i] + A[3 * j + 1] * A[3 * i + 1] + A[3 * j + 2] * A[3 * i + 2];
            h = A[3 * j + rr] * A[3 * i + cc] + (rr == cc ? tj : 0.0);
          }
          dh = dh + ((h * 4.0) * ks) * dt * dt;
        }
        val = dh;
      } else {
        const int k = t - 144, m = k / 3, comp = k % 3;
        if (m == 0) {
          val = 0.0 + (a.p[3 * b + comp] - pt[comp]) * a.mass[b];
        } else {
          const int i = m - 1;
          double gr = -A[3 * i + comp];
          for (int j = 0; j < 3; ++j) {
            const double dj = A[3 * i] * A[3 * j] + A[3 * i + 1] * A[3 * j + 1] + A[3 * i + 2] * A[3 * j + 2];
            gr = gr + dj * A[3 * j + comp];
          }
          gr = (gr * 4.0) * ks;
          gr = (dt * dt) * gr;
          val = gr + (A[3 * i + comp] - At[3 * i + comp]) * a.I0[b];
        }
      }
      // entry = inertia + vertex-ground terms + the pair contributions (adjacency order; the sum
      // is exact, so the order does not matter), rounded once
      XSum acc;
      xs_zero(acc);
      xs_add(acc, val);
      if (vg_on) {
        if (t < 144) {
          const int r = t / 12, c = t % 12;
          if (r % 3 == 1 && c % 3 == 1) ds_merge(acc, S.sum[4 + 4 * (r / 3) + c / 3]);
        } else if ((t - 144) % 3 == 1) {
          ds_merge(acc, S.sum[(t - 144) / 3]);
        }
      }
      // skipped when the pair lists of this pass overflowed (the host reruns the pass)
      const int k1 = (a.dstat[DS_STATUS] & ST_PAIR_OVERFLOW) ? a.row_ptr[b] : a.row_ptr[b + 1];
      for (int k = a.row_ptr[b]; k < k1; ++k) {
        const int pr = a.adj_pair[k];
        if (a.pair_active[pr] <= 0) continue;
        const int side = a.ij[pr].x == b ? 0 : 1;
        xs_add(acc, t < 144 ? a.pdiag[(size_t)pr * 288 + side * 144 + t] : a.pgrad[(size_t)pr * 24 + side * 12 + (t - 144)]);
      }
      val = xs_round(acc);
      if (!isfinite(val)) atomicOr(&a.dstat[DS_STATUS], ST_NAN);
    } else {
      val = (t < 144 && (t % 13) == 0) ? 1.0 : 0.0;
    }
    if (t < 144) a.diag[(size_t)b * 144 + t] = val;
    else a.g[(size_t)b * 12 + (t - 144)] = val;
  }
}

BodyArgs body_args(Sim& s, const abd_states* st, const double* A, const double* p, const double* y, const double* y1);

}  // namespace abd
