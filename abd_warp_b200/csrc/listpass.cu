// The device loop's kept candidate list.
//
// In the reference every Newton iteration culls from scratch (abd.py:170-207, 226-280): body
// boxes, body pairs and tree walks for the contacts at the iterate, and again, swept, for the CCD
// bound.  But the DOFs move little from one iteration to the next, and a pair that no pass can use
// can be left out of all of them.  So the step keeps a list of every PT / EE pair whose boxes
// meet when each body's DOFs range over a region: a segment of DOFs, widened by a displacement
// (the skin) on every axis.  While the iterates and the Newton steps stay inside that region, a
// pass only evaluates the list's candidates, with the reference's own culling predicate at its own
// DOFs, so every result is the one a full culling gives.  Each body's displacement is checked
// before a pass uses the list; a body that leaves the region has the list made again.
//
// What it saves: an iteration of the 1024-body pile made two broad phases with body bounds from
// 333k vertices (36 us), the pair lists (12 us), a chunk filter and tree walks (45 us), and went
// through four conditional nodes; 264 us, and 151 us with the list.  The list is made about once
// in one to four steps (ten iterations each), in 55 to 110 us; 64 piled-up spheres, whose Newton
// steps are long, make it every fourth iteration.
//
// The skin follows the scene (from list to list: the DOFs are checked against the one that the list in
// use was made with).  It doubles when a step's iteration asks for a list while the list is short
// (k_round_begin): the new one is four to five times as long, which the GPU still takes in a round or
// two, a candidate a thread (a pass over 65k candidates takes about as long as one over 10k).  (Doubled
// only for the list after that, the same step often asked again: 512 scenes stepped together went
// through a third round, 20.0 ms a step against 19.3, and 16 spheres' ten steps and back took 91 ms
// against 87.)  It halves when the list is long, and the next step makes the list again.  A list that
// outgrows its capacity and is long for its scene is not given the memory: the step starts again with
// half the skin, the most it may have from then on (else the rerun would double it as the run did),
// down to the least; only a list that this does not shorten gets a larger buffer.  With 65k and 262k
// candidates as the bounds the list of 16 spheres alternated between the two, and where many scenes
// share the GPU long lists cost as much as they are long: 48 scenes of four spheres with 2,562
// vertices took 24.1 ms a step, 22.0 with these bounds, 21.4 without a list.
//
// The skin is counted in units of dhat, or of 1/64 of the bodies' half extent where that is less: with
// dhat in place of it, 28 bodies of 0.2 m with dhat = 60 mm made lists of 20 GB and took 340 ms a step
// (2.2 ms without a list; 1.3 now).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "abd_listccd.cuh"

namespace abd {

using ccd::CcdArgs;

namespace {

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

constexpr double kSkinMin = 1.0;                          // in skin units (skin_unit)

// The list's region around the step: its segment runs from the iterate q to q - dq when an
// iteration asked for the list (its solve is done), else, at the step's start, to the prediction
// q~ that the first Newton iteration aims at (fixed bodies stay).  One thread per body: the
// segment's ends, their FP32 copies for the traversal, and the box that holds the body's box over
// the region.  Thread 0 also clears the counters of the traversal and of a GH pass that will be
// made again (its energy, its friction contacts).
__global__ void k_region(int n, abd_params P, abd_states st, const double* dq, const int* fixed, const Box* body_rest,
                         const double* skin, double* reg, float* fdof, Box* body_sup, int* chunk_count, Mailbox* box,
                         int friction) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = b; i < 256; i += gridDim.x * blockDim.x) (&box->prof[0][0])[i] = 0;
  if (b == 0) {
    *chunk_count = 0;
    box->dstat[DS_NLIST] = 0;
    if (box->step.it == 0) {
      xs_zero(box->energy);
      if (friction) box->dstat[DS_NFRIC] = 0;
    }
  }
  if (b >= n) return;
  double R[12], S[12];
  load_dofs(st.A, st.p, b, R);
  if (box->step.resume) {
    dofs_at(st.A, st.p, dq, b, 1.0, S);
  } else if (fixed[b]) {
#pragma unroll
    for (int k = 0; k < 12; ++k) S[k] = R[k];
  } else {
    tilde_of(P, st, b, S, S + 9);
  }
  float f[24];
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    reg[24 * (size_t)b + k] = R[k];
    reg[24 * (size_t)b + 12 + k] = S[k];
    f[k] = (float)R[k];
    f[12 + k] = (float)S[k];
  }
#pragma unroll
  for (int k = 0; k < 24; ++k) fdof[24 * (size_t)b + k] = f[k];
  store_box(&body_sup[b], affine_box2(load_box(&body_rest[b]), f, f + 12,
                                      __double2float_ru(0.5 * P.dhat) + __double2float_ru(*skin)));
}

// The list is made (unless a capacity was short: the step is run again): it may be used while the DOFs
// stay within its own skin, and the skin of the next one follows from it.  Also the traversal's time (kernel profiling).
// unit: of the skin; very_long: candidates
__global__ void k_list_made(Mailbox* box, int* bad, double* dpar, double unit, int cap_list, int very_long,
                            int prof_bytes) {
  StepDev& S = box->step;
  const double skin = dpar[kParSkinNext];
  if (S.t1 > S.t0 && S.t0 != ~0ULL) {
    S.prof_ns += S.t1 - S.t0;
    ++S.prof_n;
    if (prof_bytes) {
      // the weights of kProfBytes (bytes per counted access)
      const double w[PF_N] = {24.0, 36.0, 140.0, 36.0, 36.0, 36.0, 16.0};
      for (int row = 0; row < 32; ++row)
        for (int c = 0; c < PF_N; ++c) S.prof_bytes += w[c] * (double)box->prof[row][c];
    }
  }
  S.t0 = ~0ULL;
  S.t1 = 0ULL;
  if (box->dstat[DS_STATUS] & kRerunMask) {
    const double need = (double)(unsigned)box->dstat[DS_NLIST], last = dpar[kParListNeed];
    if (!(box->dstat[DS_STATUS] & ST_LIST_OVERFLOW)) return;
    dpar[kParListNeed] = need;
    // (a list that half the skin left as long is long for the segment's sake)
    if (need > (double)very_long && skin > kSkinMin * unit && !(last > 0.0 && need > 0.75 * last)) {
      // (for good: a rerun that doubled its displacement again would end where this one did)
      dpar[kParSkinNext] = dpar[kParSkinMost] = fmax(0.5 * skin, kSkinMin * unit);
      S.shrunk = 1;  // (the host does not grow the list)
    }
    return;
  }
  *bad = 0;
  dpar[kParListNeed] = 0.0;
  ++S.lists;
  const int m = min(box->dstat[DS_NLIST], cap_list);
  dpar[kParSkin] = skin;
  if (m > kListLong) dpar[kParSkinNext] = fmax(0.5 * skin, kSkinMin * unit);
}

// Blocks [0, G): the list's candidates, one thread each; blocks [G, G + Gb): one thread per body;
// blocks [G + Gb, ...): with vertex-ground contacts, a CTA per body for its times of impact.
__global__ void __launch_bounds__(128) k_list_ccd(const __grid_constant__ CcdArgs a, int G, int Gb) {
  const int* ds = a.box->dstat;
  if (ds[DS_STATUS] & kRerunMask) return;
  const int bx = (int)blockIdx.x;
  if (bx < G) {
    const int n = min(ds[DS_NLIST], a.cap_list);
    for (int i = bx * 128 + threadIdx.x; i < n; i += G * 128) ccd::candidate(a, i);
  } else if (bx < G + Gb) {
    ccd::body(a, (bx - G) * 128 + (int)threadIdx.x);
  } else {
    ccd::ground(a, bx - G - Gb);
  }
}

}  // namespace

cudaError_t list_build(Sim& s, const abd_states& st) {
  const bool fr = s.prm.friction_mu > 0.0;
  k_region<<<blocks(s.n, 128), 128, 0, s.stream>>>(s.n, s.prm, st, s.dq, s.fixed, s.body_rest,
                                                  s.dpar + kParSkinNext, s.reg, s.fdof, s.body_sup, s.chunk_act + s.nch, s.box,
                                                  fr ? 1 : 0);
  ++s.launches;
  cudaError_t e = list_pairs(s, fr ? s.fric_mask : nullptr);
  if (e == cudaSuccess) e = list_traverse(s);
  if (e != cudaSuccess) return e;
  const int very_long = (int)std::min((long long)INT_MAX, std::max((long long)kListLong, ((long long)s.V + s.E) / 2));
  k_list_made<<<1, 1, 0, s.stream>>>(s.box, s.dint + kListBad, s.dpar, skin_unit(s, s.prm.dhat), s.cap_list, very_long,
                                     s.prof_on == 2 ? 1 : 0);
  ++s.launches;
  return cudaGetLastError();
}

CcdArgs ccd_args(Sim& s, const abd_states& st) {
  CcdArgs a;
  a.prm = s.prm;
  a.n = s.n;
  a.A = st.A;
  a.p = st.p;
  a.dq = s.dq;
  a.x0 = s.x0;
  a.vbody = s.vbody;
  a.voff = s.voff;
  a.tris = s.tris;
  a.edges = s.edges;
  a.ext = s.ext;
  a.list = s.list;
  a.cap_list = s.cap_list;
  a.ecand = s.ecand;
  a.cap_ecand = s.cap_ecand;
  a.box = s.box;
  a.reg = s.reg;
  a.body_rest = s.body_rest;
  a.skin = s.dpar + kParSkin;
  a.bad = s.dint + kListBad;
  a.gh_q = s.gh_q;
  return a;
}

cudaError_t list_ccd(Sim& s, const abd_states& st) {
  const CcdArgs a = ccd_args(s, st);
  const int G = scene_grid(s, 128, kRedBlocks), Gb = (int)blocks(s.n, 128);
  const int Gv = s.prm.ground_enabled && s.prm.enable_vg ? s.n : 0;
  k_list_ccd<<<G + Gb + Gv, 128, 0, s.stream>>>(a, G, Gb);
  ++s.launches;
  return cudaGetLastError();
}

}  // namespace abd
