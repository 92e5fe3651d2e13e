// What the narrow passes (narrow.cu) and the pair assembly (assemble.cu) share: the arguments of
// a pass and the access to its candidates.
#pragma once

#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "abd_body.cuh"
#include "abd_geometry.cuh"

namespace abd {

struct NarrowArgs {
  int mode;
  abd_params prm;
  int n, cap_adj;
  const int2* ij;
  const int *row_ptr, *adj_col, *row_cnt;
  const uint32_t* pair_mask;
  const int* pair_wpre;
  const int* nbr;
  const float* fdof;
  const Box* chunk_box;
  const int* vperm;
  int W;
  const Box* body_box;
  const int2* chunk;
  const int* adj_pair;
  int cap_ccd;
  int4* ccd_cand;
  int nch;
  int* chunk_act;               // [nch + 1] the chunks of a pass with work (k_chunk_active), then their count
  int gh_energy;                // GH: also sum the candidates' barrier energies into energy
  const int* energy_gate;       // GH in the device loop: the energy only while this counter is 0
  unsigned long long* gtime;    // CCD_LS: first start / last end of the launch (global timer)
  const int* sup_valid;         // GH: take the candidates from ecand instead of the traversal
  int cap_act;
  int4* act_pairs;              // GH: active pairs with their coupling weights (preconditioner)
  FricRec* fric;                // lagged friction contacts (null: friction off)
  int cap_fric;
  uint32_t* fric_mask;          // their body pairs, as bits of the overlap matrix
  int fric_lag;                 // GH: this pass fixes the step's friction contacts (gated by
                                // energy_gate in the device loop: its first iteration)
  const Box* body_sup;          // CCD_LS: body boxes over every DOF set between the two
  const int* vbody;
  int cap_ecand;
  int4* ecand;                  // CCD_LS: line-search candidates
  // CCD_LS making the kept list (list_build): its candidates with their pairs; the displacement
  // it is made with dilates every box
  int make_list;
  int cap_list;
  int4* list;
  const double* skin;
  int cap_contacts;
  int4 *contacts, *contacts_by_pair;
  XSum* energy;                  // exact energy of the pass
  XSum* ls_energy;               // CCD_LS: the energies of the line-search batch that follows
  int prof;                     // kernel profiling: count the data read into prof rows
  unsigned long long* prof_rows;
  unsigned long long* toi_key;        // complemented bits of the minimum time of impact
  abd_states st;
  const double *mass, *I0;
  const int* fixed;
  const int *voff, *toff, *eoff, *tris, *edges;
  const double *y0, *y1, *x0;     // (y0 null: positions from the DOFs A, p, vertex_at)
  const double *A, *p, *A1, *p1;  // DOFs of y0 / y1 (affine node boxes), or null
  int affine;
  Tree tri, edge;
  int *pt_list, *ee_list;
  int cap_pt, cap_ee;
  int* pair_cand;
  int* dstat;
  double *offdiag, *pdiag, *pgrad;
  int* pair_active;
};

constexpr int kFricContact = 8;  // contact record y of a lagged friction contact (k_fric_pairs)

// A slot of an append-only list: one atomic per group of lanes that append together.
__device__ inline int append_slot(int* counter) {
  namespace cg = cooperative_groups;
  cg::coalesced_group g = cg::coalesced_threads();
  int base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(counter, (int)g.size());
  return g.shfl(base, 0) + (int)g.thread_rank();
}

// global vertex ids of a candidate: PT (point v, triangle t), EE (edge a, edge b)
__device__ inline void cand_vertices(const NarrowArgs& a, int type, int pa, int pb, int ids[4]) {
  if (type == 0) {
    ids[0] = pa;
    ids[1] = __ldg(&a.tris[3 * pb]);
    ids[2] = __ldg(&a.tris[3 * pb + 1]);
    ids[3] = __ldg(&a.tris[3 * pb + 2]);
  } else {
    ids[0] = __ldg(&a.edges[2 * pa]);
    ids[1] = __ldg(&a.edges[2 * pa + 1]);
    ids[2] = __ldg(&a.edges[2 * pb]);
    ids[3] = __ldg(&a.edges[2 * pb + 1]);
  }
}

__device__ inline void fetch(const double* y, const int ids[4], d3 xs[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) xs[k] = mk(__ldg(&y[3 * ids[k]]), __ldg(&y[3 * ids[k] + 1]), __ldg(&y[3 * ids[k] + 2]));
}

// position of vertex v of a pass: given, or from the DOFs (k_vertex_broad's arithmetic)
__device__ inline d3 vertex_at(const NarrowArgs& a, int v) {
  if (a.y0) return mk(__ldg(&a.y0[3 * v]), __ldg(&a.y0[3 * v + 1]), __ldg(&a.y0[3 * v + 2]));
  double M[12];
  load_dofs(a.A, a.p, __ldg(&a.vbody[v]), M);
  return position_of(M, a.x0, v);
}
__device__ inline void positions_at(const NarrowArgs& a, const int ids[4], d3 xs[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) xs[k] = vertex_at(a, ids[k]);
}

NarrowArgs narrow_args(Sim& s, int mode, const double* A, const double* p, const double* A1, const double* p1,
                       const double* y0, const double* y1, const abd_states* st);

// assemble.cu: the GH pass's pair blocks from its grouped contacts
cudaError_t pair_assemble(Sim& s, const NarrowArgs& a);
cudaError_t prepare_assemble();  // kernel attributes (once, at creation)

}  // namespace abd
