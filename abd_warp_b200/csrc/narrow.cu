// Narrow phase and per-body terms.
//
// One CTA per body pair {I, J} (I < J) walks the LBVH subtrees of the other body for
//   PT: every point of I against J's triangles, every point of J against I's triangles,
//   EE: every edge of I against J's edges,
// which is the reference's intended per-body-pair culling (cull_ / intersection_prims,
// abd/culling.py:32-52, 85-99) with the same float32 box predicate.  The pass mode decides
// what is done with each candidate:
//   LISTS / GH: candidates are written as contiguous, deterministically ordered per-pair
//       segments of the PT and EE lists (vec5i rows, as the reference's lists); GH then
//       evaluates the contacts of the segment (pt_ipc.py:111-190, ee_ipc.py:381-430) and
//       reduces them, in candidate order, into the pair's off-diagonal 12x12 block and its
//       contributions to the two diagonal blocks and gradients (put.py:25-66).  The
//       reduction replaces the reference's float atomics with a fixed-order sum, so the
//       assembled system is bitwise reproducible.
//   ENERGY: sum of barrier energies of the candidates (ipcsk/energy.py:9-48).
//   CCD: minimum time of impact over the candidates (ccd.py:20-40, 133-186).
// Per-body CTAs add inertia / orthogonality (orthogonal_energy.py:24-135) and the
// vertex-ground terms (vg_ipc.py:4-34, culling.py:54-82, ccd.py:9-18, energy.py:24-33).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "abd_graph.cuh"
#include "abd_ghpass.cuh"

namespace abd {

NarrowArgs narrow_args(Sim& s, int mode, const double* A, const double* p, const double* A1, const double* p1,
                       const double* y0, const double* y1, const abd_states* st) {
  NarrowArgs a;
  a.A = A;
  a.p = p;
  a.A1 = A1;
  a.p1 = p1;
  a.affine = A && p && (!y1 || (A1 && p1));
  a.mode = mode;
  a.prm = s.prm;
  a.n = s.n;
  a.cap_adj = s.cap_adj;
  a.ij = s.ij;
  a.row_ptr = s.row_ptr;
  a.adj_col = s.adj_col;
  a.row_cnt = s.row_cnt;
  a.pair_mask = s.pair_mask;
  a.pair_wpre = s.pair_wpre;
  a.nbr = s.nbr;
  a.fdof = s.fdof;
  a.chunk_box = s.chunk_box;
  a.vperm = s.vperm;
  a.W = s.W;
  a.body_box = s.body_box;
  a.chunk = s.chunk;
  a.nch = s.nch;
  a.chunk_act = s.chunk_act;
  a.energy = s.energy_acc;
  a.prof = s.prof_on == 2;
  a.prof_rows = &s.box->prof[0][0];
  a.adj_pair = s.adj_pair;
  a.cap_ccd = s.cap_ccd;
  a.ccd_cand = s.ccd_cand;
  a.body_sup = s.body_sup;
  a.gh_energy = s.gh_energy;
  a.energy_gate = s.energy_gate;
  a.gtime = s.prof_events < 0 ? &s.box->step.t0 : nullptr;
  a.sup_valid = s.dint + kSupValid;
  a.cap_act = s.cap_act;
  a.act_pairs = s.act_pairs;
  const bool fr = s.prm.friction_mu > 0.0;
  a.fric = fr ? s.fric : nullptr;
  a.cap_fric = s.cap_fric;
  a.fric_mask = fr ? s.fric_mask : nullptr;
  a.fric_lag = fr ? (s.energy_gate ? 1 : s.fric_lag) : 0;
  a.vbody = s.vbody;
  a.make_list = 0;
  a.cap_list = s.cap_list;
  a.list = s.list;
  a.skin = s.dpar + kParSkinNext;
  a.cap_ecand = s.cap_ecand;
  a.ecand = s.ecand;
  a.cap_contacts = s.cap_contacts;
  a.contacts = s.contacts;
  a.contacts_by_pair = s.contacts_by_pair;
  a.toi_key = s.dmin;
  a.ls_energy = s.box->ls_energy;
  a.st = st ? *st : abd_states{};
  a.mass = s.mass;
  a.I0 = s.I0;
  a.fixed = s.fixed;
  a.voff = s.voff;
  a.toff = s.toff;
  a.eoff = s.eoff;
  a.tris = s.tris;
  a.edges = s.edges;
  a.y0 = y0;
  a.y1 = y1;
  a.x0 = s.x0;
  a.tri = s.tri_tree;
  a.edge = s.edge_tree;
  a.pt_list = s.pt_list;
  a.ee_list = s.ee_list;
  a.cap_pt = s.cap_pt;
  a.cap_ee = s.cap_ee;
  a.pair_cand = s.pair_cand;
  a.dstat = s.dstat;
  a.offdiag = s.offdiag;
  a.pdiag = s.pdiag;
  a.pgrad = s.pgrad;
  a.pair_active = s.pair_active;
  return a;
}

BodyArgs body_args(Sim& s, const abd_states* st, const double* A, const double* p, const double* y, const double* y1) {
  BodyArgs a;
  a.prm = s.prm;
  a.n = s.n;
  a.voff = s.voff;
  a.x0 = s.x0;
  a.mass = s.mass;
  a.I0 = s.I0;
  a.fixed = s.fixed;
  if (st) a.st = *st;
  else a.st = abd_states{};
  a.A = A;
  a.p = p;
  a.y = y;
  a.y1 = y1;
  a.body_box = s.body_box;
  a.row_ptr = s.row_ptr;
  a.adj_pair = s.adj_pair;
  a.pair_active = s.pair_active;
  a.ij = s.ij;
  a.pdiag = s.pdiag;
  a.pgrad = s.pgrad;
  a.diag = s.diag;
  a.g = s.g;
  a.dstat = s.dstat;
  a.vg_list = s.vg_list;
  a.cap_vg = s.cap_vg;
  a.energy = s.gh_energy ? s.energy_acc : nullptr;
  a.energy_gate = s.energy_gate;
  a.exact = s.exact_hessian;
  a.highlight = s.highlight;
  return a;
}

namespace {

constexpr int NT = 128;          // threads per pair CTA
constexpr int NW = NT / 32;

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// start bringing the line at p into L2
__device__ inline void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Per-CTA view of one body's subtree boxes.  Refit mode (m0 == null): the stored boxes.
// Affine mode: internal nodes are the affine images of their rest boxes under the body's
// DOFs at y0 (m0) and, when swept, y1 (m1); leaves are computed from the positions, or, with
// sup, are the affine images of their rest boxes too (boxes that hold the leaf's box at every
// DOF set between m0 and m1).
struct NodeBoxes {
  const Tree* tr;
  const float *m0, *m1;
  float pad;
  const int* prims;   // tris or edges
  int tri;            // 1: triangle tree, 0: edge tree
  int sup;
  const double *y0, *y1;
  double dhh;
  __device__ inline Box internal(int node) const {
    if (!m0) return load_box(&tr->box[node]);
    return affine_box2(load_box(&tr->rest[node]), m0, m1, pad);
  }
  __device__ inline Box leaf(int node, int prim) const {
    if (!m0) return load_box(&tr->box[node]);
    if (sup) return affine_box2(load_box(&tr->rest[node]), m0, m1, pad);
    return tri ? tri_leaf_box(prims, y0, y1, prim) : edge_leaf_box(prims, y0, y1, prim, dhh);
  }
};

// Stack traversal of the subtree rooted at `root`; calls f(prim) for every leaf whose box
// overlaps q, in a fixed depth-first order.  A popped node's child table lists its up to four
// descendants one or two levels down, tested together: the walk is half as deep as the
// binary tree's, and in affine mode a visit costs one round of independent loads (codes and
// rest boxes, indexed by the node itself); refit mode reads the stored world boxes.
// visits: tested internal nodes and leaves (kernel profiling)
struct Visits {
  unsigned internal = 0, leaf = 0;
};

// One visit: the child table of `node` (codes and rest boxes, indexed by the node itself);
// every leaf child whose box overlaps q goes to f(prim), every internal one to push(node).
template <class F, class P>
__device__ inline void expand_node(const NodeBoxes& nb, int node, const Box& q, F&& f, P&& push, Visits& cnt) {
  const Tree& tr = *nb.tr;
  const int L0 = tr.N - 1;
  const int4 cc = __ldg(&tr.ccode[node]);
  Box R[4];
  if (nb.m0) {
#pragma unroll
    for (int h = 0; h < 4; ++h) R[h] = load_box(&tr.crest[4 * node + h]);
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int code = h == 0 ? cc.x : h == 1 ? cc.y : h == 2 ? cc.z : cc.w;
    if (code == kNoChild) continue;
    if (code < 0) {
      const int prim = ~code;
      ++cnt.leaf;
      Box B;
      if (!nb.m0) B = load_box(&tr.box[L0 + __ldg(&tr.prim_leaf[prim])]);
      else if (nb.sup) B = affine_box2(R[h], nb.m0, nb.m1, nb.pad);
      else B = nb.tri ? tri_leaf_box(nb.prims, nb.y0, nb.y1, prim) : edge_leaf_box(nb.prims, nb.y0, nb.y1, prim, nb.dhh);
      if (overlap(B, q)) f(prim);
    } else {
      ++cnt.internal;
      const Box B = nb.m0 ? affine_box2(R[h], nb.m0, nb.m1, nb.pad) : load_box(&tr.box[code]);
      if (overlap(B, q)) push(code);
    }
  }
}

// every pushed node is visited later: start bringing its child table to L2 now
__device__ inline void prefetch_node(const Tree& tr, int node) {
  prefetch_l2(&tr.ccode[node]);
  prefetch_l2(&tr.crest[4 * node]);
}

template <class F>
__device__ inline void traverse(const NodeBoxes& nb, int root, const Box& q, int* dstat, F&& f) {
  Visits v;
  traverse(nb, root, q, dstat, f, v);
}

template <class F>
__device__ inline void traverse(const NodeBoxes& nb, int root, const Box& q, int* dstat, F&& f, Visits& cnt) {
  if (root < 0) return;
  const Tree& tr = *nb.tr;
  const int L0 = tr.N - 1;
  if (root >= L0) {
    const int prim = __ldg(&tr.leaf_prim[root - L0]);
    ++cnt.leaf;
    if (overlap(nb.leaf(root, prim), q)) f(prim);
    return;
  }
  ++cnt.internal;
  if (!overlap(nb.internal(root), q)) return;
  int stack[kTraversalStack];
  int sp = 0;
  stack[sp++] = root;
  while (sp > 0) {
    const int node = stack[--sp];
    expand_node(nb, node, q, f, [&](int c) {
      if (sp < kTraversalStack) {
        stack[sp++] = c;
        if (nb.m0) prefetch_node(tr, c);
      } else {
        atomicOr(&dstat[DS_STATUS], ST_STACK_OVERFLOW);
      }
    }, cnt);
  }
}

struct PairInfo {
  int I, J, nPT1, nPT2, nEE;
  const float* dof;  // shared [2 bodies][2 times][12] FP32 DOFs (I, J), or null
};

__device__ inline PairInfo pair_info(const NarrowArgs& a, int p) {
  PairInfo P;
  const int2 ij = a.ij[p];
  P.I = ij.x;
  P.J = ij.y;
  P.nPT1 = a.prm.enable_pt ? a.voff[P.I + 1] - a.voff[P.I] : 0;
  P.nPT2 = a.prm.enable_pt ? a.voff[P.J + 1] - a.voff[P.J] : 0;
  P.nEE = a.prm.enable_ee ? a.eoff[P.I + 1] - a.eoff[P.I] : 0;
  P.dof = nullptr;
  return P;
}

// tree boxes of one body: m = its FP32 DOFs [y0: 12][y1: 12] in shared memory, or null
__device__ inline NodeBoxes node_boxes(const NarrowArgs& a, const Tree* tr, bool tri, const float* m) {
  NodeBoxes nb;
  nb.tr = tr;
  nb.m0 = m;
  nb.m1 = m && a.y1 ? m + 12 : nullptr;
  nb.pad = tri ? 0.f : __double2float_ru(0.5 * a.prm.dhat);  // triangle boxes are undilated
  nb.prims = tri ? a.tris : a.edges;
  nb.tri = tri;
  nb.sup = 0;
  nb.y0 = a.y0;
  nb.y1 = a.y1;
  nb.dhh = 0.5 * a.prm.dhat;
  return nb;
}

// Visit every candidate of item k: f(type, pointOrEdgeBody, primA_global, primB_global)
template <class F>
__device__ inline void visit_item(const NarrowArgs& a, const PairInfo& P, int k, F&& f) {
  const float dhf = (float)a.prm.dhat;
  if (k < P.nPT1 + P.nPT2) {
    const bool first = k < P.nPT1;
    const int body = first ? P.I : P.J, other = first ? P.J : P.I;
    const int v = a.voff[body] + (first ? k : k - P.nPT1);
    const Box q = point_box(a.y0, a.y1, v, dhf);
    traverse(node_boxes(a, &a.tri, true, P.dof ? P.dof + 24 * (first ? 1 : 0) : nullptr),
             __ldg(&a.tri.body_root[other]), q, a.dstat, [&](int t) { f(0, first ? 0 : 1, v, t); });
  } else {
    const int e = a.eoff[P.I] + (k - P.nPT1 - P.nPT2);
    const Box q = P.dof ? edge_leaf_box(a.edges, a.y0, a.y1, e, 0.5 * a.prm.dhat)
                        : load_box(&a.edge.box[(a.edge.N - 1) + __ldg(&a.edge.prim_leaf[e])]);
    traverse(node_boxes(a, &a.edge, false, P.dof ? P.dof + 24 : nullptr), __ldg(&a.edge.body_root[P.J]), q,
             a.dstat, [&](int eb) { f(1, 0, e, eb); });
  }
}

// block-wide exclusive scan of one int per thread; returns the total
__device__ inline int block_scan(int v, int* sh, int& excl) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int w = 0; w < NW; ++w) {
      const int c = sh[w];
      sh[w] = acc;
      acc += c;
    }
    sh[NW] = acc;
  }
  __syncthreads();
  excl = sh[warp] + x - v;
  const int total = sh[NW];
  __syncthreads();
  return total;
}

// Candidate lists (the reference's vec5i PT / EE lists, culling.py:85-99): one CTA per body
// pair (grid = pair capacity), each pair a contiguous segment in traversal order.
__global__ void __launch_bounds__(NT) k_pair_lists(NarrowArgs a) {
  const int p = blockIdx.x;
  // pair count of this pass (device); an overflowed pass is rerun by the host
  if (p >= a.dstat[DS_NPAIRS] || (a.dstat[DS_STATUS] & ST_PAIR_OVERFLOW)) return;
  PairInfo P = pair_info(a, p);
  const int items = P.nPT1 + P.nPT2 + P.nEE;
  const int tid = threadIdx.x;
  __shared__ int sh[NW + 1];
  __shared__ float sdof[2][2][12];  // [I, J][y0, y1][A row-major, p]
  if (a.affine) {
    if (tid < 48) {
      const int side = tid / 24, t = (tid / 12) & 1, c = tid % 12;
      const int b = side ? P.J : P.I;
      const double* A = t ? a.A1 : a.A;
      const double* q = t ? a.p1 : a.p;
      if (!t || a.y1) sdof[side][t][c] = (float)(c < 9 ? A[9 * b + c] : q[3 * b + c - 9]);
    }
    __syncthreads();
    P.dof = &sdof[0][0][0];
  }

  // ---- LISTS / GH: two passes over the candidates (count, then write in order) ----
  int cpt = 0, cee = 0;
  for (int k = tid; k < items; k += NT)
    visit_item(a, P, k, [&](int type, int, int, int) {
      if (type == 0) ++cpt;
      else ++cee;
    });
  int opt, oee;
  const int tpt = block_scan(cpt, sh, opt);
  const int tee = block_scan(cee, sh, oee);
  __shared__ int base_pt, base_ee, ok;
  if (tid == 0) {
    base_pt = atomicAdd(&a.dstat[DS_PT_COUNT], tpt);
    base_ee = atomicAdd(&a.dstat[DS_EE_COUNT], tee);
    ok = 1;
    if (base_pt + tpt > a.cap_pt) {
      atomicOr(&a.dstat[DS_STATUS], ST_PT_OVERFLOW);
      ok = 0;
    }
    if (base_ee + tee > a.cap_ee) {
      atomicOr(&a.dstat[DS_STATUS], ST_EE_OVERFLOW);
      ok = 0;
    }
    a.pair_cand[4 * p + 0] = base_pt;
    a.pair_cand[4 * p + 1] = tpt;
    a.pair_cand[4 * p + 2] = base_ee;
    a.pair_cand[4 * p + 3] = tee;
  }
  __syncthreads();
  if (!ok) {
    return;
  }
  {
    int wpt = base_pt + opt, wee = base_ee + oee;
    for (int k = tid; k < items; k += NT)
      visit_item(a, P, k, [&](int type, int swap, int pa, int pb) {
        // (I, J, pair, local prim of I, local prim of J) with I the point's / first edge's body
        int* row = type == 0 ? &a.pt_list[5 * (size_t)wpt++] : &a.ee_list[5 * (size_t)wee++];
        const int bI = swap ? P.J : P.I, bJ = swap ? P.I : P.J;
        row[0] = bI;
        row[1] = bJ;
        row[2] = p;
        row[3] = type == 0 ? pa - a.voff[bI] : pa - a.eoff[bI];
        row[4] = type == 0 ? pb - a.toff[bJ] : pb - a.eoff[bJ];
      });
  }
}

// ---------------------------------------------------------------------------------------
// GH assembly: the active contacts found by the chunk pass, grouped by body pair
// ---------------------------------------------------------------------------------------
// (skipped when the pass overflowed: it is made again)
__global__ void __launch_bounds__(1024) k_contact_scan(int cap_pairs, int* pair_cand, int* dstat, int cap_contacts,
                                                       const int4* in, int4* out, int* pair_active) {
  if (dstat[DS_STATUS] & (ST_PAIR_OVERFLOW | ST_CONTACT_OVERFLOW)) return;
  contact_scan(cap_pairs, pair_cand, dstat, cap_contacts, in, out, pair_active);
}

// the contacts into their segments, one thread per contact (lists above kScanScatter)
__global__ void k_contact_scatter(int cap_contacts, const int4* in, int* pair_cand, int4* out,
                                  const int* dstat) {
  if (dstat[DS_STATUS] & (ST_PAIR_OVERFLOW | ST_CONTACT_OVERFLOW)) return;
  scatter_contacts(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, cap_contacts, in, pair_cand, out,
                   dstat);
}

// ---------------------------------------------------------------------------------------
// per-body terms shared by the body kernels and the energy / CCD chunks
// ---------------------------------------------------------------------------------------
// time of impact of a vertex with the ground plane (ccd.py:9-18); 1 when none
__device__ inline double vg_toi(const abd_params& P, const double* y0, const double* y1, int v) {
  const double d1 = y1[3 * v + 1] - P.ground;
  double tt = 1.0;
  if (d1 < 0) {
    const double d0 = y0[3 * v + 1] - P.ground;
    tt = d0 / (d0 - d1);
  }
  return tt;
}

// minimum of non-negative doubles by atomicMax on the complemented bit patterns (0 = none)
__device__ inline void toi_min(unsigned long long* key, double t) {
  atomicMax(key, ~(unsigned long long)__double_as_longlong(t));
}

// ---------------------------------------------------------------------------------------
// energy / CCD passes: one CTA per chunk of one body's points and edges
// ---------------------------------------------------------------------------------------
constexpr int CT = 128;  // threads per chunk CTA
static_assert(kChunk <= CT && kChunk <= 256, "a chunk's queries: one thread each when loaded, 8-bit ids");
constexpr int kNoQuery = INT_MIN;  // a chunk item whose primitive kind is disabled
constexpr int NBB = 64;     // neighbours staged per batch

// The k-th neighbour (increasing order) of body I from the overlap bit matrix: the word by
// binary search over the row's prefix counts, then the bit inside it.
__device__ inline int kth_neighbour(const NarrowArgs& a, int I, int k) {
  const int* pre = a.pair_wpre + (size_t)I * a.W;
  int lo = 0, hi = a.W - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= k) lo = mid;
    else hi = mid - 1;
  }
  uint32_t m = a.pair_mask[(size_t)I * a.W + lo];
  for (int r = k - pre[lo]; r > 0; --r) m &= m - 1;
  return 32 * lo + __ffs(m) - 1;
}

// Which body of a pair {I, J} queries the other's edge tree for the EE candidates: the one
// with more edges; at equal edge counts the one with fewer neighbours (dI, dJ: the pass's row
// counts), then the higher index.  A body with many neighbours (a ground box among cubes of
// as many edges) would otherwise query every neighbour's tree from its one chunk, in series.
// The candidate set does not depend on the choice (the box predicate is symmetric).
__device__ inline bool ee_owner(int I, int nEI, int dI, int J, int nEJ, int dJ) {
  return nEI > nEJ || (nEI == nEJ && (dI < dJ || (dI == dJ && I > J)));
}

// Body I's points against the triangle trees of all its neighbours J (PT pairs (I, J); the
// pairs (J, I) come from J's chunks), and its edges against the edge trees of the neighbours
// it owns the EE candidates with -- the same candidates as the per-pair kernel, each query
// box built once.  A query is only traversed into J's tree when it overlaps J's body box,
// which contains every leaf box of J.  The overlapping (query, neighbour) combinations of a
// batch are compacted and their traversals spread over the CTA's threads.  The first chunk
// of every body also adds the body's own terms: inertia + orthogonality and the
// vertex-ground barriers (ENERGY) or the vertex-ground times of impact (CCD).
// ENERGY adds every nonzero term to one exact accumulator of the whole pass (any order gives
// the same sum); CCD takes the minimum time of impact by an atomic maximum on complemented
// bits.  (ipcsk/energy.py:9-48, orthogonal_energy.py:24-32, ccd.py:9-40, 133-186)
// CCD_LS is the CCD pass of the step: it culls with boxes that hold every box of the
// primitives at all DOF sets between the pass's two (body_sup, the affine images of the
// queries' and leaves' rest boxes) and appends every pair found to the line-search
// candidates; the pairs that also pass the CCD pass's own boxes (body pair, query and leaf)
// become CCD candidates, the same set as the CCD pass finds.
// The displacement that dilates the boxes of a pass that makes the kept list (each body moves at
// most that far from the pass's DOF segment)
__device__ inline float list_skin(const NarrowArgs& a) { return a.make_list ? __double2float_ru(*a.skin) : 0.f; }

// The world box of chunk c of body I: the affine image of its rest box at the pass's DOFs
// (with y1: the union over both DOF sets), dilated by dhat.  Every query box of the chunk lies
// inside.
__device__ inline Box chunk_world_box(const NarrowArgs& a, int c, int I) {
  const Box R = load_box(&a.chunk_box[c]);
  const float pad = __double2float_ru(a.prm.dhat) + list_skin(a);
  Box b = affine_box(R, a.fdof + 24 * (size_t)I, pad);
  if (a.y1) {
    const Box B1 = affine_box(R, a.fdof + 24 * (size_t)I + 12, pad);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b.lo[k] = fminf(b.lo[k], B1.lo[k]);
      b.hi[k] = fmaxf(b.hi[k], B1.hi[k]);
    }
  }
  return b;
}

// The chunks of a pass with work, one warp per chunk: those whose world box overlaps the body
// box of a neighbour (CCD_LS: the box over the DOF range), and a body's first chunk when the
// pass adds the body's own terms there (ENERGY; CCD with vertex-ground contacts).  They are
// appended to chunk_act, whose entry nch counts them; k_chunk_narrow's first CTAs take them.
// In a resting pile most chunks face no neighbour, and finding that out costs a chunk CTA a
// chain of dependent loads; here it costs a warp.  (The tests are k_chunk_narrow's own: a
// chunk that is left out would have found no neighbour there.)
constexpr int KA = 256;  // threads of the chunk filter
template <int MODE>
__global__ void __launch_bounds__(KA) k_chunk_active(NarrowArgs a) {
  constexpr bool ls = MODE == NARROW_CCD_LS;
  constexpr bool ccd = MODE == NARROW_CCD || ls, gh = MODE == NARROW_GH;
  if constexpr (gh) {
    if (*a.sup_valid) return;
  }
  if (ls && a.gtime && threadIdx.x == 0) atomicMin(&a.gtime[0], globaltimer_ns());
  const int lane = (int)(threadIdx.x & 31);
  const int c = (int)((blockIdx.x * KA + threadIdx.x) >> 5);
  if (c >= a.nch) return;
  const int2 ch = a.chunk[c];
  const int I = ch.x;
  const int nEI = a.eoff[I + 1] - a.eoff[I];
  const int nV = a.voff[I + 1] - a.voff[I];
  const int Q = max(0, min(kChunk, nV + nEI - ch.y));
  bool need = !gh && ch.y == 0 && (!ccd || (a.prm.ground_enabled && a.prm.enable_vg && !a.make_list));
  const bool adj = gh || (ls && a.make_list);  // neighbours from the adjacency (with their pairs)
  int r0 = 0, deg;
  if (adj) {
    r0 = a.row_ptr[I];
    deg = (a.dstat[DS_STATUS] & ST_PAIR_OVERFLOW) ? 0 : min(a.row_ptr[I + 1], a.cap_adj) - r0;
  } else {
    deg = a.row_cnt[I];
  }
  if (Q == 0) deg = 0;
  if (ls && a.prof && lane == 0 && deg > 0)
    atomicAdd(&a.prof_rows[8 * (c & 31) + PF_NEIGHBOUR], (unsigned long long)deg);
  if (!need && deg > 0) {
    const Box cbx = chunk_world_box(a, c, I);
    for (int k0 = 0; k0 < deg && !need; k0 += 32) {
      const int k = k0 + lane;
      bool rel = false;
      if (k < deg) {
        const int J = adj ? a.adj_col[r0 + k] : (k < kNbList ? a.nbr[(size_t)I * kNbList + k] : kth_neighbour(a, I, k));
        rel = overlap(cbx, load_box(&(ls ? a.body_sup : a.body_box)[J]));
      }
      need = __any_sync(0xffffffffu, rel);
    }
  }
  if (need && lane == 0) a.chunk_act[atomicAdd(&a.chunk_act[a.nch], 1)] = c;
}

constexpr int CW = 4 * CT;  // (query, neighbour) combinations tested per round
constexpr int kFront = 512;  // entries of a breadth-first frontier
constexpr int kCandBuf = 256;  // candidates a chunk CTA gathers before it writes them out
template <int MODE>
__global__ void __launch_bounds__(CT, 5) k_chunk_narrow(NarrowArgs a) {
  constexpr bool ls = MODE == NARROW_CCD_LS;
  constexpr bool ccd = MODE == NARROW_CCD || ls, gh = MODE == NARROW_GH;
  if constexpr (gh) {
    if (*a.sup_valid) return;  // k_gh_scan takes the candidates from ecand
  }
  const int tid = threadIdx.x;
  if ((int)blockIdx.x >= a.chunk_act[a.nch]) {  // more CTAs than chunks with work
    if (ls && a.gtime && tid == 0) atomicMax(&a.gtime[1], globaltimer_ns());
    return;
  }
  const int c = a.chunk_act[blockIdx.x];
  const int2 ch = a.chunk[c];
  const int I = ch.x;
  const int nEI = a.eoff[I + 1] - a.eoff[I];
  const int nV = a.voff[I + 1] - a.voff[I];  // items: the body's points, then its edges
  const int Q = max(0, min(kChunk, nV + nEI - ch.y));
  __shared__ Box qbox[kChunk];  // query boxes (CCD_LS: over the DOF range)
  __shared__ int qprim[kChunk];  // point id, ~edge id, or kNoQuery (primitive kind disabled)
  __shared__ Box nbox[NBB];
  __shared__ __align__(16) float ndof[NBB][24];
  __shared__ int nJ[NBB], ntri[NBB], nedge[NBB], nown[NBB], npair[NBB], nrel[NBB];
  __shared__ unsigned short work[CW];
  __shared__ int nwork;
  __shared__ int2 front[2][kFront];  // breadth-first frontiers: (query | neighbour << 8, node)
  __shared__ int nfr[2];
  int fcur = 0;
  // frontier entries in use: all of them, or fewer when a test injects a small capacity
  const int fcap = a.prm.min_capacity > 0 ? min(kFront, a.prm.min_capacity) : kFront;
  __shared__ XSum xe;
  __shared__ unsigned long long tkey;
  __shared__ Box cbx;  // the chunk's world box: every query box of the chunk lies inside
  if (tid == 0 && Q > 0) cbx = chunk_world_box(a, c, I);
  // The candidates (GH, CCD, CCD_LS) gather in shared memory and go to their list in blocks,
  // one global atomic per block: a hit does not wait on the list's counter, which every CTA
  // of the launch shares.  A full buffer sends the rest straight to the list.
  constexpr bool lists = gh || ccd;
  __shared__ int4 cbuf[kCandBuf];
  __shared__ int ncb, cbase;
  const bool mk_list = ls && a.make_list;
  const bool adj = gh || mk_list;  // neighbours from the adjacency (with their pairs)
  int* const ccount = &a.dstat[mk_list ? DS_NLIST : ls ? DS_NECAND : DS_NCCD];
  int4* const cdst = mk_list ? a.list : ls ? a.ecand : a.ccd_cand;
  const int ccap = mk_list ? a.cap_list : ls ? a.cap_ecand : a.cap_ccd;
  const int cflag = mk_list ? ST_LIST_OVERFLOW : ls ? ST_ECAND_OVERFLOW : ST_CCD_OVERFLOW;
  const float skin = ls ? list_skin(a) : 0.f;
  auto emit = [&](int4 rec) {
    const int k = atomicAdd(&ncb, 1);
    if (k < kCandBuf) {
      cbuf[k] = rec;
    } else {
      const int pos = append_slot(ccount);
      if ((unsigned)pos < (unsigned)ccap) cdst[pos] = rec;
      else atomicOr(&a.dstat[DS_STATUS], cflag);
    }
  };
  // the buffer to the list: every thread, after a barrier that follows the emits
  auto flush = [&]() {
    const int n = min(ncb, kCandBuf);
    if (n == 0) return;
    if (tid == 0) cbase = atomicAdd(ccount, n);
    __syncthreads();
    for (int e = tid; e < n; e += CT) {
      if ((unsigned)(cbase + e) < (unsigned)ccap) cdst[cbase + e] = cbuf[e];
      else atomicOr(&a.dstat[DS_STATUS], cflag);
    }
    __syncthreads();
    if (tid == 0) ncb = 0;  // the next barrier orders it before the next emit
  };
  if (tid == 0) ncb = 0;
  if (tid == 0) nfr[0] = nfr[1] = 0;
  if (ccd) {
    if (tid == 0) tkey = 0;
  } else {
    for (int e = tid; e < kXD + 1; e += CT) reinterpret_cast<long long*>(&xe)[e] = 0;
  }
  __syncthreads();
  unsigned pf_node = 0, pf_tri = 0, pf_edge = 0, pf_cand = 0;  // profiling: entries tested, candidates
  // the body's own terms, in its first chunk (GH: the body kernel adds them)
  if (!gh && ch.y == 0 && !mk_list) {
    const Box bb = load_box(&a.body_box[I]);
    const bool vg = a.prm.ground_enabled && a.prm.enable_vg;
    for (int v = a.voff[I] + tid; vg && v < a.voff[I + 1]; v += CT) {
      if (!vg_candidate_of(a.prm, bb, a.y0, a.y1, v)) continue;
      if constexpr (ccd) {
        const double t = vg_toi(a.prm, a.y0, a.y1, v);
        if (t < 1.0) toi_min(&tkey, t);
      } else {
        const double d = a.y0[3 * v + 1] - a.prm.ground;
        const double e = barrier(d * d, a.prm);
        if (e != 0.0) xs_add_atomic(&xe, e);
      }
    }
    if (!ccd && tid == 0 && !a.fixed[I])
      xs_add_atomic(&xe, inertia_energy(a.prm, a.st, a.mass, a.I0, I, a.A + 9 * I, a.p + 3 * I));
  }
  // neighbours of I in increasing order: GH from the adjacency (it needs the pair indices;
  // an overflowed pass is rerun), ENERGY / CCD straight from the overlap bit matrix
  int r0 = 0, deg;
  if (adj) {
    r0 = a.row_ptr[I];
    deg = (a.dstat[DS_STATUS] & ST_PAIR_OVERFLOW) ? 0 : min(a.row_ptr[I + 1], a.cap_adj) - r0;
  } else {
    deg = a.row_cnt[I];
  }
  if (Q == 0) deg = 0;
  bool loaded = false;  // queries are loaded when the first neighbour overlaps the chunk
  for (int b0 = 0; b0 < deg; b0 += NBB) {
    const int nb = min(NBB, deg - b0);
    __syncthreads();
    // ENERGY / CCD past the listed neighbours: the CTA decodes the batch from the row's overlap
    // words (their prefix counts place each word's bits), one round of loads for the batch
    const bool decode = !adj && b0 + nb > kNbList;
    if (decode) {
      for (int w = tid; w < a.W; w += CT) {
        const int pre = a.pair_wpre[(size_t)I * a.W + w];
        if (pre >= b0 + nb) continue;
        uint32_t m = a.pair_mask[(size_t)I * a.W + w];
        if (pre + __popc(m) <= b0) continue;
        for (int k = pre; m; m &= m - 1, ++k)
          if (k >= b0 && k < b0 + nb) nJ[k - b0] = 32 * w + __ffs(m) - 1;
      }
      __syncthreads();
    }
    int rel = 0;
    if (tid < nb) {
      const int k = b0 + tid;
      const int J = adj ? a.adj_col[r0 + k] : (decode ? nJ[tid] : a.nbr[(size_t)I * kNbList + k]);
      nJ[tid] = J;
      nbox[tid] = load_box(&(ls ? a.body_sup : a.body_box)[J]);
      rel = overlap(cbx, nbox[tid]) ? 1 : 0;
      nrel[tid] = rel;
      ntri[tid] = a.tri.body_root[J];
      nedge[tid] = a.edge.body_root[J];
      nown[tid] = ee_owner(I, nEI, a.row_cnt[I], J, a.eoff[J + 1] - a.eoff[J], a.row_cnt[J]);
      if (adj) npair[tid] = a.adj_pair[r0 + b0 + tid];
    }
    if (!__syncthreads_or(rel)) continue;  // the chunk touches none of these neighbours
    if (!loaded) {
      loaded = true;
      if (tid < Q) {
        const int k = ch.y + tid;
        const float* m = a.fdof + 24 * (size_t)I;
        if (k < nV) {
          const int v = __ldg(&a.vperm[a.voff[I] + k]);
          qprim[tid] = a.prm.enable_pt ? v : kNoQuery;
          if constexpr (ls) {  // the point's box over the DOF range, from its rest position
            Box R;
#pragma unroll
            for (int d = 0; d < 3; ++d) R.lo[d] = R.hi[d] = (float)__ldg(&a.x0[3 * v + d]);
            qbox[tid] = affine_box2(R, m, m + 12, __double2float_ru(a.prm.dhat) + skin);
          } else {
            qbox[tid] = point_box(a.y0, a.y1, v, (float)a.prm.dhat);
          }
        } else {
          const int e = __ldg(&a.edge.leaf_prim[a.eoff[I] + (k - nV)]);
          qprim[tid] = a.prm.enable_ee ? ~e : kNoQuery;
          if constexpr (ls)  // the edge's box over the DOF range, from its rest box
            qbox[tid] = affine_box2(load_box(&a.edge.rest[(a.edge.N - 1) + a.eoff[I] + (k - nV)]), m, m + 12,
                                    __double2float_ru(0.5 * a.prm.dhat) + skin);
          else
            qbox[tid] = edge_leaf_box(a.edges, a.y0, a.y1, e, 0.5 * a.prm.dhat);
        }
      }
      if constexpr (ls) {
        if (a.prof && tid == 0) {
          const int qp = max(0, min(Q, nV - ch.y));
          atomicAdd(&a.prof_rows[8 * (blockIdx.x & 31) + PF_POINT], (unsigned long long)qp);
          atomicAdd(&a.prof_rows[8 * (blockIdx.x & 31) + PF_EDGE], (unsigned long long)(Q - qp));
        }
      }
    }
    // FP32 DOFs of the neighbours, as the broad phase wrote them (6 x 16 B per neighbour)
    for (int e = tid; e < 6 * nb; e += CT) {
      const int j = e / 6, q = e % 6;
      if (q < 3 || a.y1)
        reinterpret_cast<float4*>(ndof[j])[q] = __ldg(reinterpret_cast<const float4*>(a.fdof + 24 * (size_t)nJ[j]) + q);
    }
    for (int w0 = 0; w0 < Q * nb; w0 += CW) {
      if (tid == 0) nwork = 0;
      __syncthreads();
      // overlapping (query, neighbour) combinations of this round
      for (int it = w0 + tid; it < min(Q * nb, w0 + CW); it += CT) {
        const int q = it % Q, j = it / Q;
        if (!nrel[j] || qprim[q] == kNoQuery || (qprim[q] < 0 && !nown[j])) continue;
        if (!overlap(qbox[q], nbox[j])) continue;
        work[atomicAdd(&nwork, 1)] = (unsigned short)(q | (j << 8));
      }
      __syncthreads();
      // the compacted (query, neighbour) combinations walk their neighbour's tree breadth
      // first: each round every thread takes frontier entries (query, neighbour, node) and
      // expands them into the next frontier, so the visits of a chunk in heavy contact spread
      // over the CTA instead of queueing on the threads that drew its longest walks.  When the
      // frontier is full a thread walks the subtree itself, depth first.
      auto visit = [&](int q, int j, int type, int pa, int pb) {
        if constexpr (gh) {
          // evaluated by k_gh_eval, one thread per candidate.  PT: the point is I's, the
          // pair's first body is min(I, J); EE: the lower body's edge comes first
          const int swap = (type == 0 && I > nJ[j]) ? 1 : 0;
          emit(make_int4(npair[j], type | (swap << 1), pa, pb));
        } else if constexpr (ls) {
          // line-search candidates; k_ccd_eval takes those that pass the CCD pass's boxes
          ++pf_cand;
          emit(make_int4(type, pa, pb, mk_list ? npair[j] : 0));
        } else if constexpr (ccd) {  // evaluated by k_ccd_eval, one thread per candidate
          emit(make_int4(type, pa, pb, 0));
        } else {
          int ids[4];
          d3 xs[4];
          cand_vertices(a, type, pa, pb, ids);
          fetch(a.y0, ids, xs);
          const double e = candidate_energy(a, type, ids, xs);
          if (e != 0.0) xs_add_atomic(&xe, e);
        }
      };
      // a leaf of J's tree reached by query q: PT (I's point, J's triangle) or EE (the lower
      // body's edge first, as the per-pair lists)
      auto hit = [&](int q, int j, int prim) {
        const int qp = qprim[q];
        if (qp >= 0) visit(q, j, 0, qp, prim);
        else if (I < nJ[j]) visit(q, j, 1, ~qp, prim);
        else visit(q, j, 1, prim, ~qp);
      };
      auto boxes_of = [&](int q, int j) {
        const bool tri = qprim[q] >= 0;
        NodeBoxes nbx = node_boxes(a, tri ? &a.tri : &a.edge, tri, ndof[j]);
        nbx.sup = ls;
        nbx.pad += skin;
        return nbx;
      };
      auto tally = [&](bool tri, const Visits& vc) {
        pf_node += vc.internal;
        if (tri) pf_tri += vc.leaf;
        else pf_edge += vc.leaf;
      };
      // frontier entry: (q | j << 8, node); a full frontier makes the pusher walk the subtree
      auto push = [&](int nxt, int q, int j, int node) {
        const NodeBoxes nbx = boxes_of(q, j);
        const int slot = atomicAdd(&nfr[nxt], 1);
        if (slot < fcap) {
          front[nxt][slot] = make_int2(q | (j << 8), node);
          prefetch_node(*nbx.tr, node);
        } else {
          Visits vc;
          traverse(nbx, node, qbox[q], a.dstat, [&](int prim) { hit(q, j, prim); }, vc);
          tally(nbx.tri, vc);
        }
      };
      // the roots
      for (int k = tid; k < nwork; k += CT) {
        const int q = work[k] & 0xff, j = work[k] >> 8;
        const NodeBoxes nbx = boxes_of(q, j);
        const int root = nbx.tri ? ntri[j] : nedge[j];
        const int L0 = nbx.tr->N - 1;
        Visits vc;
        if (root >= L0) {  // a tree of one leaf
          const int prim = __ldg(&nbx.tr->leaf_prim[root - L0]);
          ++vc.leaf;
          if (overlap(nbx.leaf(root, prim), qbox[q])) hit(q, j, prim);
        } else if (root >= 0) {
          ++vc.internal;
          if (overlap(nbx.internal(root), qbox[q])) push(fcur, q, j, root);
        }
        tally(nbx.tri, vc);
      }
      // the rounds
      for (;;) {
        __syncthreads();
        const int n = min(nfr[fcur], fcap);
        if (n == 0) break;
        const int nxt = fcur ^ 1;
        for (int e = tid; e < n; e += CT) {
          const int2 en = front[fcur][e];
          const int q = en.x & 0xff, j = en.x >> 8;
          const NodeBoxes nbx = boxes_of(q, j);
          Visits vc;
          expand_node(nbx, en.y, qbox[q], [&](int prim) { hit(q, j, prim); }, [&](int c) { push(nxt, q, j, c); }, vc);
          tally(nbx.tri, vc);
        }
        __syncthreads();
        if (lists && ncb >= kCandBuf / 2) flush();
        if (tid == 0) nfr[fcur] = 0;
        fcur = nxt;
      }
    }
  }
  if constexpr (lists) {
    __syncthreads();
    flush();
  }
  if constexpr (gh) return;
  if (ls && a.prof) {  // kernel profiling: the data this chunk read and wrote
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      pf_node += __shfl_xor_sync(0xffffffffu, pf_node, o);
      pf_tri += __shfl_xor_sync(0xffffffffu, pf_tri, o);
      pf_edge += __shfl_xor_sync(0xffffffffu, pf_edge, o);
      pf_cand += __shfl_xor_sync(0xffffffffu, pf_cand, o);
    }
    unsigned long long* row = a.prof_rows + 8 * (blockIdx.x & 31);
    if ((tid & 31) == 0) {
      atomicAdd(&row[PF_NODE], (unsigned long long)pf_node);
      atomicAdd(&row[PF_TRI], (unsigned long long)pf_tri);
      atomicAdd(&row[PF_EDGELEAF], (unsigned long long)pf_edge);
      atomicAdd(&row[PF_CAND], (unsigned long long)pf_cand);
    }
  }
  __syncthreads();
  if (tid == 0) {
    if constexpr (ls) {
      if (a.gtime) atomicMax(&a.gtime[1], globaltimer_ns());
    }
    if constexpr (ccd) {
      if (tkey) atomicMax(a.toi_key, tkey);
    } else {
      const long long* src = reinterpret_cast<const long long*>(&xe);
      long long* dst = reinterpret_cast<long long*>(a.energy);
      for (int e = 0; e < kXD; ++e)
        if (src[e]) atomicAdd((unsigned long long*)&dst[e], (unsigned long long)src[e]);
      if (src[kXD]) atomicOr((unsigned long long*)&dst[kXD], (unsigned long long)src[kXD]);
    }
  }
}

// Times of impact of the CCD candidates, one thread per candidate (ccd.py:20-40, 133-186);
// the minimum below 1 goes to the mailbox key.  LS: the candidates are the line-search
// candidates of a CCD_LS pass, and each is first put to the CCD pass's own culling
// predicate: the exact swept body boxes overlap and the two swept primitive boxes overlap;
// block 0 also clears the energies of the line-search batch that follows the pass.
template <bool LS>
__global__ void __launch_bounds__(128) k_ccd_eval(NarrowArgs a) {
  if (LS && blockIdx.x == 0) {
    static_assert(sizeof(XSum) == (kXD + 1) * sizeof(long long), "XSum layout");
    for (int i = threadIdx.x; i < kLsMax * (kXD + 1); i += blockDim.x)
      reinterpret_cast<long long*>(a.ls_energy)[i] = 0;
  }
  const int n = LS ? min(a.dstat[DS_NECAND], a.cap_ecand) : min(a.dstat[DS_NCCD], a.cap_ccd);
  if (a.dstat[DS_STATUS] & (LS ? ST_ECAND_OVERFLOW : ST_CCD_OVERFLOW)) return;
  const int4* cand = LS ? a.ecand : a.ccd_cand;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int4 c = cand[k];
    int ids[4];
    cand_vertices(a, c.x, c.y, c.z, ids);
    if (LS) {
      const int bA = __ldg(&a.vbody[ids[0]]), bB = __ldg(&a.vbody[ids[c.x == 0 ? 1 : 2]]);
      if (!overlap(load_box(&a.body_box[bA]), load_box(&a.body_box[bB]))) continue;
      const double dhh = 0.5 * a.prm.dhat;
      const bool hit = c.x == 0 ? overlap(point_box(a.y0, a.y1, c.y, (float)a.prm.dhat), tri_leaf_box(a.tris, a.y0, a.y1, c.z))
                                : overlap(edge_leaf_box(a.edges, a.y0, a.y1, c.y, dhh),
                                          edge_leaf_box(a.edges, a.y0, a.y1, c.z, dhh));
      if (!hit) continue;
    }
    d3 x0[4], x1[4];
    fetch(a.y0, ids, x0);
    fetch(a.y1, ids, x1);
    const double t = collision_time(c.x, x0, x1, a.prm.ipc_full != 0);
    if (t < 1.0) toi_min(a.toi_key, t);
  }
}

// Sets dint[kSupValid] (gh_superset_check); one CTA
__global__ void k_sup_check(int n, const double* A0, const double* p0, const double* q_last, const int* have,
                            int* valid, int mode) {
  __shared__ int ok;
  if (threadIdx.x == 0) ok = mode == 2 ? 1 : (mode == 1 ? (*have != 0) : 0);
  __syncthreads();
  if (mode == 1 && ok)
    for (int i = threadIdx.x; i < 12 * n; i += blockDim.x) {
      const double v = i < 9 * n ? A0[i] : p0[i - 9 * n];
      if (__double_as_longlong(v) != __double_as_longlong(q_last[i])) ok = 0;
    }
  __syncthreads();
  if (threadIdx.x == 0) *valid = ok;
}

// The friction contacts of the GH pass, one thread per lagged contact: each joins its body
// pair's contact list (found in the adjacency) as a pseudo-contact (y = kFricContact, z = its
// record); the pair assembly adds its friction terms to the pair's exact sums.  They are not
// active contacts (DS_ACTIVE is compensated for the contact scan's count).
__global__ void __launch_bounds__(128) k_fric_pairs(NarrowArgs a) {
  if (a.dstat[DS_STATUS] & (ST_PAIR_OVERFLOW | ST_CONTACT_OVERFLOW | ST_FRIC_OVERFLOW)) return;
  const int n = min(a.dstat[DS_NFRIC], a.cap_fric);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int I = a.fric[k].I, J = a.fric[k].J, lo = min(I, J), hi = max(I, J);
    int pr = -1;
    const int k1 = min(a.row_ptr[lo + 1], a.cap_adj);
    for (int q = a.row_ptr[lo]; q < k1 && pr < 0; ++q)
      if (a.adj_col[q] == hi) pr = a.adj_pair[q];
    if (pr < 0) continue;
    const int pos = atomicAdd(&a.dstat[DS_NCONTACT], 1);
    if (pos < a.cap_contacts) a.contacts[pos] = make_int4(pr, kFricContact, k, 0);
    else atomicOr(&a.dstat[DS_STATUS], ST_CONTACT_OVERFLOW);
    atomicAdd(&a.pair_cand[4 * pr + 1], 1);
    atomicSub(&a.dstat[DS_ACTIVE], 1);
  }
}

// The friction potential of every lagged contact at the pass's positions y0, into the pass's
// exact energy (the energy pass), one thread per contact
__global__ void __launch_bounds__(128) k_fric_energy(NarrowArgs a) {
  const int n = min(a.dstat[DS_NFRIC], a.cap_fric);
  XSum en;
  xs_zero(en);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const FricRec& f = a.fric[k];
    double x12[12];
    for (int q = 0; q < 12; ++q) x12[q] = a.y0[3 * f.ids[q / 3] + q % 3];
    const double e = ipc::friction_d(lag_of(f), x12, f.xt, a.prm.friction_mu, a.prm.friction_epsv * a.prm.dt);
    if (e != 0.0) xs_add(en, e);
  }
  xs_warp_sum(en);
  if ((threadIdx.x & 31) == 0) {
    long long* d = reinterpret_cast<long long*>(a.energy);
#pragma unroll
    for (int i = 0; i < kXD; ++i)
      if (en.d[i]) atomicAdd((unsigned long long*)&d[i], (unsigned long long)en.d[i]);
    if (en.flags) atomicOr((unsigned long long*)&d[kXD], (unsigned long long)en.flags);
  }
}

// The candidates of the tree traversal (when the kept line-search candidates did not cover the
// pass; k_gh_scan evaluates them otherwise), one thread per candidate
__global__ void __launch_bounds__(128) k_gh_eval(NarrowArgs a) {
  if (*a.sup_valid || (a.dstat[DS_STATUS] & (ST_CCD_OVERFLOW | ST_PAIR_OVERFLOW))) return;
  const int n = min(a.dstat[DS_NCCD], a.cap_ccd);
  int cpt = 0, cee = 0;
  XSum en;  // the candidates' barrier energy (ipcsk/energy.py:9-48)
  xs_zero(en);
  const bool with_energy = gh_with_energy(a), lag = gh_lag(a);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int4 c = a.ccd_cand[k];
    int ids[4];
    d3 xs[4];
    cand_vertices(a, c.y & 1, c.z, c.w, ids);
    fetch(a.y0, ids, xs);
    gh_candidate(a, c, ids, xs, with_energy, lag, cpt, cee, en);
  }
  gh_flush(a, cpt, cee, en, with_energy);
}

// The GH pass's candidates without a traversal, when the kept line-search candidates hold
// every pair its culling can produce (sup_valid): the pass's DOFs lie on the segment the step's
// last CCD pass covered (the accepted step q - alpha dq, 0 <= alpha <= 1).  Each candidate is
// put to the GH pass's own culling predicate -- the exact body boxes overlap and the static
// primitive boxes overlap (culling2.py:32-79, 213-227) -- and evaluated as the traversal's
// candidates are, with its pair index from the adjacency of the point's (or lower edge's) body.
__global__ void __launch_bounds__(128) k_gh_scan(NarrowArgs a) {
  if (!*a.sup_valid || (a.dstat[DS_STATUS] & (ST_CCD_OVERFLOW | ST_PAIR_OVERFLOW))) return;
  const int n = min(a.dstat[DS_NECAND], a.cap_ecand);
  const float dhf = (float)a.prm.dhat;
  const double dhh = 0.5 * a.prm.dhat;
  int cpt = 0, cee = 0;
  XSum en;
  xs_zero(en);
  const bool with_energy = gh_with_energy(a), lag = gh_lag(a);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int4 c = a.ecand[k];
    const int type = c.x, pa = c.y, pb = c.z;
    int ids[4];
    cand_vertices(a, type, pa, pb, ids);
    const int I = __ldg(&a.vbody[ids[0]]), J = __ldg(&a.vbody[ids[type == 0 ? 1 : 2]]);
    if (!overlap(load_box(&a.body_box[I]), load_box(&a.body_box[J]))) continue;
    const bool hit = type == 0 ? overlap(point_box(a.y0, nullptr, pa, dhf), tri_leaf_box(a.tris, a.y0, nullptr, pb))
                               : overlap(edge_leaf_box(a.edges, a.y0, nullptr, pa, dhh),
                                         edge_leaf_box(a.edges, a.y0, nullptr, pb, dhh));
    if (!hit) continue;
    // row I of the adjacency lists its neighbours in increasing order
    int lo = a.row_ptr[I], hi = min(a.row_ptr[I + 1], a.cap_adj) - 1, pr = -1;
    while (lo <= hi) {
      const int mid = (lo + hi) >> 1, col = a.adj_col[mid];
      if (col == J) {
        pr = a.adj_pair[mid];
        break;
      }
      if (col < J) lo = mid + 1;
      else hi = mid - 1;
    }
    if (pr < 0) continue;  // (the body boxes overlap, so the pair is listed)
    const int swap = (type == 0 && I > J) ? 1 : 0;
    d3 xs[4];
    fetch(a.y0, ids, xs);
    gh_candidate(a, make_int4(pr, type | (swap << 1), pa, pb), ids, xs, with_energy, lag, cpt, cee, en);
  }
  gh_flush(a, cpt, cee, en, with_energy);
}

__global__ void __launch_bounds__(128) k_list_gh(const __grid_constant__ NarrowArgs a) { list_gh_pass(a, (int)blockIdx.x, (int)gridDim.x); }

// ---------------------------------------------------------------------------------------
// per-body kernels
// ---------------------------------------------------------------------------------------
constexpr int BT = 160;
__global__ void __launch_bounds__(BT) k_body_gh(const __grid_constant__ BodyArgs a) {
  if (a.dstat[DS_STATUS] & kRerunMask) return;  // (a short list: the pass is made again)
  __shared__ BodyShared S;
  body_gh_pass(a, (int)blockIdx.x, S);
}

__global__ void k_vg_list(BodyArgs a) {
  const int b = blockIdx.x;
  const Box bb = load_box(&a.body_box[b]);
  for (int v = a.voff[b] + threadIdx.x; v < a.voff[b + 1]; v += blockDim.x) {
    if (!vg_candidate(a, bb, a.y, a.y1, v)) continue;
    const int pos = atomicAdd(&a.dstat[DS_VG_COUNT], 1);
    if (pos < a.cap_vg) {
      a.vg_list[2 * pos] = b;
      a.vg_list[2 * pos + 1] = v;
    } else {
      atomicOr(&a.dstat[DS_STATUS], ST_VG_OVERFLOW);
    }
  }
}

// exported blocks follow the solver's view: pairs without active contacts or touching a fixed
// (Dirichlet) body have no coupling block
__global__ void k_export_off(int np, const int* pair_active, const int* fixed, const double* offdiag, const int2* ij,
                             double* out, int* ijout, int cap) {
  const int p = blockIdx.x;
  if (p >= np || p >= cap) return;
  const bool live = pair_active[p] > 0 && !fixed[ij[p].x] && !fixed[ij[p].y];
  for (int e = threadIdx.x; e < 144; e += blockDim.x) out[(size_t)p * 144 + e] = live ? offdiag[(size_t)p * 288 + e] : 0.0;
  if (threadIdx.x == 0 && ijout) {
    ijout[2 * p] = ij[p].x;
    ijout[2 * p + 1] = ij[p].y;
  }
}

// (Ao, po) = (A, p) - alpha dq (alpha_dev: the step length on the device); also into (Ao2, po2)
// when given
__global__ void k_update_dofs(int n, const double* A, const double* p, const double* dq, double alpha, double* Ao,
                              double* po, const double* alpha_dev, double* Ao2, double* po2) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  update_body_dofs(b, A, p, dq, alpha_dev ? *alpha_dev : alpha, Ao, po, Ao2, po2);
}

__global__ void k_finish(int n, double dt, abd_states st) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  for (int k = 0; k < 3; ++k) {
    st.pdot[3 * b + k] = (st.p[3 * b + k] - st.p0[3 * b + k]) / dt;
    st.p0[3 * b + k] = st.p[3 * b + k];
  }
  for (int k = 0; k < 9; ++k) {
    st.Adot[9 * b + k] = (st.A[9 * b + k] - st.A0[9 * b + k]) / dt;
    st.A0[9 * b + k] = st.A[9 * b + k];
  }
}

// Exact dot products a.b and c.d (c may be null) on a fixed grid of kRedDot CTAs; the last CTA
// to finish sums the partials and writes the rounded results to out[0], out[1].
constexpr int kRedDot = 64;
__global__ void __launch_bounds__(256) k_dots(int N, const double* a, const double* b, const double* c,
                                              const double* d, XSum* part, int* count, double* out) {
  __shared__ XSum sh[8];
  __shared__ bool last;
  XSum x0, x1;
  xs_zero(x0);
  xs_zero(x1);
  for (int i = blockIdx.x * 256 + threadIdx.x; i < N; i += kRedDot * 256) {
    xs_add(x0, a[i] * b[i]);
    if (c) xs_add(x1, c[i] * d[i]);
  }
  xs_block_sum(x0, sh);
  xs_block_sum(x1, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = x0;
    part[kRedDot + blockIdx.x] = x1;
    __threadfence();
    last = atomicAdd(count, 1) == kRedDot - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = 0; k < (c ? 2 : 1); ++k) {
    XSum t;
    xs_zero(t);
    for (int i = threadIdx.x; i < kRedDot; i += 256) {
      const long long* q = reinterpret_cast<const long long*>(part + k * kRedDot + i);
#pragma unroll
      for (int j = 0; j < kXD; ++j) t.d[j] += __ldcg(q + j);
      t.flags |= __ldcg(q + kXD);
    }
    xs_block_sum(t, sh);
    if (threadIdx.x == 0) out[k] = xs_round(t);
  }
  if (threadIdx.x == 0) *count = 0;
}


// A chunk pass: the chunk filter, then the chunk kernel over the chunks with work (a grid of
// every chunk; the CTAs past the count return at once).  Counts the filter's launch.
template <int MODE>
cudaError_t chunk_pass(Sim& s, const NarrowArgs& a) {
  // (the body-box kernel of the pass cleared the filter's count)
  constexpr int per = KA / 32;
  k_chunk_active<MODE><<<(s.nch + per - 1) / per, KA, 0, s.stream>>>(a);
  k_chunk_narrow<MODE><<<s.nch, CT, 0, s.stream>>>(a);
  ++s.launches;
  return cudaGetLastError();
}

}  // namespace

// the active contacts grouped by body pair, then the pairs' blocks
static cudaError_t group_and_assemble(Sim& s, const NarrowArgs& a) {
  if (a.fric) {
    k_fric_pairs<<<scene_grid(s, 512, kRedBlocks), 128, 0, s.stream>>>(a);
    ++s.launches;
  }
  const bool one_cta = s.cap_contacts <= kScanScatter;
  k_contact_scan<<<1, 1024, 0, s.stream>>>(s.cap_pairs, s.pair_cand, s.dstat, s.cap_contacts,
                                           one_cta ? s.contacts : nullptr, s.contacts_by_pair, s.pair_active);
  ++s.launches;
  if (!one_cta) {
    k_contact_scatter<<<blocks(s.cap_contacts, 256), 256, 0, s.stream>>>(s.cap_contacts, s.contacts, s.pair_cand,
                                                                         s.contacts_by_pair, s.dstat);
    ++s.launches;
  }
  return pair_assemble(s, a);
}

cudaError_t list_gh(Sim& s, const abd_states& st) {
  const NarrowArgs a = narrow_args(s, NARROW_GH, st.A, st.p, nullptr, nullptr, nullptr, nullptr, nullptr);
  k_list_gh<<<scene_grid(s, 128, kRedBlocks), 128, 0, s.stream>>>(a);
  ++s.launches;
  return group_and_assemble(s, a);
}

// The tree traversal that makes the kept list: the line-search candidate traversal over the region
// (its DOFs in fdof and body_sup, its pairs in the adjacency: list_build)
cudaError_t list_traverse(Sim& s) {
  NarrowArgs a = narrow_args(s, NARROW_CCD_LS, s.reg, s.reg, s.reg, s.reg, s.x, s.xk, nullptr);
  a.make_list = 1;
  const cudaError_t e = chunk_pass<NARROW_CCD_LS>(s, a);
  ++s.launches;
  return e;
}

cudaError_t narrow(Sim& s, int mode, const double* A, const double* p, const double* A1, const double* p1,
                   const double* y0, const double* y1, const abd_states* st) {
  const NarrowArgs a = narrow_args(s, mode, A, p, A1, p1, y0, y1, st);
  if (mode == NARROW_ENERGY || mode == NARROW_CCD || mode == NARROW_CCD_LS || mode == NARROW_GH) {
    // energy, CCD and GH always run at DOFs; the energy needs the states (inertia terms)
    if (!a.affine || (mode == NARROW_ENERGY && !(st && st->A0 && st->Adot && st->p0 && st->pdot)))
      return cudaErrorInvalidValue;
    if (s.nch == 0) return cudaSuccess;
    if (mode == NARROW_ENERGY) {
      if (cudaError_t e = chunk_pass<NARROW_ENERGY>(s, a)) return e;
      if (a.fric) {  // the friction potential of the step's lagged contacts
        k_fric_energy<<<kRedBlocks, 128, 0, s.stream>>>(a);
        ++s.launches;
      }
    } else if (mode == NARROW_CCD || mode == NARROW_CCD_LS) {
      // (the body-box kernel of the pass cleared DS_NCCD and DS_NECAND)
      cudaError_t e = cudaSuccess;
      if (mode == NARROW_CCD_LS) {
        if (!a.y1) return cudaErrorInvalidValue;
        if (s.prof_events > 0 && record_event(s.prof_ev[0], s.stream))
          return cudaErrorUnknown;
        if ((e = chunk_pass<NARROW_CCD_LS>(s, a)) != cudaSuccess) return e;
        if (s.prof_events > 0 && record_event(s.prof_ev[1], s.stream))
          return cudaErrorUnknown;
        k_ccd_eval<true><<<kRedBlocks, 128, 0, s.stream>>>(a);
      } else {
        if ((e = chunk_pass<NARROW_CCD>(s, a)) != cudaSuccess) return e;
        k_ccd_eval<false><<<kRedBlocks, 128, 0, s.stream>>>(a);
      }
      ++s.launches;
    } else {
      // (the pass's pair scan cleared the per-pair contact counts, DS_NCONTACT, DS_NCCD and
      // DS_NACTP; the contact scan sets the offsets and scatter counters)
      cudaError_t e = cudaSuccess;
      if ((e = chunk_pass<NARROW_GH>(s, a)) != cudaSuccess) return e;
      k_gh_eval<<<kRedBlocks, 128, 0, s.stream>>>(a);
      ++s.launches;
      k_gh_scan<<<kRedBlocks, 128, 0, s.stream>>>(a);
      ++s.launches;
      if ((e = group_and_assemble(s, a)) != cudaSuccess) return e;
    }
  } else {
    if (s.cap_pairs == 0) return cudaSuccess;
    k_pair_lists<<<s.cap_pairs, NT, 0, s.stream>>>(a);
  }
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t prepare_narrow(Sim& s) {
  (void)s;
  return prepare_assemble();
}

cudaError_t gh_superset_check(Sim& s, const abd_states* st, int mode) {
  k_sup_check<<<1, 1024, 0, s.stream>>>(s.n, st ? st->A0 : nullptr, st ? st->p0 : nullptr, s.q_last,
                                        s.dint + kSupHave, s.dint + kSupValid, st ? mode : 0);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t body_gh(Sim& s, const abd_states& st, const double* A, const double* p, const double* y) {
  k_body_gh<<<s.n, BT, 0, s.stream>>>(body_args(s, &st, A, p, y, nullptr));
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t vg_list(Sim& s, const double* y0) {
  if (!(s.prm.ground_enabled && s.prm.enable_vg)) return cudaSuccess;
  k_vg_list<<<s.n, 128, 0, s.stream>>>(body_args(s, nullptr, nullptr, nullptr, y0, nullptr));
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t vg_list_swept(Sim& s, const double* y0, const double* y1) {
  if (!(s.prm.ground_enabled && s.prm.enable_vg)) return cudaSuccess;
  k_vg_list<<<s.n, 128, 0, s.stream>>>(body_args(s, nullptr, nullptr, nullptr, y0, y1));
  ++s.launches;
  return cudaGetLastError();
}

// Pair q of the exact set x_ij in a system numbered by the kept list's pairs, looked up in the adjacency
// (row I lists its neighbours in increasing order): its blocks and active contacts (none when it is
// not listed: the list holds every pair that has a contact)
__global__ void __launch_bounds__(128) k_gather_blocks(const int2* x_ij, const int* row_ptr, const int* adj_col,
                                                       const int* adj_pair, const int* pair_active,
                                                       const double* offdiag, double* x_off, int* x_act) {
  const int q = blockIdx.x;
  const int2 ij = x_ij[q];
  int pr = -1;
  for (int lo = row_ptr[ij.x], hi = row_ptr[ij.x + 1] - 1; lo <= hi && pr < 0;) {
    const int mid = (lo + hi) >> 1, col = adj_col[mid];
    if (col == ij.y) pr = adj_pair[mid];
    else if (col < ij.y) lo = mid + 1;
    else hi = mid - 1;
  }
  const bool live = pr >= 0 && pair_active[pr] > 0;
  for (int e = threadIdx.x; e < 288; e += blockDim.x) x_off[(size_t)q * 288 + e] = live ? offdiag[(size_t)pr * 288 + e] : 0.0;
  if (threadIdx.x == 0) x_act[q] = live ? pair_active[pr] : 0;
}

cudaError_t gather_blocks(Sim& s, int n_pairs) {
  if (n_pairs == 0) return cudaSuccess;
  k_gather_blocks<<<n_pairs, 128, 0, s.stream>>>(s.x_ij, s.row_ptr, s.adj_col, s.adj_pair, s.pair_active, s.offdiag,
                                                 s.x_off, s.x_act);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t export_system(Sim& s, double* off_dev, int* ij_dev, int cap) {
  const int have = s.sys_list ? s.x_n : std::min(s.n_pairs, s.cap_pairs), np = std::min(have, cap);
  if (np <= 0) return cudaSuccess;
  if (s.sys_list)
    k_export_off<<<np, 128, 0, s.stream>>>(np, s.x_act, s.fixed, s.x_off, s.x_ij, off_dev, ij_dev, cap);
  else
    k_export_off<<<np, 128, 0, s.stream>>>(np, s.pair_active, s.fixed, s.offdiag, s.ij, off_dev, ij_dev, cap);
  ++s.launches;
  return cudaGetLastError();
}

cudaError_t update_dofs(Sim& s, const double* A, const double* p, const double* dq, double alpha, double* Aout,
                        double* pout) {
  k_update_dofs<<<blocks(s.n, 128), 128, 0, s.stream>>>(s.n, A, p, dq, alpha, Aout, pout, nullptr, nullptr, nullptr);
  ++s.launches;
  return cudaGetLastError();
}


// k_finish, unless the device loop stopped for a rerun (the states are then left as they
// were).  The host loop's kept candidates are gone (the line search's were replaced).
__global__ void k_finish_dev(int n, double dt, abd_states st, const int* dstat, int* sup_have) {
  if (dstat[DS_STATUS] & kRerunMask) return;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < n) {
    for (int k = 0; k < 3; ++k) {
      st.pdot[3 * b + k] = (st.p[3 * b + k] - st.p0[3 * b + k]) / dt;
      st.p0[3 * b + k] = st.p[3 * b + k];
    }
    for (int k = 0; k < 9; ++k) {
      st.Adot[9 * b + k] = (st.A[9 * b + k] - st.A0[9 * b + k]) / dt;
      st.A0[9 * b + k] = st.A[9 * b + k];
    }
  }
  if (b == 0) *sup_have = 0;
}

cudaError_t finish_step_dev(Sim& s, const abd_states& st, double* xview) {
  k_finish_dev<<<blocks(s.n, 128), 128, 0, s.stream>>>(s.n, s.prm.dt, st, s.dstat, s.dint + kSupHave);
  ++s.launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !xview) return e;
  return transform(s, st.A0, st.p0, xview);
}

cudaError_t finish_step(Sim& s, const abd_states& st, double* xview) {
  k_finish<<<blocks(s.n, 128), 128, 0, s.stream>>>(s.n, s.prm.dt, st);
  ++s.launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !xview) return e;
  return transform(s, st.A0, st.p0, xview);
}

cudaError_t dots(Sim& s, const double* a, const double* b, const double* c, const double* d, double* out_dev,
                 cudaStream_t st) {
  static_assert(2 * kRedDot <= 2 * kRedBlocks, "dot partials fit two reduction slots");
  k_dots<<<kRedDot, 256, 0, st ? st : s.stream>>>(12 * s.n, a, b, c, d, s.partials + 10 * (size_t)kRedBlocks,
                                        s.red_count + 10, out_dev);
  ++s.launches;
  return cudaGetLastError();
}

}  // namespace abd
