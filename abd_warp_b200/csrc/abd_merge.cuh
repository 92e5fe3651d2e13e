// The merging rounds of the preconditioner's clustering (abd_precond.cuh), without CUDA headers: the
// threads that share the work come as a Team, so the host tests run the same code.
#pragma once

#if defined(__CUDACC__)
#define ABD_TEAM __device__ __forceinline__
#else
#define ABD_TEAM inline
#endif

namespace abd {
namespace precond {

// Rounds in which every cluster picks its strongest admissible pair to another cluster (make_clusters
// describes the rule): w.label [n] in: each body's own index, out: its cluster's first body; w.size in:
// 1, out: the clusters' bodies (at their first).  Team: id() of size() threads; sync(), a barrier
// after which all see what was written before it; any(p), a barrier that also tells every thread
// whether p held for one of them; best(p, key), the atomic maximum.
// A round's end must be the same for every thread, so it is any()'s result, which each thread holds
// itself.  (A shared flag, read after one barrier and cleared before the next, ended the rounds
// for a thread that read it late: the threads then waited at different barriers.)
template <class Team, class Pair, class Work>
ABD_TEAM void merge_rounds(const Team& t, int n, int cap, int rounds, const Pair* act, int m, const Work& w) {
  for (int round = 0; cap > 1 && round < rounds; ++round) {
    for (int b = t.id(); b < n; b += t.size()) {
      w.best[b] = 0ULL;
      w.to[b] = b;
    }
    t.sync();
    for (int e = t.id(); e < m; e += t.size()) {
      const Pair q = act[e];
      const int a = w.label[q.y], b = w.label[q.z];
      if (a == b || w.size[a] + w.size[b] > cap) continue;
      const unsigned long long key = ((unsigned long long)(unsigned)q.w << 32) | (0xffffffffULL - (unsigned)q.x);
      t.best(&w.best[a], key);
      t.best(&w.best[b], key);
    }
    t.sync();
    // a cluster has one best pair, so it takes part in at most one merge of the round
    bool merged = false;
    for (int e = t.id(); e < m; e += t.size()) {
      const Pair q = act[e];
      const int a = w.label[q.y], b = w.label[q.z];
      if (a == b) continue;
      const unsigned long long key = ((unsigned long long)(unsigned)q.w << 32) | (0xffffffffULL - (unsigned)q.x);
      if (w.best[a] != key || w.best[b] != key) continue;
      const int r = a < b ? a : b, o = a < b ? b : a;
      w.to[o] = r;
      w.size[r] += w.size[o];
      merged = true;
    }
    if (!t.any(merged)) break;  // (no label changes)
    for (int b = t.id(); b < n; b += t.size()) w.label[b] = w.to[w.label[b]];
    t.sync();
  }
}

}  // namespace precond
}  // namespace abd
