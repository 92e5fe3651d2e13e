// Host build of the clustering's merging rounds (abd_warp_b200/csrc/abd_merge.cuh) for the CPU tests:
// the device code's loop run by host threads, some of which are held up after a barrier.
#include <pthread.h>
#include <unistd.h>

#include <random>
#include <thread>
#include <vector>

#include "../../abd_warp_b200/csrc/abd_merge.cuh"

namespace {

struct Pair {
  int x, y, z, w;  // pair index, body, body, weight bits
};
struct Work {
  int *label, *size, *to;
  unsigned long long* best;
};

struct Shared {
  pthread_barrier_t barrier;
  std::vector<int> said;
};

struct HostTeam {
  Shared* s;
  int me, n;
  std::mt19937* rng;
  int id() const { return me; }
  int size() const { return n; }
  void late() const {  // one thread in four goes on long after the others
    if ((*rng)() % 4 == 0) usleep(200);
  }
  void sync() const {
    pthread_barrier_wait(&s->barrier);
    late();
  }
  bool any(bool p) const {
    s->said[me] = p;
    pthread_barrier_wait(&s->barrier);
    bool r = false;
    for (int q : s->said) r = r || q;
    pthread_barrier_wait(&s->barrier);
    late();
    return r;
  }
  void best(unsigned long long* p, unsigned long long key) const {
    unsigned long long v = __atomic_load_n(p, __ATOMIC_RELAXED);
    while (v < key && !__atomic_compare_exchange_n(p, &v, key, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {
    }
  }
};

}  // namespace

// the rounds by `threads` host threads: act [m][4], label and size [n] as merge_rounds takes them
extern "C" void merge_host(int threads, unsigned seed, int n, int cap, int rounds, const int* act, int m, int* label,
                           int* size) {
  Shared sh;
  pthread_barrier_init(&sh.barrier, nullptr, threads);
  sh.said.assign(threads, 0);
  std::vector<int> to(n);
  std::vector<unsigned long long> best(n);
  const Work w{label, size, to.data(), best.data()};
  std::vector<std::thread> pool;
  for (int t = 0; t < threads; ++t)
    pool.emplace_back([&, t] {
      std::mt19937 rng(seed * 1000 + t);
      abd::precond::merge_rounds(HostTeam{&sh, t, threads, &rng}, n, cap, rounds, reinterpret_cast<const Pair*>(act), m, w);
    });
  for (std::thread& t : pool) t.join();
  pthread_barrier_destroy(&sh.barrier);
}
