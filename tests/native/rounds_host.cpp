// Host build of the round loop's bound (abd_warp_b200/csrc/abd_rounds.cuh) for the CPU tests.
#include "../../abd_warp_b200/csrc/abd_rounds.cuh"

// A step whose iteration k (from 1) leaves the list's region leave[k - 1] times (a list made for an
// iteration holds it, so once at most; more stands for a list that does not): the rounds it
// makes, negated when the bound ended it.
extern "C" int rounds_host(int max_iter, const int* leave) {
  const int last = max_iter > 1 ? max_iter : 1;
  int it = 0, left = 0;
  for (int rounds = 1;; ++rounds) {
    bool again = false;
    while (it < last && !again) {
      if (left < leave[it]) {
        ++left;
        again = true;
      } else {
        ++it;
        left = 0;
      }
    }
    if (!again) return rounds;
    if (!abd::another_round(rounds, max_iter)) return -rounds;
  }
}
