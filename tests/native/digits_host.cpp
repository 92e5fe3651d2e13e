// Host build of the exact sums' digit arithmetic (abd_warp_b200/csrc/abd_digits.cuh) for the CPU tests.
#include "../../abd_warp_b200/csrc/abd_digits.cuh"

// a set of counters folded as a warp folds it (ds_fold): every lane reads before one writes
extern "C" void digits_fold(int* s) {
  int v[abd::kDSlots];
  for (int k = 0; k < abd::kDSlots; ++k) v[k] = s[k];
  for (int k = 0; k < abd::kDFlags; ++k)
    s[k] = v[k] - abd::ds_carry(v[k]) * (1 << abd::kDW) + (k ? abd::ds_carry(v[k - 1]) : 0);
}

// its limbs d [kXD], as ds_merge and ds_to_limbs add them; the counters past the last that they take
extern "C" int digits_limbs(const int* s, long long* d) {
  for (int i = 0; i < abd::kDTop; ++i) {
    int j;
    long long lo, hi;
    abd::ds_limb(i, s[i], j, lo, hi);
    d[j] += lo;
    if (j + 1 < abd::kXD) d[j + 1] += hi;
    else if (hi) return -1;
  }
  int past = 0;
  for (int i = abd::kDTop; i < abd::kDFlags; ++i) past += s[i] != 0;
  return past;
}
