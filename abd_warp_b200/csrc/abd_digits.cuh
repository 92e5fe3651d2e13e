// The digits of the exact sums (abd_exact.cuh, abd_warpsum.cuh), without CUDA headers: the host tests
// run the same arithmetic.
#pragma once

#if defined(__CUDACC__)
#define ABD_DIGITS __host__ __device__ __forceinline__
#else
#define ABD_DIGITS inline
#endif

namespace abd {

constexpr int kXD = 10;      // 32-bit digits (limbs of an XSum)
constexpr int kXB0 = -192;   // weight exponent of digit 0

constexpr int kDW = 14;                                // bits of a counter's digit
constexpr int kDN = (32 * kXD + kDW - 1) / kDW;        // digits of a term: 23
constexpr int kDFlags = 31;                            // counter of the flags (XS_*)
constexpr int kDSlots = 32;                            // counters of a sum
constexpr int kDTerms = 1 << 17;                       // terms a set of counters holds
// counters that a sum reaches: two above a term's digits (2^31 terms below 2^128)
constexpr int kDTop = kDN + 2;

// What counter value v carries to the counter above.  Rounded towards zero: what stays has v's sign,
// so a carry goes no higher than the sum's own magnitude.  (An arithmetic shift makes a negative
// value a positive rest and a carry of -1, which every further fold moves one counter up: a sum
// folded nine times lost its sign.)
ABD_DIGITS int ds_carry(int v) { return v / (1 << kDW); }

// counter i's value v in limbs: lo into limb j, hi into limb j + 1 (the top limb takes all of it: hi 0)
ABD_DIGITS void ds_limb(int i, int v, int& j, long long& lo, long long& hi) {
  j = kDW * i / 32;
  if (j >= kXD - 1) {
    j = kXD - 1;
    lo = (long long)v * (1LL << (kDW * i - 32 * j));  // i < kDTop: a shift of 48 at most
    hi = 0;
  } else {
    const long long w = (long long)v * (1LL << (kDW * i % 32));
    lo = w & 0xffffffffLL;
    hi = w >> 32;
  }
}

}  // namespace abd
