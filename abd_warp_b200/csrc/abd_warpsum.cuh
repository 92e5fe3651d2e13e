// The exact sum of abd_exact.cuh over the threads of a CTA (or of a cluster's CTAs), for the
// chains of dot products that a solve waits on.
//
// A term (a 53-bit mantissa on the grid 2^kXB0) is split into at most five signed 14-bit digits,
// which the threads add to 32-bit counters in shared memory: a 32-bit shared atomic is native
// and merges equal addresses (measured 16 cycles for 16 warps on one address), where a 64-bit
// one is a compare-and-swap loop (700 cycles) and a butterfly over an XSum is 11 64-bit values
// in five rounds of shuffles.  A counter holds 2^17 digits.  One warp then rounds the total, a
// lane per digit (ds_round).
#pragma once

#include "abd_exact.cuh"

namespace abd {

// x into the counters s [kDSlots] (shared memory)
__device__ inline void ds_add(int* s, double x) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7ff);
  const unsigned long long frac = bits & 0xfffffffffffffULL;
  const bool neg = (bits >> 63) != 0;
  if (ex == 0x7ff) {
    atomicOr(&s[kDFlags], (int)(frac ? XS_NAN : (neg ? XS_NINF : XS_PINF)));
    return;
  }
  unsigned long long m = ex ? (frac | (1ULL << 52)) : frac;
  int sft = (ex ? ex : 1) - 1075 - kXB0;
  if (sft < 0) {
    m = sft > -64 ? m >> -sft : 0ULL;
    sft = 0;
  }
  if (!m) return;
  if (sft > 32 * kXD - 53 && sft + 63 - __clzll((long long)m) >= 32 * kXD) {
    atomicOr(&s[kDFlags], (int)XS_RANGE);
    return;
  }
  const int j = sft / kDW, o = sft - kDW * j;
  const unsigned long long lo = m << o;  // with hi: 66 bits
  const unsigned hi = o > 11 ? (unsigned)(m >> (64 - o)) : 0u;
  constexpr int M = (1 << kDW) - 1;
  const int d[5] = {(int)lo & M, (int)(lo >> kDW) & M, (int)(lo >> (2 * kDW)) & M, (int)(lo >> (3 * kDW)) & M,
                    (int)(lo >> (4 * kDW)) | (int)(hi << (64 - 4 * kDW))};
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if (d[k]) atomicAdd(&s[j + k], neg ? -d[k] : d[k]);
}

// The carries of a set of counters to the counters above (one warp), which makes room for more
// terms: after it, a counter is at most 2^17 + 2^kDW in magnitude, with the sign of what it held
__device__ inline void ds_fold(int* s) {
  const int lane = (int)(threadIdx.x & 31), v = s[lane], c = ds_carry(v);
  const int up = __shfl_up_sync(0xffffffffu, c, 1);
  __syncwarp();
  if (lane < kDFlags) s[lane] = v - c * (1 << kDW) + (lane ? up : 0);
}

// Counter i of the set s into the limbs (or flags) of an XSum in global memory (a thread per counter)
__device__ inline void ds_to_limbs(const int* s, int i, XSum* x) {
  const int v = s[i];
  if (!v) return;
  if (i == kDFlags) {
    atomicOr((unsigned long long*)&x->flags, (unsigned long long)v);
    return;
  }
  if (i >= kDTop) {  // (no sum reaches it)
    atomicOr((unsigned long long*)&x->flags, (unsigned long long)XS_RANGE);
    return;
  }
  int j;
  long long lo, hi;
  ds_limb(i, v, j, lo, hi);
  atomicAdd((unsigned long long*)&x->d[j], (unsigned long long)lo);
  if (hi) atomicAdd((unsigned long long*)&x->d[j + 1], (unsigned long long)hi);
}

// The counters of the set s added to a register accumulator
__device__ inline void ds_merge(XSum& x, const int* s) {
#pragma unroll
  for (int i = 0; i < kDTop; ++i) {
    int j;
    long long lo, hi;
    ds_limb(i, s[i], j, lo, hi);
    x.d[j] += lo;
    if (j + 1 < kXD) x.d[j + 1] += hi;
  }
  x.flags |= s[kDFlags];
}

// The sum whose digits (below 2^40 in magnitude) the warp's lanes hold, the flags in lane kDFlags,
// rounded to FP64 as xs_round rounds; every lane gets it.  The carries are resolved by all lanes
// at once: the positive and the negative digits each become a canonical number -- a digit's high
// bits go to the lanes above, and the carries of one that remain are those of an integer addition
// over the lanes' generate and propagate bits -- then their difference, with the borrows alike.
static __device__ __noinline__ double ds_round(long long acc) {
  constexpr unsigned kAll = 0xffffffffu, M = (1u << kDW) - 1u;
  const int lane = (int)(threadIdx.x & 31);
  const int fl = __shfl_sync(kAll, (int)acc, kDFlags);
  if (fl) {
    if (fl & (int)(XS_NAN | XS_RANGE)) return __longlong_as_double(0x7ff8000000000000LL);
    if (fl & (int)XS_PINF) return (fl & (int)XS_NINF) ? __longlong_as_double(0x7ff8000000000000LL) : INFINITY;
    return -INFINITY;
  }
  const long long d = lane < kDFlags ? acc : 0;
  auto canonical = [&](unsigned long long v) {  // v >= 0 per lane -> the lane's digit
    unsigned a = (unsigned)(v >> kDW) & M, b = (unsigned)(v >> (2 * kDW));
    a = __shfl_up_sync(kAll, a, 1);
    b = __shfl_up_sync(kAll, b, 2);
    unsigned t = ((unsigned)v & M) + (lane > 0 ? a : 0u) + (lane > 1 ? b : 0u);  // b below 2^12
    const unsigned c = __shfl_up_sync(kAll, t >> kDW, 1);                        // 0, 1 or 2
    t = (t & M) + (lane > 0 ? c : 0u);
    const unsigned G = __ballot_sync(kAll, t > M), P = __ballot_sync(kAll, t == M);
    const unsigned X = G | P, cy = (X + G) ^ X ^ G;  // carries into each lane
    return (int)((t + ((cy >> lane) & 1u)) & M);
  };
  const int p = canonical(d > 0 ? (unsigned long long)d : 0ULL);
  const int m = canonical(d < 0 ? (unsigned long long)-d : 0ULL);
  int e = p - m;
  const unsigned pos = __ballot_sync(kAll, e > 0), ngt = __ballot_sync(kAll, e < 0);
  if (!(pos | ngt)) return 0.0;
  const bool neg = ngt > pos;  // the highest nonzero digit decides
  if (neg) e = -e;
  const unsigned G = neg ? pos : ngt, X = G | ~(pos | ngt), bw = (X + G) ^ X ^ G;
  const unsigned g = (unsigned)(e - (int)((bw >> lane) & 1u)) & M;
  const unsigned nz = __ballot_sync(kAll, g != 0);
  const int h = 31 - __clz((int)nz);
  // the top digit and the four below it (70 bits, at least 57 of them from the top set bit), and
  // whether anything is left below
  const unsigned long long t4 = __shfl_sync(kAll, g, h);
  unsigned long long t3 = __shfl_sync(kAll, g, (h - 1) & 31), t2 = __shfl_sync(kAll, g, (h - 2) & 31),
                     t1 = __shfl_sync(kAll, g, (h - 3) & 31), t0 = __shfl_sync(kAll, g, (h - 4) & 31);
  if (h < 1) t3 = 0;
  if (h < 2) t2 = 0;
  if (h < 3) t1 = 0;
  if (h < 4) t0 = 0;
  const bool rest = h > 4 && (nz & ((1u << (h - 4)) - 1u)) != 0;
  const unsigned long long hi = (t4 << (2 * kDW)) | (t3 << kDW) | t2;  // 29 .. 42 bits
  const unsigned long long lo = (t1 << kDW) | t0;                      // 28 bits
  const int drop = 53 - (64 - __clzll((long long)hi));                 // bits of lo in the mantissa: 11 .. 24
  unsigned long long mant = (hi << drop) | (lo >> (2 * kDW - drop));
  const unsigned long long rem = lo & ((1ULL << (2 * kDW - drop)) - 1ULL), half = 1ULL << (2 * kDW - 1 - drop);
  if (rem > half || (rem == half && (rest || (mant & 1ULL)))) ++mant;
  // value = mant 2^(2 kDW - drop) 2^(kDW (h - 4) + kXB0), 2^52 <= mant <= 2^53: a normal number
  const int ex = 2 * kDW - drop + kDW * (h - 4) + kXB0 + 52 + 1023;
  const unsigned long long bits = ((unsigned long long)ex << 52) + (mant - (1ULL << 52));
  return __longlong_as_double((long long)(bits | (neg ? 1ULL << 63 : 0ULL)));
}

}  // namespace abd
