// lgt_intsum.cuh -- sums of a few FP64 values with integer operations.
//
// GB300 issues 1.7 FP64 additions a clock and SM (measured) against about 96
// integer operations, so adding the neighbours of a row costs less as some
// twenty integer operations each, and the two pipes overlap.  Every column
// keeps one 64-bit accumulator in units of 2^-57 of the largest magnitude
// met so far; a mantissa is shifted to that unit and added with its sign,
// and one conversion at the end rounds the sum to FP64.  Bits below the unit
// are dropped: at most 2^-57 of the largest entry per term, where an FP64
// addition rounds at 2^-53 of its partial sum.  kMaxIntTerms 58-bit terms
// cannot overflow an accumulator; longer lists (no lattice whose sector fits
// has them, but a sector of few states might) add the rest in FP64.
// Infinities, NaNs,
// magnitudes within 2^15 of overflow and subnormal ranges take plain FP64
// additions instead (below 2^-1042 a value counts as zero).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace lgt {

constexpr int kMaxIntTerms = 31;

// s = sum of the W-column slices load(entry index) of lst[n0 .. n1), U of
// them in flight; SGN: bit 31 of an entry flips the sign.  At most
// kMaxIntTerms entries.
template <int W, int U, bool SGN, class Load>
__device__ __forceinline__ void int_sum_part(const uint32_t* lst, int n0, int n1, double (&s)[W],
                                        Load load) {
  long long acc[W];
  int top[W];  // largest high word without its sign
#pragma unroll
  for (int e = 0; e < W; ++e) {
    acc[e] = 0;
    top[e] = 0;
  }
  for (int n = n0; n < n1; n += U) {
    double v[U][W];
    uint32_t ent[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (n + u < n1) {
        ent[u] = lst[n + u];
        load(ent[u] & 0x7fffffffu, v[u]);
      } else {
        ent[u] = 0u;
#pragma unroll
        for (int e = 0; e < W; ++e) v[u][e] = 0.0;
      }
    }
#pragma unroll
    for (int e = 0; e < W; ++e) {
      int t = top[e];
#pragma unroll
      for (int u = 0; u < U; ++u) t = max(t, __double2hiint(v[u][e]) & 0x7fffffff);
      const int eb = t & 0x7ff00000, drop = (eb - (top[e] & 0x7ff00000)) >> 20;
      acc[e] >>= min(drop, 63);
      top[e] = t;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int hi = __double2hiint(v[u][e]);
        const uint32_t lo = uint32_t(__double2loint(v[u][e]));
        const int sh = min((eb - (hi & 0x7ff00000)) >> 20, 63);
        const uint32_t mh = (uint32_t(hi) & 0xfffffu) | 0x100000u;
        unsigned long long m =
            (static_cast<unsigned long long>((mh << 5) | (lo >> 27)) << 32) | (lo << 5);
        m >>= sh;
        const int neg = (SGN ? hi ^ int(ent[u]) : hi) >> 31;  // 0 or -1
        const unsigned long long sg = static_cast<unsigned long long>(static_cast<long long>(neg));
        acc[e] += static_cast<long long>((m ^ sg) - sg);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < W; ++e) {
    const int eb = top[e] & 0x7ff00000;
    s[e] = 0.0;
    if (eb >= (100 << 20) && eb <= (0x7ef << 20)) {
      // acc 2^(E - 1080) with E the largest exponent field: the field moves
      if (acc[e] != 0) {
        const double d = __ll2double_rn(acc[e]);
        s[e] = __hiloint2double(__double2hiint(d) + (eb - (1080 << 20)), __double2loint(d));
      }
    } else if (top[e] != 0) {
      for (int n = n0; n < n1; ++n) {
        double v[W];
        load(lst[n] & 0x7fffffffu, v);
        s[e] += (SGN && (lst[n] >> 31)) ? -v[e] : v[e];
      }
    }
  }
}

// The same for any number of entries.
template <int W, int U, bool SGN, class Load>
__device__ __forceinline__ void int_sum(const uint32_t* lst, int n0, int n1, double (&s)[W],
                                        Load load) {
  int_sum_part<W, U, SGN>(lst, n0, n1 - n0 > kMaxIntTerms ? n0 + kMaxIntTerms : n1, s, load);
  for (int n = n0 + kMaxIntTerms; n < n1; ++n) {  // the rest one by one
    double v[W];
    load(lst[n] & 0x7fffffffu, v);
#pragma unroll
    for (int e = 0; e < W; ++e) s[e] += (SGN && (lst[n] >> 31)) ? -v[e] : v[e];
  }
}

}  // namespace lgt
