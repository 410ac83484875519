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
// additions instead; a row whose high words are all zero (values below
// 2^-1042, or zeros) is summed exactly in units of 2^-1074.  (The solvers'
// sums over a warp's lanes count such values as zeros.)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace lgt {

constexpr int kMaxIntTerms = 31;

// Whether values whose largest high word (sign cleared) is `top` can be
// summed in units of that exponent.
__device__ __forceinline__ bool fix_range(int top) {
  const int eb = top & 0x7ff00000;
  return eb >= (100 << 20) && eb <= (0x7ef << 20);
}
// v in units of 2^-57 of the exponent eb (a high word's exponent field, no
// smaller than v's), truncated towards zero; eor flips the sign by its bit 31.
__device__ __forceinline__ long long fix_of(double v, int eb, uint32_t eor = 0u) {
  const int hi = __double2hiint(v);
  const uint32_t lo = uint32_t(__double2loint(v));
  const int sh = min((eb - (hi & 0x7ff00000)) >> 20, 63);
  const uint32_t mh = (uint32_t(hi) & 0xfffffu) | 0x100000u;
  unsigned long long m =
      (static_cast<unsigned long long>((mh << 5) | (lo >> 27)) << 32) | (lo << 5);
  m >>= sh;
  const int neg = int(uint32_t(hi) ^ eor) >> 31;  // 0 or -1
  const unsigned long long sg = static_cast<unsigned long long>(static_cast<long long>(neg));
  return static_cast<long long>((m ^ sg) - sg);
}
// The FP64 value of a sum t of such terms: t 2^(E - 1080), E the exponent.
__device__ __forceinline__ double fix_to(long long t, int eb) {
  if (t == 0) return 0.0;
  const double d = __ll2double_rn(t);
  return __hiloint2double(__double2hiint(d) + (eb - (1080 << 20)), __double2loint(d));
}

// The sum of terms whose high words are all zero, from the sum t of their
// fix_of(v, 0): each is +-(2^57 + 32 m) for a value of +-m 2^-1074, so what
// is left of t modulo 2^57 is 32 times the sum of the +-m.
__device__ __forceinline__ double fix_tiny(long long t) {
  const long long m = static_cast<long long>(static_cast<unsigned long long>(t) << 7) >> 12;
  const double d = __longlong_as_double(m < 0 ? -m : m);
  return m < 0 ? -d : d;
}

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
      for (int u = 0; u < U; ++u) acc[e] += fix_of(v[u][e], eb, SGN ? ent[u] : 0u);
    }
  }
#pragma unroll
  for (int e = 0; e < W; ++e) {
    s[e] = 0.0;
    if (fix_range(top[e])) {
      s[e] = fix_to(acc[e], top[e] & 0x7ff00000);
    } else if (top[e] == 0) {
      s[e] = fix_tiny(acc[e]);
    } else {
      for (int n = n0; n < n1; ++n) {
        double v[W];
        load(lst[n] & 0x7fffffffu, v);
        s[e] += (SGN && (lst[n] >> 31)) ? -v[e] : v[e];
      }
    }
  }
}

// The sum over a warp of one double per lane (32 terms of 58 bits just fit):
// every lane gets it.
__device__ __forceinline__ double warp_sum_int(double v) {
  const int top = int(__reduce_max_sync(0xffffffffu, uint32_t(__double2hiint(v)) & 0x7fffffffu));
  if (top == 0) return 0.0;
  if (!fix_range(top)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  const int eb = top & 0x7ff00000;
  long long x = fix_of(v, eb);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return fix_to(x, eb);
}

// The warp totals of eight values per lane, value q in lanes 4 q .. 4 q + 3:
// three exchange steps halve the values, two finish them.  add(x, y), and
// shfl(x, lane mask), of type A.
template <class A, class Add, class Shfl>
__device__ __forceinline__ A warp_scatter8(const A* p, int lane, Add add, Shfl shfl) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  A k[4], h[2];
#pragma unroll
  for (int q = 0; q < 4; ++q) k[q] = add(b4 ? p[q + 4] : p[q], shfl(b4 ? p[q] : p[q + 4], 16));
#pragma unroll
  for (int q = 0; q < 2; ++q) h[q] = add(b3 ? k[q + 2] : k[q], shfl(b3 ? k[q] : k[q + 2], 8));
  A v = add(b2 ? h[1] : h[0], shfl(b2 ? h[0] : h[1], 4));
  v = add(v, shfl(v, 2));
  return add(v, shfl(v, 1));
}

// The same for doubles, by integers where their ranges allow.
__device__ __forceinline__ double warp_scatter8_int(const double* p, int lane) {
  int top[8];
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    top[q] = int(__reduce_max_sync(0xffffffffu, uint32_t(__double2hiint(p[q])) & 0x7fffffffu));
    ok = ok && (top[q] == 0 || fix_range(top[q]));
  }
  if (!ok)
    return warp_scatter8<double>(
        p, lane, [](double x, double y) { return x + y; },
        [](double x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); });
  long long x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = top[q] == 0 ? 0 : fix_of(p[q], top[q] & 0x7ff00000);
  const long long v = warp_scatter8<long long>(
      x, lane, [](long long y, long long z) { return y + z; },
      [](long long y, int o) { return __shfl_xor_sync(0xffffffffu, y, o); });
  int t = top[0];
#pragma unroll
  for (int q = 1; q < 8; ++q) t = (lane >> 2) == q ? top[q] : t;
  return fix_to(v, t & 0x7ff00000);
}

// int_sum_part for any number of entries.
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
