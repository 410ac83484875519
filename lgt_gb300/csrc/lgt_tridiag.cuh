// lgt_tridiag.cuh -- lowest eigenpair of the Lanczos tridiagonal T, on one
// warp: Sturm-count multisection (division-free recurrence) and inverse
// iteration, in FP64 or, for the FP32-mixed path, FP32; and the FP64 path's
// convergence check, which decides in FP32 and forms the FP64 pair by defect
// correction.  Used by the per-CTA solver (small.cu) and the panel solver's
// checks (krylov.cu, lanczos_grid.cu).
// The work array holds at least 3 * kTriMax doubles, z at least kTriMax.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace lgt {

constexpr int kTriMax = 64;  // largest Krylov dimension + 1

// Number of eigenvalues of the tridiagonal (a, b) below x: sign changes of
// the leading principal minors p_i = det(T_i - x I), from the three-term
// recurrence p_i = (a_i - x) p_{i-1} - b_{i-1}^2 p_{i-2} (bb holds b^2).
// Division-free (FP64 division is a long dependent chain on this part); the
// minors are rescaled by 2^-600 when they grow past 2^600; an exact zero
// takes the sign opposite to its predecessor.  Signs, zeros and magnitudes
// are read from the bit patterns (integer operations), so a step costs
// three FP64 operations.
__device__ __forceinline__ int sign_bit(double v) { return int(uint32_t(__double2hiint(v)) >> 31); }
__device__ __forceinline__ bool is_zero(double v) {
  return ((uint32_t(__double2hiint(v)) & 0x7fffffffu) | uint32_t(__double2loint(v))) == 0u;
}
__device__ __forceinline__ int exp_bits(double v) {
  return int((uint32_t(__double2hiint(v)) >> 20) & 0x7ffu);
}

__device__ inline int sturm_below(const double* a, const double* bb, int n, double x) {
  double p0 = 1.0, p1 = a[0] - x;
  int sp = 0;  // sign bit of the previous minor (p_{-1} = 1 > 0)
  int s1 = is_zero(p1) ? 1 - sp : sign_bit(p1);
  int cnt = (s1 != sp) ? 1 : 0;
  sp = s1;
  for (int i = 1; i < n; ++i) {
    double p2 = fma(a[i] - x, p1, -bb[i - 1] * p0);
    const int e2 = exp_bits(p2);
    if (e2 > 1023 + 600) {
      p2 *= 0x1.0p-600;
      p1 *= 0x1.0p-600;
    } else if (e2 < 1023 - 600 && exp_bits(p1) < 1023 - 600) {
      p2 *= 0x1.0p600;
      p1 *= 0x1.0p600;
    }
    const int s2 = is_zero(p2) ? 1 - sp : sign_bit(p2);
    cnt += (s2 != sp) ? 1 : 0;
    sp = s2;
    p0 = p1;
    p1 = p2;
  }
  return cnt;
}

// Lowest eigenpair of the n x n symmetric tridiagonal (a, b) by warp-parallel
// multisection of the Sturm count (32 probes per round) over the Gershgorin
// interval, then two inverse iterations on the positive-definite T - (theta -
// delta) I by lane 0, starting from ones.  Called by one full warp; bb (n
// entries of work space after the first kTriMax) and z are written by lane 0 /
// the warp.
__device__ inline double warp_lowest_eig(const double* a, const double* b, int n, double* z,
                                         double* work) {
  const int lane = threadIdx.x & 31;
  double* bb = work + 2 * kTriMax;
  for (int i = lane; i < n - 1; i += 32) bb[i] = b[i] * b[i];
  __syncwarp();
  double lo = a[0], hi = a[0];
  for (int i = 0; i < n; ++i) {
    const double r = ((i > 0) ? fabs(b[i - 1]) : 0.0) + ((i < n - 1) ? fabs(b[i]) : 0.0);
    lo = fmin(lo, a[i] - r);
    hi = fmax(hi, a[i] + r);
  }
  const double scale = fmax(fmax(fabs(lo), fabs(hi)), 1e-300);
  for (int it = 0; it < 40; ++it) {
    if (hi - lo <= 2.2e-16 * scale) break;
    const double step = (hi - lo) / 33.0;
    const double x = lo + step * double(lane + 1);
    const unsigned bal = __ballot_sync(0xffffffffu, sturm_below(a, bb, n, x) >= 1);
    if (bal) {
      const int L = __ffs(bal) - 1;
      const double nhi = lo + step * double(L + 1);
      const double nlo = (L > 0) ? lo + step * double(L) : lo;
      if (!(nhi < hi) && !(nlo > lo)) break;  // no progress at this precision
      hi = nhi;
      lo = nlo;
    } else {
      const double nlo = lo + step * 32.0;
      if (!(nlo > lo)) break;
      lo = nlo;
    }
  }
  const double theta = 0.5 * (lo + hi);
  // inverse iteration on the positive-definite T - (theta - delta) I: the
  // two triangular sweeps by lane 0 (factorisation merged into the forward
  // sweep, diagonal scaling into the backward one), operands read eight
  // entries ahead; the scaling by the whole warp
  const double shift = theta - 4.0 * 2.2e-16 * scale;
  double* d = work;  // reciprocal pivots
  double* l = work + kTriMax;
  for (int i = lane; i < n; i += 32) z[i] = 1.0;
  __syncwarp();
  for (int rep = 0; rep < 2; ++rep) {
    if (lane == 0) {
      double dprev = 0.0, bprev = 0.0, zprev = 0.0;
      for (int i0 = 0; i0 < n; i0 += 8) {
        double ac[8], bc[8], zc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u;
          ac[u] = (i < n) ? a[i] : 0.0;
          bc[u] = (i < n - 1) ? b[i] : 0.0;
          zc[u] = (i < n) ? z[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u;
          if (i < n) {
            double piv;
            if (i == 0) {
              piv = ac[u] - shift;
            } else {
              const double li = bprev * dprev;
              l[i - 1] = li;
              piv = (ac[u] - shift) - li * bprev;
              zc[u] = fma(-li, zprev, zc[u]);
            }
            if (piv <= 0.0) piv = 1e-300;
            const double di = 1.0 / piv;
            d[i] = di;
            z[i] = zc[u];
            dprev = di;
            bprev = bc[u];
            zprev = zc[u];
          }
        }
      }
      double znext = 0.0;
      for (int i1 = n - 1; i1 >= 0; i1 -= 8) {
        double zc[8], dc[8], lc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i1 - u;
          zc[u] = (i >= 0) ? z[i] : 0.0;
          dc[u] = (i >= 0) ? d[i] : 0.0;
          lc[u] = (i >= 0 && i < n - 1) ? l[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i1 - u;
          if (i >= 0) {
            double t = zc[u] * dc[u];
            if (i < n - 1) t = fma(-lc[u], znext, t);
            z[i] = t;
            znext = t;
          }
        }
      }
    }
    __syncwarp();
    double mx = 0.0;
    for (int i = lane; i < n; i += 32) mx = fmax(mx, fabs(z[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const double inv = 1.0 / mx;
    double nn = 0.0;
    for (int i = lane; i < n; i += 32) {
      const double zi = z[i] * inv;
      z[i] = zi;
      nn = fma(zi, zi, nn);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    const double in2 = 1.0 / sqrt(nn);
    for (int i = lane; i < n; i += 32) z[i] *= in2;
    __syncwarp();
  }
  const bool neg = z[0] < 0.0;
  __syncwarp();
  if (neg)
    for (int i = lane; i < n; i += 32) z[i] = -z[i];
  __syncwarp();
  return theta;
}

// FP32 counterpart of sturm_below for the mixed path's checks (minors
// rescaled by 2^-60 / 2^60 to stay inside the FP32 range).  The count is
// that of a matrix within a few FP32 ulps of T (Sturm counts by the LDL^T
// recurrence are backward stable), so brackets are reliable to ~1e-6 |T|.
__device__ inline int sturm_below_f(const float* a, const float* bb, int n, float x) {
  float p0 = 1.0f, p1 = a[0] - x;
  int sp = 0;
  int s1 = (p1 == 0.0f) ? 1 - sp : (p1 < 0.0f ? 1 : 0);
  int cnt = (s1 != sp) ? 1 : 0;
  sp = s1;
  for (int i = 1; i < n; ++i) {
    float p2 = fmaf(a[i] - x, p1, -bb[i - 1] * p0);
    if (fabsf(p2) > 0x1.0p60f) {
      p2 *= 0x1.0p-60f;
      p1 *= 0x1.0p-60f;
    } else if (fabsf(p2) < 0x1.0p-60f && fabsf(p1) < 0x1.0p-60f) {
      p2 *= 0x1.0p60f;
      p1 *= 0x1.0p60f;
    }
    const int s2 = (p2 == 0.0f) ? 1 - sp : (p2 < 0.0f ? 1 : 0);
    cnt += (s2 != sp) ? 1 : 0;
    sp = s2;
    p0 = p1;
    p1 = p2;
  }
  return cnt;
}

// Lowest eigenpair for the FP32-mixed path: as warp_lowest_eig, in FP32
// (GB300's FP64 pipe makes a one-warp FP64 recurrence a long latency
// chain).  theta is good to ~1e-6 |T| and z to FP32 accuracy: the FP32
// Krylov basis resolves no more, and the energy returned by the solver is
// the FP64 Rayleigh quotient of the final vector.  When warm, the previous
// lowest Ritz value th_prev (an upper bound: the lowest Ritz value only
// decreases as the Krylov space grows) and its residual r_prev bracket the
// search, [th_prev - 2 r_prev, th_prev], if Sturm counts confirm its ends;
// otherwise the Gershgorin interval is used.
__device__ inline double warp_lowest_eig_f32(const double* a64, const double* b64, int n,
                                             double* z, double* work, bool warm, double th_prev,
                                             double r_prev) {
  const int lane = threadIdx.x & 31;
  float* a = reinterpret_cast<float*>(work);
  float* b = a + kTriMax;
  float* bb = b + kTriMax;
  float* d = bb + kTriMax;
  float* l = d + kTriMax;
  float* zf = l + kTriMax;
  for (int i = lane; i < n; i += 32) {
    a[i] = float(a64[i]);
    const float bi = (i < n - 1) ? float(b64[i]) : 0.0f;
    b[i] = bi;
    bb[i] = bi * bi;
  }
  __syncwarp();
  // Gershgorin bounds: lane i covers rows i, i + 32
  float lo = 3.0e38f, hi = -3.0e38f;
  for (int i = lane; i < n; i += 32) {
    const float r = ((i > 0) ? fabsf(b[i - 1]) : 0.0f) + fabsf(b[i]);
    lo = fminf(lo, a[i] - r);
    hi = fmaxf(hi, a[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const float scale = fmaxf(fmaxf(fabsf(lo), fabsf(hi)), 1e-30f);
  lo -= 1e-6f * scale;  // FP32 rounding of the bounds
  hi += 1e-6f * scale;
  if (warm) {
    const float whi = fminf(hi, float(th_prev) + 4e-6f * scale);
    const float wlo = fmaxf(lo, float(th_prev) - fmaxf(2.0f * float(r_prev), 1e-5f * scale));
    const int c = sturm_below_f(a, bb, n, (lane == 0) ? wlo : whi);
    const int c_lo = __shfl_sync(0xffffffffu, c, 0), c_hi = __shfl_sync(0xffffffffu, c, 1);
    if (c_lo == 0 && c_hi >= 1) {
      lo = wlo;
      hi = whi;
    }
  }
  for (int it = 0; it < 24; ++it) {
    if (hi - lo <= 2e-7f * scale) break;
    const float step = (hi - lo) * (1.0f / 33.0f);
    const float x = lo + step * float(lane + 1);
    const unsigned bal = __ballot_sync(0xffffffffu, sturm_below_f(a, bb, n, x) >= 1);
    if (bal) {
      const int L = __ffs(bal) - 1;
      const float nhi = lo + step * float(L + 1);
      const float nlo = (L > 0) ? lo + step * float(L) : lo;
      if (!(nhi < hi) && !(nlo > lo)) break;
      hi = nhi;
      lo = nlo;
    } else {
      const float nlo = lo + step * 32.0f;
      if (!(nlo > lo)) break;
      lo = nlo;
    }
  }
  const float theta = 0.5f * (lo + hi);
  // inverse iteration on T - (theta - delta) I, positive definite: the two
  // triangular sweeps by lane 0 (the factorisation merged into the forward
  // sweep, the diagonal scaling into the backward one), each reading its
  // operands eight entries ahead so that the sweep waits on its arithmetic
  // rather than on shared-memory loads; the scaling by the whole warp
  const float shift = theta - 4e-7f * scale;
  for (int i = lane; i < n; i += 32) zf[i] = 1.0f;
  __syncwarp();
  for (int rep = 0; rep < 2; ++rep) {
    if (lane == 0) {
      float dprev = 0.0f, bprev = 0.0f, zprev = 0.0f;
      for (int i0 = 0; i0 < n; i0 += 8) {
        float ac[8], bc[8], zc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u;
          ac[u] = (i < n) ? a[i] : 0.0f;
          bc[u] = (i < n) ? b[i] : 0.0f;
          zc[u] = (i < n) ? zf[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i0 + u;
          if (i < n) {
            float piv;
            if (i == 0) {
              piv = ac[u] - shift;
            } else {
              const float li = bprev * dprev;
              l[i - 1] = li;
              piv = (ac[u] - shift) - li * bprev;
              zc[u] = fmaf(-li, zprev, zc[u]);
            }
            if (piv <= 0.0f) piv = 1e-30f;
            const float di = 1.0f / piv;
            d[i] = di;
            zf[i] = zc[u];
            dprev = di;
            bprev = bc[u];
            zprev = zc[u];
          }
        }
      }
      float znext = 0.0f;
      for (int i1 = n - 1; i1 >= 0; i1 -= 8) {
        float zc[8], dc[8], lc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i1 - u;
          zc[u] = (i >= 0) ? zf[i] : 0.0f;
          dc[u] = (i >= 0) ? d[i] : 0.0f;
          lc[u] = (i >= 0 && i < n - 1) ? l[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = i1 - u;
          if (i >= 0) {
            float t = zc[u] * dc[u];
            if (i < n - 1) t = fmaf(-lc[u], znext, t);
            zf[i] = t;
            znext = t;
          }
        }
      }
    }
    __syncwarp();
    float mx = 0.0f;
    for (int i = lane; i < n; i += 32) mx = fmaxf(mx, fabsf(zf[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float inv = 1.0f / mx;
    float nn = 0.0f;
    for (int i = lane; i < n; i += 32) {
      const float zi = zf[i] * inv;
      zf[i] = zi;
      nn = fmaf(zi, zi, nn);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    const float in2 = rsqrtf(nn);
    for (int i = lane; i < n; i += 32) zf[i] *= in2;
    __syncwarp();
  }
  const float sg = (zf[0] < 0.0f) ? -1.0f : 1.0f;
  for (int i = lane; i < n; i += 32) z[i] = double(sg * zf[i]);
  __syncwarp();
  return double(theta);
}

// ---- FP64 convergence check ---------------------------------------------------
//
// A dependent FP64 operation takes 64 cycles on GB300 (2 lanes a clock and
// SM), so the FP64 multisection of warp_lowest_eig costs about 150 000 cycles
// at n = 40 -- 45 % of a 4x2 FP64 solve at a check every five steps.  The
// check itself needs little precision:
//   * T - a_0 in FP32, multisection there (4-cycle operations);
//   * the bottom-up pivots u_i = d_i - s - b_i^2 / u_{i+1} at the lower end s
//     of the bracket (all positive but the top one) give the eigenvector by
//     its ratios z_i / z_{i-1} = -b_{i-1} / u_i: products, no differences, so
//     even a tail component of 1e-13 has a few FP32 ulps per factor.  The
//     shift lies up to 1e-6 of the spread below the eigenvalue: the residual
//     |beta_n z_n| is known to 3e-4 of itself where the start vector holds
//     1e-3 of the state or more, to 4e-3 at 1e-4 and a tenth at 2e-5; one
//     inverse iteration leaves 4e-6 (300 levels, the second one 1/38 of the
//     spread above).
// "Not converged" is decided by that residual (a wrong one costs steps, not
// accuracy).  A converged check, or one that must hand out the vector, goes on
// to FP64: one inverse iteration in FP32, then defect correction, the residual
// (T - theta) z in FP64 by all lanes, the correction from the FP32 pivots
// (projected against z), about six digits a round.  Clustered lowest eigenvalues (a second one within 4e-6 of the
// spread), a start vector with less than 1e-5 of the state (the ratios' tail
// is 10 % low there), ranges FP32 cannot hold and corrections that stall take
// warp_lowest_eig instead, at 260k (n = 33) to 440k cycles (n = 60), so none
// of these may be common: among 64 points of random start vectors one in two
// batches has a share below 1e-3 (whose pivots FP32 rounds to 10 % and the
// inverse iteration puts right).  A check (n = 25, warm): not converged 7.6k
// cycles (15.1k with the branching count), converged 28k; mixed 9.8k (18.2k).
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Solves (T - s) y = y through the bottom-up pivots (reciprocals ru, couplings
// bf): up, then down, by lane 0, operands read eight ahead.
__device__ __forceinline__ void pivot_solve(const float* bf, const float* ru, int n, float* y) {
  float yp = 0.0f;
  for (int i1 = n - 1; i1 >= 0; i1 -= 8) {
    float yc[8], c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i1 - q;
      yc[q] = (i >= 0) ? y[i] : 0.0f;
      c[q] = (i >= 0 && i < n - 1) ? bf[i] * ru[i + 1] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (i1 - q >= 0) {
        yp = fmaf(-c[q], yp, yc[q]);
        y[i1 - q] = yp;
      }
  }
  float xp = 0.0f;
  for (int i0 = 0; i0 < n; i0 += 8) {
    float yc[8], c[8], r[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = i0 + q;
      yc[q] = (i < n) ? y[i] : 0.0f;
      r[q] = (i < n) ? ru[i] : 0.0f;
      c[q] = (i > 0 && i < n) ? bf[i - 1] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (i0 + q < n) {
        xp = r[q] * fmaf(-c[q], xp, yc[q]);
        y[i0 + q] = xp;
      }
  }
}

// Whether the tridiagonal with diagonal d and squared couplings e (e[i]
// between i - 1 and i, e[0] = 0) has an eigenvalue below x: some leading minor
// of T - x is negative.  Arrays padded to a multiple of four with d = 8, e = 0
// and scaled to a spread of 1 to 2, so that four steps stay in range between
// the exact rescalings; no branches (the general count took 100 cycles a row).
__device__ __forceinline__ bool below_scaled(const float* d, const float* e, int n, float x) {
  float p0 = 0.0f, p1 = 1.0f;
  int neg = 0;
  for (int i = 0; i < n; i += 4) {
    const float4 D = *reinterpret_cast<const float4*>(d + i);
    const float4 E = *reinterpret_cast<const float4*>(e + i);
    const float q0 = fmaf(D.x - x, p1, -E.x * p0);
    const float q1 = fmaf(D.y - x, q0, -E.y * p1);
    p0 = fmaf(D.z - x, q1, -E.z * q0);
    p1 = fmaf(D.w - x, p0, -E.w * q1);
    neg |= __float_as_int(q0) | __float_as_int(q1) | __float_as_int(p0) | __float_as_int(p1);
    const int m =
        max(__float_as_int(p0) & 0x7f800000, __float_as_int(p1) & 0x7f800000);
    const float sc = __int_as_float(0x7f000000 - m);
    p0 *= sc;
    p1 *= sc;
  }
  return neg < 0;
}

// FP32 part: true when the FP32 data describe T's lowest pair (see above);
// theta relative to a[0] (*th), the vector's residual factor |z_{n-1}| / |z|
// (*tail), the power of two (*scale) that the FP32 matrix is T - a[0] times,
// and in work (16-byte aligned): its diagonal, squared couplings, couplings,
// reciprocal pivots and the normalised vector (five arrays of kTriMax
// floats).  warm: th_prev, r_prev are an earlier check's theta and residual;
// the lowest value lies in [th_prev - 2 r_prev, th_prev] unless the counts at
// its ends say otherwise.
__device__ inline bool warp_lowest_f32_pivots(const double* a, const double* b, int n,
                                              float* work, bool warm, double th_prev,
                                              double r_prev, float* th, float* tail,
                                              float* spread, float* scale) {
  const int lane = threadIdx.x & 31;
  float* d = work;
  float* ee = d + kTriMax;
  float* bf = ee + kTriMax;
  float* ru = bf + kTriMax;
  float* zf = ru + kTriMax;
  const double c0 = a[0];
  // rows lane and lane + 32: diagonal and the couplings on both sides
  float dv[2], bl[2], br[2];
  float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = lane + 32 * h;
    dv[h] = (i < n) ? float(a[i] - c0) : 0.0f;
    br[h] = (i < n - 1) ? float(b[i]) : 0.0f;
    bl[h] = (i > 0 && i < n) ? float(b[i - 1]) : 0.0f;
    if (i < n) {
      const float r = fabsf(bl[h]) + fabsf(br[h]);
      lo = fminf(lo, dv[h] - r);
      hi = fmaxf(hi, dv[h] + r);
    }
  }
  lo = -warp_max_f(-lo);  // Gershgorin
  hi = warp_max_f(hi);
  float width = hi - lo;
  if (!(width > 1e-15f && width < 1e15f && fabsf(lo) < 1e15f)) return false;
  *spread = width;
  const float sc = __int_as_float(0x7f000000 - (__float_as_int(width) & 0x7f800000));
  *scale = sc;
  lo *= sc;
  hi *= sc;
  width *= sc;  // in [1, 2)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = lane + 32 * h;
    const float l = bl[h] * sc;
    d[i] = (i < n) ? dv[h] * sc : 8.0f;
    ee[i] = l * l;
    bf[i] = br[h] * sc;
  }
  __syncwarp();
  lo -= 1e-6f * width;
  hi += 1e-6f * width;
  if (warm) {
    const float tp = float(th_prev - c0) * sc, rp = float(r_prev) * sc;
    const float whi = fminf(hi, tp + 2e-6f * width);
    const float wlo = fmaxf(lo, tp - fmaxf(2.0f * rp, 4e-6f * width));
    // the first round's probes include both ends
    const float step = (whi - wlo) * (1.0f / 31.0f);
    const float x = (lane == 31) ? whi : wlo + step * float(lane);
    const unsigned bal = __ballot_sync(0xffffffffu, below_scaled(d, ee, n, x));
    if (!(bal & 1u) && (bal >> 31)) {
      const int L = __ffs(bal) - 1;
      lo = wlo + step * float(L - 1);
      hi = (L == 31) ? whi : wlo + step * float(L);
    }
  }
  for (int it = 0; it < 12; ++it) {
    if (hi - lo <= 4e-7f * width) break;
    const float step = (hi - lo) * (1.0f / 33.0f);
    const float x = lo + step * float(lane + 1);
    const unsigned bal = __ballot_sync(0xffffffffu, below_scaled(d, ee, n, x));
    const int L = bal ? __ffs(bal) - 1 : 32;
    const float nlo = lo + step * float(L), nhi = (L < 32) ? lo + step * float(L + 1) : hi;
    if (!(nhi < hi) && !(nlo > lo)) break;
    if (L > 0) lo = nlo;
    hi = nhi;
  }
  const float s = lo - 4e-7f * width;
  // pivots and ratios from the bottom, by lane 0, operands read eight ahead
  int ok = 1;
  if (lane == 0) {
    float rn = 0.0f;
    const float small = 1e-6f * width;
    for (int i1 = n - 1; i1 >= 0; i1 -= 8) {
      float dc[8], bc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int i = i1 - q;
        dc[q] = (i >= 0) ? d[i] - s : 0.0f;
        bc[q] = (i >= 0 && i < n - 1) ? ee[i + 1] : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int i = i1 - q;
        if (i >= 0) {
          float un = fmaf(-bc[q], rn, dc[q]);
          // below the spectrum every pivot is positive; one of rounding size
          // (a start vector with little of the lowest state) moves the matrix
          // by no more than rounding when it is raised
          if (!(un > -small)) ok = 0;
          un = fmaxf(un, 0.1f * small);
          rn = __fdividef(1.0f, un);
          ru[i] = rn;
        }
      }
    }
    float z = 1.0f;
    for (int i0 = 0; i0 < n; i0 += 8) {
      float f[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int i = i0 + q;
        f[q] = (i > 0 && i < n) ? bf[i - 1] * ru[i] : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int i = i0 + q;
        if (i > 0) z = -z * f[q];
        if (i < n) zf[i] = z;
      }
    }
  }
  __syncwarp();
  ok = __shfl_sync(0xffffffffu, ok, 0);
  float m = 0.0f;
  for (int i = lane; i < n; i += 32) m = fmaxf(m, fabsf(zf[i]));
  m = warp_max_f(m);
  if (!ok || !(m < 1e15f)) return false;
  const float im = __fdividef(1.0f, m);
  float q = 0.0f;
  for (int i = lane; i < n; i += 32) q = fmaf(zf[i] * im, zf[i] * im, q);
  const float inv = im * rsqrtf(warp_sum_f(q));
  *tail = fabsf(zf[n - 1]) * inv;
  __syncwarp();
  for (int i = lane; i < n; i += 32) zf[i] *= inv;
  __syncwarp();
  // No second eigenvalue near the bracket.  It is above the lowest one of the
  // matrix without any one row (interlacing), here the row of the largest
  // component; if that is near too, by count.
  // (a start vector with less than 1e-5 of the state: the ratios are off)
  if (!(zf[0] > 1e-5f)) return false;
  const float top = 0.99f * m * inv;
  const unsigned b0 = __ballot_sync(0xffffffffu, lane < n && fabsf(zf[lane]) >= top);
  const unsigned b1 = __ballot_sync(0xffffffffu, lane + 32 < n && fabsf(zf[lane + 32]) >= top);
  const int row = b0 ? __ffs(b0) - 1 : (b1 ? __ffs(b1) + 31 : 0);
  const float x = hi + 4e-6f * width;
  const float od = d[row], oe = ee[row], on = (row + 1 < n) ? ee[row + 1] : 0.0f;
  __syncwarp();
  if (lane == 0) {
    d[row] = 8.0f;
    ee[row] = 0.0f;
    if (row + 1 < n) ee[row + 1] = 0.0f;
  }
  __syncwarp();
  if (below_scaled(d, ee, n, x)) {
    __syncwarp();
    if (lane == 0) {
      d[row] = od;
      ee[row] = oe;
      if (row + 1 < n) ee[row + 1] = on;
    }
    __syncwarp();
    if (sturm_below_f(d, ee + 1, n, x) > 1) return false;
  }
  *th = 0.5f * (lo + hi) / sc;
  return true;
}

// One inverse iteration on the vector of warp_lowest_f32_pivots with its
// pivots (the ratios alone are the solution for the right-hand side e_0: they
// carry the shift's distance from theta over the start vector's share of the
// lowest state); unit length again.
__device__ __forceinline__ void improve_f32(float* work, int n) {
  const int lane = threadIdx.x & 31;
  float* zf = work + 4 * kTriMax;
  if (lane == 0) pivot_solve(work + 2 * kTriMax, work + 3 * kTriMax, n, zf);
  __syncwarp();
  const float f0 = (lane < n) ? zf[lane] : 0.0f, f1 = (lane + 32 < n) ? zf[lane + 32] : 0.0f;
  const float im = __fdividef(1.0f, warp_max_f(fmaxf(fabsf(f0), fabsf(f1))));
  const float g0 = f0 * im, g1 = f1 * im;
  const float inv = rsqrtf(warp_sum_f(fmaf(g0, g0, g1 * g1)));
  if (lane < n) zf[lane] = g0 * inv;
  if (lane + 32 < n) zf[lane + 32] = g1 * inv;
  __syncwarp();
}

// The mixed path's check: theta to FP32 accuracy of the spread, z (normalised,
// first component positive) and *resid = |bn z_{n-1}|; what the FP32 pivots
// cannot do through warp_lowest_eig_f32.
__device__ inline double warp_check_lowest_f32(const double* a, const double* b, int n, double bn,
                                               bool warm, double th_prev, double r_prev,
                                               double* z, double* work, double* resid) {
  const int lane = threadIdx.x & 31;
  float* w = reinterpret_cast<float*>(work);
  float th = 0.0f, tail = 0.0f, width = 0.0f, sc = 1.0f;
  if (n > 1 &&
      warp_lowest_f32_pivots(a, b, n, w, warm, th_prev, r_prev, &th, &tail, &width, &sc)) {
    improve_f32(w, n);
    for (int i = lane; i < n; i += 32) z[i] = double(w[4 * kTriMax + i]);
    __syncwarp();
    *resid = fabs(bn * z[n - 1]);  // (`tail` is off by up to a tenth, see above)
    return a[0] + double(th);
  }
  const double t = warp_lowest_eig_f32(a, b, n, z, work, false, 0.0, 0.0);
  *resid = fabs(bn * z[n - 1]);
  return t;
}

// The check of the n x n Lanczos tridiagonal (a, b) with beta_n = bn, by one
// warp: *theta and the residual |bn z_{n-1}| in *resid, and whether it is at
// most tol.  z (kTriMax doubles) holds the FP64 eigenvector when the check
// converged or `need` is set (theta is FP64-accurate only then).  work: 3 *
// kTriMax doubles.
__device__ inline bool warp_check_lowest(const double* a, const double* b, int n, double bn,
                                         double tol, bool need, bool warm, double th_prev,
                                         double r_prev, double* z, double* work, double* theta,
                                         double* resid) {
  const int lane = threadIdx.x & 31;
  float* w = reinterpret_cast<float*>(work);
  float th = 0.0f, tail = 0.0f, width = 0.0f, sc = 1.0f;
  if (n > 1 &&
      warp_lowest_f32_pivots(a, b, n, w, warm, th_prev, r_prev, &th, &tail, &width, &sc)) {
    const double r = fabs(bn) * double(tail);
    *resid = r;
    const bool conv = r <= tol;
    const double s0 = a[0] + double(th);
    if (!conv && !need) {
      *theta = s0;
      return false;
    }
    improve_f32(w, n);
    const float* bf = w + 2 * kTriMax;
    const float* ru = w + 3 * kTriMax;
    float* x = w + 4 * kTriMax;  // the FP32 vector, then residuals and corrections
    const int i0 = lane, i1 = lane + 32;
    double z0 = (i0 < n) ? double(x[i0]) : 0.0, z1 = (i1 < n) ? double(x[i1]) : 0.0;
    const double t0 = (i0 < n) ? a[i0] - s0 : 0.0, t1 = (i1 < n) ? a[i1] - s0 : 0.0;
    const double bl0 = (i0 > 0 && i0 < n) ? b[i0 - 1] : 0.0, br0 = (i0 < n - 1) ? b[i0] : 0.0;
    const double bl1 = (i1 < n) ? b[i1 - 1] : 0.0, br1 = (i1 < n - 1) ? b[i1] : 0.0;
    bool good = false;
    double dth = 0.0;
    float last = 3.0e38f;
    for (int it = 0; it < 6; ++it) {
      if (i0 < n) z[i0] = z0;
      if (i1 < n) z[i1] = z1;
      __syncwarp();
      const double l0 = (i0 > 0 && i0 < n) ? z[i0 - 1] : 0.0, r0 = (i0 < n - 1) ? z[i0 + 1] : 0.0;
      const double l1 = (i1 < n) ? z[i1 - 1] : 0.0, r1 = (i1 < n - 1) ? z[i1 + 1] : 0.0;
      const double v0 = fma(t0, z0, fma(bl0, l0, br0 * r0));
      double v1 = 0.0;
      if (n > 32) v1 = fma(t1, z1, fma(bl1, l1, br1 * r1));
      double zv = z0 * v0, zz = z0 * z0;
      if (n > 32) {
        zv = fma(z1, v1, zv);
        zz = fma(z1, z1, zz);
      }
      zv = warp_sum_d(zv);
      zz = warp_sum_d(zz);
      // |z|^2 is 1 to FP32 accuracy or better: first-order reciprocals
      dth = zv * (2.0 - zz);
      const double e0 = fma(-dth, z0, v0), e1 = fma(-dth, z1, v1);
      const float f0 = float(e0), f1 = float(e1);
      const float big = warp_max_f(fmaxf(fabsf(f0), fabsf(f1)));
      if (!(big <= 0.25f * last)) {  // no further gain: at rounding level, or stalled
        good = big <= 4e-15f * width;
        break;
      }
      last = big;
      if (big == 0.0f) {
        good = true;
        break;
      }
      __syncwarp();
      const float ib = 1.0f / big;
      if (i0 < n) x[i0] = f0 * ib;
      if (i1 < n) x[i1] = f1 * ib;
      __syncwarp();
      if (lane == 0) pivot_solve(bf, ru, n, x);  // (T - s) x = residual / big
      __syncwarp();
      const float g0 = (i0 < n) ? x[i0] : 0.0f, g1 = (i1 < n) ? x[i1] : 0.0f;
      const float zf0 = float(z0), zf1 = float(z1);
      const float along = warp_sum_f(fmaf(zf0, g0, zf1 * g1));
      const float h0 = fmaf(-along, zf0, g0), h1 = fmaf(-along, zf1, g1);
      const float ds = big * sc;  // the FP32 matrix is sc (T - a_0)
      z0 -= double(ds * h0);
      z1 -= double(ds * h1);
      // unit length again (to first order in |z|^2 - 1)
      const double sc = fma(-0.5, zz, 1.5);
      z0 *= sc;
      z1 *= sc;
    }
    if (good) {
      *theta = s0 + dth;
      __syncwarp();
      *resid = fabs(bn * z[n - 1]);
      return *resid <= tol;
    }
  }
  *theta = warp_lowest_eig(a, b, n, z, work);
  *resid = fabs(bn * z[n - 1]);
  return *resid <= tol;
}

}  // namespace lgt
