// cheb.cu -- exp(-iHt) steps by Chebyshev expansion (the path of
// evolve_ED!, finite_ed.jl:405-431, wherever a step's expansion is short).
//
// With the spectrum of H inside [c - d, c + d] and H~ = (H - c) / d,
//   exp(-i H tau) = exp(-i c tau) sum_n (2 - [n = 0]) (-i)^n J_n(d tau) T_n(H~)
// (Tal-Ezer and Kosloff, J. Chem. Phys. 81, 3967 (1984)).  H is real, so the
// real and imaginary parts of every point are two real columns of one panel
// and T_n needs real arithmetic only.  Against a Krylov step of the same
// number of products this drops the orthogonalisation (two passes over all
// earlier vectors per product, 55 % of a 4x4 K = 8 step): a product reads
// T_n (gathered) and T_{n-1} once and writes T_{n+1}, and one pass at the end
// sums the stored panels.  Measured against the Krylov step, observables
// included: 4x4 K = 8 mixed, two steps of dt = 0.05, 114.6 -> 35.0 ms; 4x4
// K = 3 FP64 with plaquettes, one step, 85.1 -> 36.5 ms (issue of the products'
// integer sums); 3x4 K = 1 FP64, ten steps, 13.5 -> 2.3 ms.
//
// Errors.  FP64: that of the Krylov steps (3e-15 to 9e-15).  Mixed: every T_n is
// rounded to FP32 once, when it is stored.  The couplings of the products are
// scaled on the host and kept as pairs of FP32 numbers (pair_coefs), the
// neighbours are added pairwise, and of T_1, which a short step is made of
// beside T_0, the part that the rounding drops is kept too.  The state's
// distance from the FP64 one, against that of the Krylov steps (three sets of
// points each): 4x4 K = 8, two steps of 0.05: 1.3e-8 - 1.6e-8 (3.5e-8); 4x3
// K = 2 with plaquettes, the same: 1.0e-8 - 1.1e-8 (1.7e-8 - 3.3e-8); 3x4
// K = 2, six steps of 0.1: 6.9e-8 - 8.1e-8 (8.5e-8 - 9.4e-8); 3x3, one step of
// 0.03: 2.1e-10 - 2.7e-10 (2.0e-9).  (With FP32 couplings, the scale apart and
// one chain of sums it was 3.0e-8 - 3.9e-8 for the first of these.)
//
// The bounds are Gershgorin's, per point, from the table's row meta words
// (diagonal and entry counts) in FP32, widened by 1e-5 of their size.  The
// expansion stops where the tail of the Bessel coefficients is below 2e-16
// (FP64) or min(tol, 1e-11) (mixed), so the truncation never exceeds the
// tolerance of the Krylov step's error estimate; its length depends on
// (d tau) alone and is known before the first product.  The global phase
// exp(-i c tau) commutes with everything and is applied once, with the last
// step's normalisation.
#include <cmath>
#include <cstdint>

#include "lgt_cheb.h"
#include "lgt_dfloat.cuh"
#include "lgt_internal.h"

namespace lgt {

namespace {

constexpr int kT = 256;
constexpr int kBoundBlocks = 304;
constexpr int kMaxBlocks = 1216;  // of the summing passes

#define CCK(call)                                                                  \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
  } while (0)

// Per-block Gershgorin bounds of every point: out[blk][k] = (min, max).
__global__ void __launch_bounds__(kT) k_cheb_bounds(const uint32_t* meta, int64_t N, int K,
                                                    const float* cE, const float* cm,
                                                    const float* ch, const float* cp, float2* out) {
  __shared__ float s_lo[kT], s_hi[kT];
  const int RG = kT / K;
  const int k = threadIdx.x % K, rg = threadIdx.x / K;
  float lo = INFINITY, hi = -INFINITY;
  if (rg < RG) {
    const float e = cE[k], m = cm[k], h = fabsf(ch[k]), p = fabsf(cp[k]);
    for (int64_t r = int64_t(blockIdx.x) * RG + rg; r < N; r += int64_t(gridDim.x) * RG) {
      const uint32_t w = __ldg(meta + r);
      const int cnt = int(w & 255u), nh = int((w >> 8) & 255u);
      const float dg = e * float(int((w >> 16) & 255u)) + m * float(int(w >> 24) - 128);
      const float off = h * float(nh) + p * float(cnt - nh);
      lo = fminf(lo, dg - off);
      hi = fmaxf(hi, dg + off);
    }
  }
  s_lo[threadIdx.x] = lo;
  s_hi[threadIdx.x] = hi;
  __syncthreads();
  if (threadIdx.x < K) {
    for (int g = 1; g < RG; ++g) {
      lo = fminf(lo, s_lo[g * K + threadIdx.x]);
      hi = fmaxf(hi, s_hi[g * K + threadIdx.x]);
    }
    out[size_t(blockIdx.x) * K + threadIdx.x] = make_float2(lo, hi);
  }
}

// The bounds over all blocks, one warp per point.
__global__ void k_cheb_bounds_finish(const float2* part, int nblk, int K, float2* out) {
  const int k = blockIdx.x, lane = threadIdx.x;
  float lo = INFINITY, hi = -INFINITY;
  for (int b = lane; b < nblk; b += 32) {
    const float2 v = part[size_t(b) * K + k];
    lo = fminf(lo, v.x);
    hi = fmaxf(hi, v.y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) out[k] = make_float2(lo, hi);
}

// Adds a thread's value of point k over its block in a fixed order into
// part[blk][k] (threads: k = tid % K, row groups tid / K).
__device__ __forceinline__ void block_point_sum(double v, int K, double* red, double* part) {
  const int RG = kT / K;
  red[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0.0;
    for (int g = 0; g < RG; ++g) s += red[g * K + threadIdx.x];
    part[size_t(blockIdx.x) * K + threadIdx.x] = s;
  }
}

// |psi_k|^2 partial sums of the panel the steps start from.
__global__ void __launch_bounds__(kT) k_cheb_norm(const double2* X, int64_t N, int K, int64_t rpb,
                                                  double* part) {
  __shared__ double red[kT];
  const int RG = kT / K;
  const int k = threadIdx.x % K, rg = threadIdx.x / K;
  const int64_t r0 = int64_t(blockIdx.x) * rpb;
  const int64_t r1 = (r0 + rpb < N) ? r0 + rpb : N;
  double n2 = 0.0;
  if (rg < RG)
    for (int64_t r = r0 + rg; r < r1; r += RG) {
      const double2 v = X[size_t(r) * K + k];
      n2 = fma(v.x, v.x, fma(v.y, v.y, n2));
    }
  block_point_sum(n2, K, red, part);
}

// rho[k] = ||psi_k||; drift[k] = max over the steps of |1 - rho|, where the
// first step's norm counts the start's (rho0); a norm that is not finite
// raises `fail`.  One warp per point.
__global__ void k_cheb_finish(const double* part, int nblk, int K, double* rho,
                              const double* rho0, double* drift, int* fail) {
  const int k = blockIdx.x, lane = threadIdx.x;
  double s = 0.0;
  for (int b = lane; b < nblk; b += 32) s += part[size_t(b) * K + k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane != 0) return;
  const double r = sqrt(s);
  rho[k] = r;
  if (!isfinite(r)) atomicOr(fail, 1);
  if (drift) drift[k] = fmax(drift[k], fabs((rho0 ? r * rho0[k] : r) - 1.0));
}

// X /= rho per point (times the phase, when given), and the panel's T_0 in
// the storage precision and row order of the products (V_0 row n is X row
// perm[n]); V null: none is needed.  Moves 2 x 16 + 2 S bytes per entry.
template <typename S>
__global__ void __launch_bounds__(kT) k_cheb_start(double2* X, S* V, int64_t N, int K,
                                                   const double* rho, const double* phase,
                                                   const int* perm) {
  const int RG = kT / K;
  const int k = threadIdx.x % K, rg = threadIdx.x / K;
  if (rg >= RG) return;
  const double b = rho[k];
  const double inv = (b > 0.0) ? 1.0 / b : 0.0;
  double pr = 0.0, pi = 0.0;
  if (phase) {
    pr = phase[2 * k];
    pi = phase[2 * k + 1];
  }
  for (int64_t r = int64_t(blockIdx.x) * RG + rg; r < N; r += int64_t(gridDim.x) * RG) {
    const size_t at = size_t(perm ? perm[r] : r) * K + k;
    double2 v = X[at];
    v.x *= inv;
    v.y *= inv;
    if (phase) v = make_double2(fma(v.x, pr, -(v.y * pi)), fma(v.x, pi, v.y * pr));
    X[at] = v;
    if (V) {
      const size_t to = (size_t(r) * K + k) * 2;
      if constexpr (sizeof(S) == 4)
        *reinterpret_cast<float2*>(V + to) = make_float2(narrow(v.x), narrow(v.y));
      else
        *reinterpret_cast<double2*>(V + to) = v;
    }
  }
}

// X <- a_0 X + sum_{n >= 1} of the expansion's terms, in place, and the
// partial sums of the new norms.  coef[n][k] = +-J_n (2 - [n = 0]): an even n
// adds coef T_n, an odd one -i coef T_n, to (re, im).  FP32 panels: double-
// float sums (coefficients split into FP32 pairs once per block) beside the
// FP64 first term, which is taken from X itself, and the part of T_1 that FP32
// drops from `low` (a short step is little more than its first two terms);
// FP64 panels: FP64 sums.  Bound by the panels' bytes ((terms + 1) S 2 N K read
// once) in FP32.
template <typename S>
__global__ void __launch_bounds__(kT) k_cheb_combine(const S* __restrict__ V, size_t vstride,
                                                     const S* __restrict__ low,
                                                     const double* coef, int terms, double2* X,
                                                     int64_t N, int K, int64_t rpb,
                                                     const int* perm, double* part) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[kT];
  const int ncf = terms * K;
  double* s_cd = reinterpret_cast<double*>(smem);
  float* s_hi = reinterpret_cast<float*>(smem);
  float* s_lo = s_hi + ncf;
  for (int i = threadIdx.x; i < ncf; i += kT) {
    const double c = coef[i];
    if constexpr (sizeof(S) == 4) {
      const float h = narrow(c);
      s_hi[i] = h;
      s_lo[i] = narrow(c - widen(h));
    } else {
      s_cd[i] = c;
    }
  }
  __syncthreads();
  const int RG = kT / K;
  const int k = threadIdx.x % K, rg = threadIdx.x / K;
  const int64_t r0 = int64_t(blockIdx.x) * rpb;
  const int64_t r1 = (r0 + rpb < N) ? r0 + rpb : N;
  double n2 = 0.0;
  if (rg < RG) {
    const double a0 = coef[k];
    for (int64_t r = r0 + rg; r < r1; r += RG) {
      const size_t at = size_t(perm ? perm[r] : r) * K + k;
      const double2 x0 = X[at];
      const S* v = V + (size_t(r) * K + k) * 2;
      double re, im;
      if constexpr (sizeof(S) == 4) {
        df ar{0.f, 0.f}, ai{0.f, 0.f};
        auto term = [](df& acc, float ch, float cl, float t) {
          float p, e, q;
          two_prod(ch, t, p, e);
          e = df_fma_rn(cl, t, e);
          two_sum(acc.hi, p, acc.hi, q);
          acc.lo = df_add_rn(acc.lo, df_add_rn(q, e));
        };
        for (int n = 1; n < terms; n += 4) {
          float2 t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n + u < terms) t[u] = __ldcs(reinterpret_cast<const float2*>(v + size_t(n + u) * vstride));
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n + u < terms) {
              const float h = s_hi[(n + u) * K + k], l = s_lo[(n + u) * K + k];
              if (u & 1) {  // n + u even
                term(ar, h, l, t[u].x);
                term(ai, h, l, t[u].y);
              } else {
                term(ar, h, l, t[u].y);
                term(ai, -h, -l, t[u].x);
              }
            }
        }
        if (terms > 1) {
          const float2 t =
              __ldcs(reinterpret_cast<const float2*>(low + (size_t(r) * K + k) * 2));
          ar.lo = df_fma_rn(s_hi[K + k], t.y, ar.lo);
          ai.lo = df_fma_rn(-s_hi[K + k], t.x, ai.lo);
        }
        re = fma(a0, x0.x, widen(ar.hi) + widen(ar.lo));
        im = fma(a0, x0.y, widen(ai.hi) + widen(ai.lo));
      } else {
        re = 0.0;
        im = 0.0;
        for (int n = 1; n < terms; n += 4) {
          double2 t[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n + u < terms)
              t[u] = __ldcs(reinterpret_cast<const double2*>(v + size_t(n + u) * vstride));
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n + u < terms) {
              const double c = s_cd[(n + u) * K + k];
              if (u & 1) {
                re = fma(c, t[u].x, re);
                im = fma(c, t[u].y, im);
              } else {
                re = fma(c, t[u].y, re);
                im = fma(-c, t[u].x, im);
              }
            }
        }
        re = fma(a0, x0.x, re);
        im = fma(a0, x0.y, im);
      }
      X[at] = make_double2(re, im);
      n2 = fma(re, re, fma(im, im, n2));
    }
  }
  block_point_sum(n2, K, red, part);
}

int blocks_for(int64_t N, int K, int64_t* rpb) {
  const int RG = kT / K;
  // two rows a thread at least (four: 2.69 ms for 3x4 K = 1 FP64, ten steps;
  // two 2.59, one 2.60)
  int64_t b = (N + 2 * RG - 1) / (2 * RG);
  if (b > kMaxBlocks) b = kMaxBlocks;
  if (b < 1) b = 1;
  *rpb = (N + b - 1) / b;
  return int((N + *rpb - 1) / *rpb);
}

// The FP32 products' coefficients (PairCoef) of one point: out[q * K].  cc:
// cE, cm, ch, cp at [q * K].  The leading parts of the diagonal's three terms
// are multiples of a unit of which no sum of them reaches 2^24: a row's
// diagonal is then exact in FP32, however its terms are added.
void pair_coefs(const Geom& G, const double* cc, int K, double shift, double scale, float* out) {
  const double el = scale * cc[0], mass = scale * cc[K], sh = scale * shift;
  const double most = std::fabs(el) * double((G.nR + G.nU) * G.dg * G.dg) +
                      std::fabs(mass) * double(G.ns) + std::fabs(sh);
  int e = 0;
  std::frexp(most, &e);  // most < 2^e
  const double unit = std::ldexp(1.0, e - 23);
  auto put = [&](int q, double v, double hi) {
    out[size_t(q) * K] = float(hi);
    out[size_t(q + 1) * K] = float(v - double(float(hi)));
  };
  put(kElHi, el, std::nearbyint(el / unit) * unit);
  put(kMassHi, mass, std::nearbyint(mass / unit) * unit);
  put(kShiftHi, sh, std::nearbyint(sh / unit) * unit);
  put(kHopHi, scale * cc[2 * K], scale * cc[2 * K]);
  put(kPlaqHi, scale * cc[3 * K], scale * cc[3 * K]);
}

// Dynamic shared memory of k_cheb_combine.
size_t comb_smem(int terms, int K) { return sizeof(double) * size_t(terms) * K; }

// Device memory and shared memory for an expansion of `terms` panels of `vs`
// elements (FP32: and T_1's dropped part behind them); false (with nothing
// held) where they cannot be had.
template <typename S>
bool reserve(ChebWork* w, int terms, int K, size_t vs, cudaStream_t s) {
  const size_t need = sizeof(S) * vs * size_t(terms + (sizeof(S) == 4 ? 1 : 0)) + 256;
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k_cheb_combine<S>),
                                   int(comb_smem(terms, K)));
  if (e == cudaSuccess && w->v_bytes < need) {
    dev_free(w->V, s);
    w->V = nullptr;
    w->v_bytes = 0;
    e = dev_alloc(&w->V, need, s);
    if (e == cudaSuccess) w->v_bytes = need;
  }
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  w->release(s);
  return false;
}

template <typename S>
std::string run(const OpDev& op, ChebWork* w, const NbrTable& T, int n_steps,
                const std::vector<std::vector<double>>& J, const std::vector<double>& c,
                const std::vector<double>& d, int terms, double dt, double* Xd, double* drift,
                StepObserver* obs, cudaStream_t s, KrylovReport* rep, double tail) {
  const int64_t N = op.R.dim;
  const int K = op.K;
  const size_t vs = size_t(N) * 2 * K;
  S* V = static_cast<S*>(w->V);
  S* low = V + size_t(terms) * vs;  // (FP32 only)
  int64_t rpb = 1;
  const int nblk = blocks_for(N, K, &rpb);
  // aux (the bounds in it have been read): coefficients, norms, partial sums
  double* a_coef = static_cast<double*>(w->aux);
  double* a_phase = a_coef + size_t(terms) * K;
  double* a_rho = a_phase + 2 * K;
  double* a_rho0 = a_rho + K;
  double* a_drift = a_rho0 + K;
  // coefficients of the first product; of the others
  constexpr int kCoefs = sizeof(S) == 4 ? int(kPairCoefs) : 6;  // (12 K doubles hold both)
  S* a_c1 = reinterpret_cast<S*>(a_drift + K);
  S* a_c2 = a_c1 + kCoefs * size_t(K);
  const size_t host_n = size_t(terms) * K + 5 * size_t(K) + 12 * size_t(K);
  int* a_fail = reinterpret_cast<int*>(a_coef + host_n);
  double* a_part = a_coef + host_n + 1;
  std::vector<double> h(host_n + 1, 0.0);
  std::vector<double> cc(4 * size_t(K));
  CCK(cudaMemcpyAsync(cc.data(), op.cE_d, sizeof(double) * 4 * K, cudaMemcpyDeviceToHost, s));
  CCK(cudaStreamSynchronize(s));
  S* h1 = reinterpret_cast<S*>(h.data() + size_t(terms) * K + 5 * size_t(K));
  S* h2 = h1 + kCoefs * size_t(K);
  for (int k = 0; k < K; ++k) {
    for (size_t n = 0; n < J[k].size(); ++n) {
      const double j = (n == 0 ? 1.0 : 2.0) * J[k][n];
      h[n * K + k] = ((n / 2) & 1) ? -j : j;
    }
    const double ph = -c[k] * dt * double(n_steps);
    h[size_t(terms) * K + 2 * k] = std::cos(ph);
    h[size_t(terms) * K + 2 * k + 1] = std::sin(ph);
    const double* ck = cc.data() + k;
    if constexpr (sizeof(S) == 4) {
      pair_coefs(op.G, ck, K, -c[k], 1.0 / d[k], h1 + k);
      pair_coefs(op.G, ck, K, -c[k], 2.0 / d[k], h2 + k);
    } else {
      for (int q = 0; q < 5; ++q)
        h1[size_t(q) * K + k] = h2[size_t(q) * K + k] = q < 4 ? ck[size_t(q) * K] : -c[k];
      h1[5 * size_t(K) + k] = 1.0 / d[k];
      h2[5 * size_t(K) + k] = 2.0 / d[k];
    }
  }
  // (a copy from pageable memory has staged the host data when it returns)
  CCK(cudaMemcpyAsync(a_coef, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, s));

  double2* X = reinterpret_cast<double2*>(Xd);
  const int* perm = T.perm;
  const size_t sh = comb_smem(terms, K);
  auto comb = k_cheb_combine<S>;
  const int RG = kT / K;
  int64_t gs = (N + RG - 1) / RG;
  if (gs > 152 * 16) gs = 152 * 16;
  EventPair ev;
  CCK(ev.create());
  cudaEventRecord(ev.a, s);
  if (obs) {
    const std::string e = obs->on_step(0, Xd);
    if (!e.empty()) return e;
  }
  k_cheb_norm<<<nblk, kT, 0, s>>>(X, N, K, rpb, a_part), note_launch();
  k_cheb_finish<<<K, 32, 0, s>>>(a_part, nblk, K, a_rho0, nullptr, nullptr, a_fail), note_launch();
  k_cheb_start<S><<<unsigned(gs), kT, 0, s>>>(X, V, N, K, a_rho0, nullptr, perm), note_launch();
  CCK(cudaGetLastError());
  for (int step = 1; step <= n_steps; ++step) {
    for (int n = 1; n < terms; ++n) {
      const S* x = V + size_t(n - 1) * vs;
      S* y = V + size_t(n) * vs;
      const S* prev = n > 1 ? V + size_t(n - 2) * vs : nullptr;
      const S* cf = n > 1 ? a_c2 : a_c1;
      if constexpr (sizeof(S) == 4)
        CCK(launch_cheb_product(T, op.model, N, K, x, y, prev, n == 1 ? low : nullptr, cf, s));
      else
        CCK(launch_cheb_product(T, op.model, N, K, x, y, prev, cf, s));
    }
    comb<<<nblk, kT, sh, s>>>(V, vs, low, a_coef, terms, X, N, K, rpb, perm, a_part),
        note_launch();
    k_cheb_finish<<<K, 32, 0, s>>>(a_part, nblk, K, a_rho, step == 1 ? a_rho0 : nullptr, a_drift,
                                   a_fail), note_launch();
    const bool last = step == n_steps;
    k_cheb_start<S><<<unsigned(gs), kT, 0, s>>>(X, last ? nullptr : V, N, K, a_rho,
                                                last ? a_phase : nullptr, perm), note_launch();
    CCK(cudaGetLastError());
    if (obs) {
      const std::string e = obs->on_step(step, Xd);
      if (!e.empty()) return e;
    }
  }
  int fail = 0;
  CCK(cudaMemcpyAsync(&fail, a_fail, sizeof(int), cudaMemcpyDeviceToHost, s));
  std::vector<double> dr(K);
  CCK(cudaMemcpyAsync(dr.data(), a_drift, sizeof(double) * K, cudaMemcpyDeviceToHost, s));
  cudaEventRecord(ev.b, s);
  CCK(cudaStreamSynchronize(s));
  if (drift)
    for (int k = 0; k < K; ++k) drift[k] = dr[k];
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev.a, ev.b);
  if (rep) {
    rep->matvecs += int64_t(terms - 1) * n_steps;
    rep->converged = K;
    rep->max_residual = tail;
    rep->seconds += ms * 1e-3;
  }
  if (fail) return "NOCONV: the state's norm is not finite";
  return std::string();
}

}  // namespace

void ChebWork::release(cudaStream_t s) {
  dev_free(V, s);
  dev_free(aux, s);
  V = aux = nullptr;
  v_bytes = aux_bytes = 0;
}

std::vector<double> cheb_bessel(double z, double eps, int nmax) {
  if (!(z >= 0.0) || !(z < 1e4)) return {};
  // Miller's backward recurrence J_{m-1} = (2 m / z) J_m - J_{m+1} from far
  // above z, normalised by J_0 + 2 sum J_{2k} = 1
  const int top = nmax + 40 + int(z);
  std::vector<double> j(size_t(top) + 2, 0.0);
  if (z < 1e-30) {
    j[0] = 1.0;
  } else {
    j[top] = 1e-300;
    for (int m = top; m >= 1; --m) {
      j[m - 1] = (2.0 * m / z) * j[m] - j[m + 1];
      if (std::fabs(j[m - 1]) > 1e200)
        for (int q = m - 1; q <= top; ++q) j[q] *= 1e-200;
    }
    double sum = j[0];
    for (int m = 2; m <= top; m += 2) sum += 2.0 * j[m];
    for (double& v : j) v /= sum;
  }
  double tail = 0.0;
  int n = top;
  while (n > 0 && tail + 2.0 * std::fabs(j[n]) < eps) tail += 2.0 * std::fabs(j[n--]);
  if (n > nmax) return {};
  j.resize(size_t(n) + 1);
  return j;
}

std::string cheb_expm(const OpDev& op, const KrylovParams& p, ChebWork* w, double dt, int n_steps,
                      double* X, double* drift, StepObserver* obs, cudaStream_t s,
                      KrylovReport* rep, bool* done) {
  *done = false;
  const NbrTable* T = op.table_ord && op.table_ord->state == 1 && op.table_ord->perm
                          ? op.table_ord
                          : op.table;
  const int64_t N = op.R.dim;
  const int K = op.K;
  // (the passes move (re, im) pairs of X as 16 bytes)
  if (!T || T->state != 1 || !(dt > 0.0) || n_steps < 1 || N < 1 || 2 * K > kT ||
      (reinterpret_cast<uintptr_t>(X) & 15) != 0)
    return std::string();
  // the buffers beside the panels, sized for the longest expansion
  const int nmax = p.krylovdim;
  int64_t rpb = 1;
  const size_t aux = sizeof(double) * (size_t(nmax + 1) * K + 18 * size_t(K) + 2 +
                                       size_t(blocks_for(N, K, &rpb)) * K) +
                     sizeof(float2) * size_t(kBoundBlocks + 1) * K + 256;
  if (w->aux_bytes < aux) {
    dev_free(w->aux, s);
    w->aux = nullptr;
    w->aux_bytes = 0;
    if (dev_alloc(&w->aux, aux, s) != cudaSuccess) {
      cudaGetLastError();
      w->release(s);
      return std::string();
    }
    w->aux_bytes = aux;
  }
  float2* part = static_cast<float2*>(w->aux);
  float2* bnd = part + size_t(kBoundBlocks) * K;
  k_cheb_bounds<<<kBoundBlocks, kT, 0, s>>>(T->meta, N, K, op.cE_f, op.cm_f, op.ch_f, op.cp_f,
                                            part), note_launch();
  k_cheb_bounds_finish<<<K, 32, 0, s>>>(part, kBoundBlocks, K, bnd), note_launch();
  CCK(cudaGetLastError());
  std::vector<float2> b(K);
  CCK(cudaMemcpyAsync(b.data(), bnd, sizeof(float2) * K, cudaMemcpyDeviceToHost, s));
  CCK(cudaStreamSynchronize(s));
  const double eps = p.mixed ? std::fmin(p.tol, 1e-11) : 2e-16;
  std::vector<double> c(K), d(K);
  std::vector<std::vector<double>> J(K);
  for (int k = 0; k < K; ++k) {
    const double lo = b[k].x, hi = b[k].y;
    if (!std::isfinite(lo) || !std::isfinite(hi) || std::fmax(std::fabs(lo), std::fabs(hi)) > 1e30 ||
        !(std::fmax(std::fabs(lo), std::fabs(hi)) > 1e-25))
      return std::string();
    c[k] = double(float(0.5 * (lo + hi)));
    d[k] = 0.5 * (hi - lo) + 1e-5 * std::fmax(std::fabs(lo), std::fabs(hi)) + 1e-30;
    d[k] = 1.0 / double(std::nextafterf(float(1.0 / d[k]), 0.0f));
    J[k] = cheb_bessel(d[k] * dt, eps, nmax);
    if (J[k].empty()) return std::string();
  }
  int terms = 1;
  for (const auto& j : J) terms = int(j.size()) > terms ? int(j.size()) : terms;
  const size_t vs = size_t(N) * 2 * K;
  if (!(p.mixed ? reserve<float>(w, terms, K, vs, s) : reserve<double>(w, terms, K, vs, s)))
    return std::string();
  *done = true;
  return p.mixed ? run<float>(op, w, *T, n_steps, J, c, d, terms, dt, X, drift, obs, s, rep, eps)
                 : run<double>(op, w, *T, n_steps, J, c, d, terms, dt, X, drift, obs, s, rep, eps);
}

}  // namespace lgt
