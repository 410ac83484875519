// small.cu -- persistent batched Lanczos for small sectors: one CTA per
// (lattice, coupling point) runs a whole ground-state solve.
//
// For sectors up to kSmallMaxN states the step latency of the panel path
// (about ten dependent kernels per Lanczos step) dominates, so here every
// (problem, point) unit is one CTA, or a cluster of two that split the rows,
// of just enough warps for R rows per thread (at most 512 threads).  It keeps
// the current Lanczos residual in registers (row r of thread t: r = t + i *
// blockDim) and runs matvec, classical Gram-Schmidt against the whole basis
// (eight vectors a round; sums in double-float on the mixed path, in FP64 with
// the lanes added in integers on the other; a second pass only on
// cancellation), the tridiagonal check (lgt_tridiag.cuh), restarts and the
// FP64 finish without leaving the kernel.  Units of different sectors and
// sizes share one launch (uneven batch); the largest are scheduled first.
//
// A CTA's own rows of the Krylov basis with the whole current vector, and for
// R <= 4 its neighbour lists, sit in shared memory where the largest sector's
// fit 200 KB (on two CTAs and krylovdim 50: up to about 1900 states mixed, 950
// FP64); the basis is in global memory (L2) otherwise.  One CTA per SM either
// way.
//
// The neighbour ranks of a lattice are computed once by a device "lookup
// pass" (k_pattern_*: the move enumeration and rank of the H*psi kernel)
// and shared by all K coupling points; coefficients are per point, so
// nothing of the matrix values is stored.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "lgt_dfloat.cuh"
#include "lgt_intsum.cuh"
#include "lgt_moves.cuh"
#include "lgt_rank.cuh"
#include "lgt_small.h"
#include "lgt_tridiag.cuh"

namespace lgt {

namespace {

constexpr int kCta = 512;               // most threads per CTA
constexpr int kWarpsCta = kCta / 32;
constexpr int kMaxM = 64;

#define SCK(call)                                                                  \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) return std::string(#call ": ") + cudaGetErrorString(e_); \
  } while (0)

// ---- lookup pass --------------------------------------------------------------

template <bool PLAQ, bool JW>
__global__ void k_pattern_count(Geom G, RankView R, int64_t N, int* counts) {
  int64_t row = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= N) return;
  const Config c = decode(G, R.keys[row]);
  int n = 0;
  for_each_move<PLAQ, JW>(G, c, [&](uint64_t, uint32_t) { ++n; });
  counts[row] = n;
}

// Single-block exclusive scan of int counts into int32 row pointers.
__global__ void __launch_bounds__(1024) k_scan_rows(const int* counts, int64_t n, int* rowptr) {
  __shared__ int warp_sum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t start = 0; start < n; start += 1024) {
    const int64_t i = start + threadIdx.x;
    const int v = (i < n) ? counts[i] : 0;
    int x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int s = warp_sum[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, s, d);
        if (lane >= d) s += y;
      }
      warp_sum[lane] = s;
    }
    __syncthreads();
    const int excl = (wid > 0) ? warp_sum[wid - 1] : 0;
    if (i < n) rowptr[i] = carry + excl + x - v;
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) rowptr[n] = carry;
}

template <bool PLAQ, bool JW>
__global__ void k_pattern_fill(Geom G, RankView R, int64_t N, const int* rowptr, uint32_t* nbr,
                               int16_t* e2, int16_t* stag, int* err) {
  int64_t row = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= N) return;
  const Config c = decode(G, R.keys[row]);
  int a, s;
  diag_parts(G, c, &a, &s);
  e2[row] = int16_t(a);
  stag[row] = int16_t(s);
  int p = rowptr[row];
  const int end = rowptr[row + 1];
  for_each_move<PLAQ, JW>(G, c, [&](uint64_t nk, uint32_t kind) {
    const int64_t j = rank_key(R, R.segc, R.binom, nk);
    if (j < 0 || p >= end) {
      raise_err(err, j < 0 ? kDevErrRank : kDevErrBounds);
      return;
    }
    nbr[p++] = (uint32_t(j) << 2) | kind;
  });
}

// ---- device helpers -----------------------------------------------------------

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Same stream of normals as the panel path's start vectors (point k, row r).
__device__ __forceinline__ double start_normal(uint64_t seed, int k, int64_t row) {
  uint64_t h = mix64(mix64(seed) ^ mix64(uint64_t(k) + 0x5851F42D4C957F2Dull));
  h = mix64(h ^ uint64_t(row));
  const uint64_t h2 = mix64(h);
  const double u1 = (double((h >> 11) + 1)) * 0x1.0p-53;
  const double u2 = double(h2 >> 11) * 0x1.0p-53;
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

__device__ __forceinline__ df shfl_xor_df(df v, int o) {
  return df{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}

// x += (h + l)^2 for a double-float h + l: the leading square exactly, the
// cross term rounded (l^2 is below the pair's precision).
__device__ __forceinline__ void df_sq2(df& x, float h, float l) {
  float p, e;
  two_prod(h, h, p, e);
  e = df_fma_rn(df_add_rn(h, h), l, e);
  df_acc(x, p, e);
}

// warp_scatter8 of double-floats.
__device__ __forceinline__ df warp_scatter8_df(const df* p, int lane) {
  return warp_scatter8<df>(p, lane, [](df x, df y) { return df_add(x, y); },
                           [](df x, int o) { return shfl_xor_df(x, o); });
}

__device__ __forceinline__ df warp_total(df v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = df_add(v, shfl_xor_df(v, o));
  return v;
}
__device__ __forceinline__ double warp_total(double v) { return warp_sum_int(v); }
__device__ __forceinline__ double as_double(df v) { return widen(v.hi) + widen(v.lo); }
__device__ __forceinline__ double as_double(double v) { return v; }
__device__ __forceinline__ float flip_sign(float v, uint32_t ent) {
  return __uint_as_float(__float_as_uint(v) ^ (ent & 0x80000000u));
}

// 1 / sqrt(s): an FP32 start and two Newton steps y += y/2 (1 - s y^2) in the
// range of FP32, rsqrt() outside it; 0 for s <= 0 or NaN.
__device__ __forceinline__ double inv_sqrt(double s) {
  const int e = (__double2hiint(s) >> 20);  // negative for s < 0
  if (e > 1023 - 120 && e < 1023 + 120) {
    const float r = rsqrtf(narrow(s));
    double y = widen(r);
    y = fma(widen(0.5f * r), fma(-s * y, y, 1.0), y);
    return fma(0.5 * y, fma(-s * y, y, 1.0), y);
  }
  return (s > 0.0) ? rsqrt(s) : 0.0;
}

// Totals over a unit's CTAs of one value per thread.  Every warp adds its
// lanes and leaves the total in slot [par][rank * warps + warp] of all CTAs of
// the unit (CL = 2: its own and, through distributed shared memory, its
// peer's); after one barrier warp 0 of each CTA adds the slots in that order,
// so both CTAs hold bitwise the same sum (their control flow, which depends
// only on such sums, stays identical), and its thread 0 calls root(sum)
// before the block goes on.  `par` flips at every call, so a CTA running
// ahead never overwrites slots that its peer has yet to read.
template <int CL, class A, class Root>
__device__ __forceinline__ void unit_reduce(A v, A (*slots)[CL * kWarpsCta], int& par, Root root) {
  namespace cg = cooperative_groups;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_total(v);
  if constexpr (CL == 2) {
    cg::cluster_group cl = cg::this_cluster();
    const unsigned cr = cl.block_rank();
    A* at = &slots[par][int(cr) * nw + wid];
    if (lane == 0) {
      *at = v;
      *cl.map_shared_rank(at, cr ^ 1u) = v;
    }
    cl.sync();
  } else {
    if (lane == 0) slots[par][wid] = v;
    __syncthreads();
  }
  if (wid == 0) {
    A s;
    if constexpr (std::is_same<A, df>::value) s = (lane < CL * nw) ? slots[par][lane] : df{0.f, 0.f};
    else s = (lane < CL * nw) ? slots[par][lane] : 0.0;
    s = warp_total(s);
    if (lane == 0) root(as_double(s));
  }
  par ^= 1;
  __syncthreads();
}

// One ground-state solve per unit of CL CTAs.  S: storage/matvec precision
// of the Krylov basis (double, or float for the FP32-mixed path); R: rows
// per thread held in registers (N <= CL * R * 512).  CL = 2 runs a unit on
// a cluster of two CTAs: CTA rank c owns rows c R nthr .. (c + 1) R nthr - 1,
// every reduction adds the warps' totals of both CTAs in one order
// (unit_reduce and the dots), so both CTAs take the same branches at every
// step; a new vector's rows go into both CTAs' copy of the current vector (or
// once into the unit's global basis), which the cluster barrier after each
// store orders before the next product.
//
// A step is bound by latency: a dependent FP64 operation takes 64 cycles, a
// cluster barrier about a thousand.  So the sums over lanes and warps run in
// double-float (mixed) or in integers (FP64: lgt_intsum.cuh), warp totals go
// to both CTAs without a block barrier of their own, eight dots are reduced
// together, and for R <= 4 the rows' neighbour lists sit in shared memory and
// their diagonals in registers for the whole solve.  Cycles a step (4x2,
// K = 64, clusters of two, R = 1), before -> after: mixed 21.9k -> 15.1k
// (matvec 2.7 -> 1.2, dots 4.7 -> 3.7, their totals 2.8 -> 1.3, update 2.1 ->
// 2.6, norm 4.0 -> 3.0, checks 4.0 -> 2.4); FP64 65.3k -> 32k (matvec 5.1 ->
// 4.0, dots 15.8 -> 12.8, totals 4.1 -> 2.2, update 5.5 -> 6.3, norm 3.5 ->
// 2.6, checks 29.3 -> 3.2).
template <typename S, int R, int CL>
__global__ void __launch_bounds__(kCta, 1) k_lanczos_cta(const SmallProblem* probs,
                                                      const SmallUnit* units, SmallParams prm) {
  // The FP32-mixed path (S = float) keeps the Lanczos residual as
  // double-float pairs and runs its Gram-Schmidt dots, updates and norms in
  // double-float arithmetic on the FP32 pipe (lgt_dfloat.cuh): FP64-class
  // sums without GB300's narrow FP64 pipe.
  constexpr bool kDF = sizeof(S) == 4;
  constexpr bool kStage = R <= 4;
  using A = typename std::conditional<kDF, df, double>::type;
  extern __shared__ __align__(16) unsigned char s_dyn[];  // prm.v_smem: basis, vector; lists
  __shared__ double s_alpha[kMaxM + 1], s_beta[kMaxM + 1], s_z[kMaxM + 1];
  __shared__ A s_part[kMaxM + 2][CL * kWarpsCta];  // dot totals per slot and warp
  __shared__ A s_nslot[2][CL * kWarpsCta];         // unit_reduce, the step's norms
  __shared__ double s_dslot[2][CL * kWarpsCta];    // unit_reduce, FP64 sums
  __shared__ double s_h[kDF ? 1 : kMaxM + 2];      // FP64 coefficients
  __shared__ float s_hh[kDF ? kMaxM + 2 : 1], s_hl[kDF ? kMaxM + 2 : 1];  // mixed: FP32 pairs
  __shared__ double s_sum[3];  // unit_reduce results: sum, sqrt, 1 / sqrt
  __shared__ double s_nb;      // |w|^2 before the latest pass
  __shared__ double s_thr;     // the step's space is exhausted when beta is not above it
  __shared__ double s_lim;     // a further pass is needed when |w|^2 is below it
  __shared__ int s_exh, s_more;  // ... and whether; a further pass is needed
  __shared__ __align__(16) double s_work[3 * kMaxM];
  __shared__ double s_theta, s_resid;
  __shared__ int s_flag, s_zwarm;
  __shared__ int s_next, s_pstep;  // the next check's step; the previous check's step
  __shared__ double s_pres;        // and its residual
  __shared__ float s_rb[2];        // 1 / beta split into FP32 parts (mixed)
  int par_n = 0, par_d = 0;
  const SmallUnit U = units[blockIdx.x / CL];
  const SmallProblem P = probs[U.prob];
  const int N = P.N;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nthr = blockDim.x, nwarps = nthr >> 5;  // rows r = rbase + tid + i * nthr, i < R
  const int m = (prm.m < N) ? prm.m : N;
  // The basis: in shared memory this CTA's rows alone, [m + 1][nthr R], with
  // the whole current vector (for the gathers) behind it; else all rows in
  // the unit's global basis, [m + 1][N].  Row i of this thread is vo + i nthr.
  const bool vs = prm.v_smem != 0;
  S* V = reinterpret_cast<S*>(vs ? static_cast<void*>(s_dyn) : U.V);
  S* s_x = reinterpret_cast<S*>(s_dyn + prm.x_off);
  unsigned cr = 0;      // the CTA's rank in its unit
  S* xpeer = nullptr;   // the peer's s_x
  A* ppeer = nullptr;   // the peer's s_part
  if constexpr (CL == 2) {
    cr = cooperative_groups::this_cluster().block_rank();
    if (vs) xpeer = cooperative_groups::this_cluster().map_shared_rank(s_x, cr ^ 1u);
    ppeer = cooperative_groups::this_cluster().map_shared_rank(&s_part[0][0], cr ^ 1u);
    // both CTAs running before either touches the other's shared memory
    cooperative_groups::this_cluster().sync();
  }
  const int rbase = int(cr) * nthr * R;
  const int vst = vs ? nthr * R : N;          // elements per basis vector
  const int vo = (vs ? 0 : rbase) + tid;
  // entry of basis vector b in this thread's row i (r in the sector)
  auto put_v = [&](int b, int i, int r, S val) {
    V[size_t(b) * vst + vo + i * nthr] = val;
    if (vs) {
      s_x[r] = val;
      if (CL == 2) xpeer[r] = val;
    }
  };
  // orders this unit's stores (basis, X) before any CTA of the unit reads them
  auto unit_sync = [&]() {
    if constexpr (CL == 2) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  };
  // thread 0's root: the sum, the norm and its reciprocal into s_sum
  auto norm_root = [&](double sv) {
    const double rs = inv_sqrt(sv);
    s_sum[0] = sv;
    s_sum[1] = sv * rs;
    s_sum[2] = rs;
  };
  auto unit_sum = [&](double v) -> double {
    unit_reduce<CL>(v, s_dslot, par_d, norm_root);
    return s_sum[0];
  };
  auto zero = []() -> A {
    if constexpr (kDF) return df{0.f, 0.f};
    else return 0.0;
  };
  const S cE = S(U.cE), cm = S(U.cm), ch = S(U.ch), cp = S(U.cp);
  const bool fp32 = kDF;
  const double tiny_rel = fp32 ? 1e-6 : 1e-12;
  const double tol = fp32 ? fmax(prm.tol, 2e-5) : prm.tol;

  // The CTA's neighbour lists: entries index | hop sign << 31, a row's hops
  // first; rw[i]: the row's start, rn[i]: its hops | entries << 16.
  const bool staged = kStage && prm.list_cap > 0;
  uint32_t* s_list = reinterpret_cast<uint32_t*>(s_dyn + prm.list_off);
  int rw[kStage ? R : 1], rn[kStage ? R : 1];
  S dg[kStage ? R : 1];
  if constexpr (kStage) {
    const int rend = (rbase + nthr * R < N) ? rbase + nthr * R : N;
    const int q0 = rbase < N ? P.rowptr[rbase] : 0;
    if (staged && rbase < N) {
      const int total = P.rowptr[rend] - q0;
      for (int q = tid; q < total; q += nthr) {
        const uint32_t e = P.nbr[q0 + q];
        s_list[q] = (e >> 2) | ((e & 3u) == kHopNeg ? 0x80000000u : 0u);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rbase + tid + i * nthr;
      rw[i] = rn[i] = 0;
      dg[i] = S(0);
      if (r < N) {
        const int qa = P.rowptr[r], qb = P.rowptr[r + 1];
        int nh = 0;
        while (qa + nh < qb && (P.nbr[qa + nh] & 3u) != kPlaq) ++nh;
        rw[i] = qa - q0;
        rn[i] = nh | ((qb - qa) << 16);
        dg[i] = cE * S(P.e2[r]) + cm * S(P.stag[r]);
      }
    }
  }

  A w[R];  // this thread's rows of the residual (mixed: double-float pairs)
  double x[R];  // its rows of the start, Ritz and final vectors
  // start vector: normal(seed, k) into V_0, normalised
  double nrm = 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rbase + tid + i * nthr;
    x[i] = (r < N) ? (prm.start_given ? U.psi[size_t(r) * U.psi_stride]
                                      : start_normal(prm.seed, U.k, r))
                   : 0.0;
    nrm += x[i] * x[i];
  }
  unit_sum(nrm);
  nrm = s_sum[1];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rbase + tid + i * nthr;
    if (r < N) put_v(0, i, r, S(x[i] / nrm));
  }
  unit_sync();

  int n = 0, restarts = 0, steps = 0;
  bool converged = false;
  double theta = 0.0, resid = 0.0;
  for (int cycle = 0;; ++cycle) {
    n = 0;
    bool exhausted = false;
    if (tid == 0) {
      s_zwarm = 0;
      s_next = 2 * prm.check_every;
      s_pstep = 0;
      s_pres = 0.0;
    }
    __syncthreads();
    for (int j = 0; j < m; ++j) {
      const S* vj = vs ? s_x : V + size_t(j) * N;
      // w = H v_j (matvec in the storage precision)
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = rbase + tid + i * nthr;
        S acc = S(0);
        if (r < N) {
          bool done = false;
          if constexpr (kStage) {
            if (staged) {
              const uint32_t* l = s_list + rw[i];
              const int nh = rn[i] & 0xffff, n1 = rn[i] >> 16;
              S sh = S(0), sp = S(0);
              if constexpr (kDF) {
                for (int q = 0; q < n1; q += 4) {
                  uint32_t ent[4];
                  float v[4];
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    ent[u] = (q + u < n1) ? l[q + u] : 0u;
                    v[u] = (q + u < n1) ? float(vj[ent[u] & 0x7fffffffu]) : 0.f;
                  }
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    if (q + u < nh) sh += flip_sign(v[u], ent[u]);
                    else sp += v[u];
                  }
                }
              } else {
                double t[1];
                auto load = [&](uint32_t e, double(&v)[1]) { v[0] = vj[e]; };
                int_sum<1, 8, true>(l, 0, nh, t, load);
                sh = S(t[0]);
                if (n1 > nh) {
                  int_sum<1, 8, false>(l, nh, n1, t, load);
                  sp = S(t[0]);
                }
              }
              acc = fma(ch, sh, dg[i] * vj[r]);
              if (n1 > nh) acc = fma(cp, sp, acc);
              done = true;
            }
          }
          if (!done) {
            acc = (cE * S(P.e2[r]) + cm * S(P.stag[r])) * vj[r];
            const int q1 = P.rowptr[r + 1];
            for (int q = P.rowptr[r]; q < q1; ++q) {
              const uint32_t e = __ldg(P.nbr + q);
              const uint32_t kind = e & 3u;
              const S c = (kind == kPlaq) ? cp : ((kind == kHopNeg) ? -ch : ch);
              acc = fma(c, vj[e >> 2], acc);
            }
          }
        }
        if constexpr (kDF) w[i] = df{float(acc), 0.f};
        else w[i] = acc;
      }
      // Classical Gram-Schmidt against the whole basis V_0..V_j (which also
      // performs the three-term recurrence), eight basis vectors per round so
      // that their sums over the lanes overlap.  A further pass (up to
      // prm.reorth) runs only when a pass cancels more than two digits,
      // ||w_after||^2 < 1e-4 ||w_before||^2: the rounding error it leaves along
      // the basis is then above eps * 100 relative to w.
      // ||w||^2 before the first pass comes with that pass's dots: w against
      // itself in slot j + 1 (no separate block reduction)
      for (int pass = 0;; ++pass) {
        const int jd = (pass == 0) ? j + 1 : j;
        for (int b0 = 0; b0 <= jd; b0 += 8) {
          A pd[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) pd[q] = zero();
#pragma unroll
          for (int i = 0; i < R; ++i) {
            const int r = rbase + tid + i * nthr;
            if (r < N) {
              S v[8];
#pragma unroll
              for (int q = 0; q < 8; ++q)
                v[q] = (b0 + q <= j) ? V[size_t(b0 + q) * vst + vo + i * nthr] : S(0);
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                if constexpr (kDF) {
                  if (b0 + q <= j) df_fma2(pd[q], v[q], w[i].hi, w[i].lo);
                  else if (b0 + q == jd) df_sq2(pd[q], w[i].hi, w[i].lo);
                } else {
                  if (b0 + q <= j) pd[q] = fma(v[q], w[i], pd[q]);
                  else if (b0 + q == jd) pd[q] = fma(w[i], w[i], pd[q]);
                }
              }
            }
          }
          A kk;
          if constexpr (kDF) kk = warp_scatter8_df(pd, lane);
          else kk = warp_scatter8_int(pd, lane);
          const int slot = b0 + (lane >> 2);
          if ((lane & 3) == 0 && slot <= jd) {
            const int at = int(cr) * nwarps + wid;
            s_part[slot][at] = kk;
            if (CL == 2) ppeer[slot * (CL * kWarpsCta) + at] = kk;
          }
        }
        unit_sync();
        // eight lanes add a slot's totals of all warps of the unit
        const int nv = CL * nwarps, ngrp = nthr >> 3, sub = tid & 7;
        for (int s0 = 0; s0 <= jd; s0 += ngrp) {
          const int slot = s0 + (tid >> 3);
          A v = zero();
          if (slot <= jd)
            for (int q = sub; q < nv; q += 8) {
              if constexpr (kDF) v = df_add(v, s_part[slot][q]);
              else v += s_part[slot][q];
            }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            if constexpr (kDF) v = df_add(v, shfl_xor_df(v, o));
            else v += __shfl_xor_sync(0xffffffffu, v, o);
          }
          if (slot <= jd && sub == 0) {
            if constexpr (kDF) {
              s_hh[slot] = v.hi;
              s_hl[slot] = v.lo;
            } else {
              s_h[slot] = v;
            }
            if (slot == j) s_alpha[j] = (pass == 0) ? as_double(v) : s_alpha[j] + as_double(v);
            if (slot == j + 1) s_nb = as_double(v);
          }
        }
        __syncthreads();
        if (tid == nthr - 1) {  // for thread 0 after the next barrier
          double scl = fabs(s_alpha[j]);
          if (j > 0) scl = fmax(scl, s_beta[j - 1]);
          s_thr = tiny_rel * fmax(scl, 1.0);
          s_lim = 1e-4 * s_nb;
        }
        // w -= sum_b h_b V_b.  Mixed: the leading parts by TwoSum, the
        // trailing parts apart, renormalised at the end (Dot2 form)
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int r = rbase + tid + i * nthr;
          if (r < N) {
            for (int b0 = 0; b0 <= j; b0 += 8) {
              S v[8];
#pragma unroll
              for (int q = 0; q < 8; ++q)
                v[q] = (b0 + q <= j) ? V[size_t(b0 + q) * vst + vo + i * nthr] : S(0);
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (b0 + q <= j) {
                  if constexpr (kDF) {
                    float p, e, t;
                    two_prod(s_hh[b0 + q], v[q], p, e);
                    e = df_fma_rn(s_hl[b0 + q], v[q], e);
                    two_sum(w[i].hi, -p, w[i].hi, t);
                    w[i].lo = df_add_rn(w[i].lo, df_sub_rn(t, e));
                  } else {
                    w[i] = fma(-s_h[b0 + q], v[q], w[i]);
                  }
                }
            }
            if constexpr (kDF) fast_two_sum(w[i].hi, w[i].lo, w[i].hi, w[i].lo);
          }
        }
        A n2 = zero();
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if constexpr (kDF) df_sq2(n2, w[i].hi, w[i].lo);
          else n2 = fma(w[i], w[i], n2);
        }
        // beta = ||w||, 1 / beta, the exhaustion test of this step and the
        // need of a further pass, by thread 0
        unit_reduce<CL>(n2, s_nslot, par_n, [&](double sv) {
          const double rs = inv_sqrt(sv);
          const double b = sv * rs;
          s_beta[j] = b;
          s_sum[2] = rs;
          if (kDF) {
            const float rh = narrow(rs);
            s_rb[0] = rh;
            s_rb[1] = narrow(rs - widen(rh));
          }
          s_exh = (b > s_thr) ? 0 : 1;
          // (as integers: neither is negative, and an FP64 comparison is 64 cycles)
          s_more = __double_as_longlong(sv) < __double_as_longlong(s_lim) ? 1 : 0;
          s_nb = sv;
        });
        if (!s_more || pass + 1 >= prm.reorth) break;
      }
      const double rbeta = s_sum[2];
      n = j + 1;
      ++steps;
      if (s_exh) {
        exhausted = true;
      } else if (j + 1 < m + 1) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int r = rbase + tid + i * nthr;
          if constexpr (kDF) {
            // (wh + wl)(rh + rl) to FP32: the leading product and the two
            // cross terms, one final rounding
            if (r < N)
              put_v(j + 1, i, r,
                    S(df_fma_rn(w[i].hi, s_rb[0],
                                df_fma_rn(w[i].hi, s_rb[1], df_mul_rn(w[i].lo, s_rb[0])))));
          } else {
            if (r < N) put_v(j + 1, i, r, to_storage<S>(w[i] * rbeta));
          }
        }
      }
      // first check after 2 * check_every steps, then every check_every, or
      // sooner where the residual's geometric decay between the last two
      // checks predicts convergence (s_next)
      const bool check = exhausted || (j + 1 == m) || (j + 1 >= s_next);
      if (check) {
        unit_sync();
        if (wid == 0) {
          double th, rr = 0.0;
          bool conv = false;
          if constexpr (kDF) {
            th = warp_check_lowest_f32(s_alpha, s_beta, n, s_beta[n - 1], s_zwarm != 0, s_theta,
                                       s_resid, s_z, s_work, &rr);
          } else {
            conv = warp_check_lowest(s_alpha, s_beta, n, s_beta[n - 1], tol,
                                     exhausted || j + 1 == m, s_zwarm != 0, s_theta, s_resid, s_z,
                                     s_work, &th, &rr);
          }
          if (lane == 0) {
            if (exhausted) rr = 0.0;
            // FP32 panels resolve residuals to ~1e-6 |H|: relative floor
            const double tl = fp32 ? fmax(tol, 3e-6 * fmax(fabs(th), 1.0)) : tol;
            s_flag = (exhausted || (kDF ? rr <= tl : conv)) ? 1 : 0;
            int nxt = n + prm.check_every;
            if (s_pstep > 0 && rr > tl && s_pres > rr) {
              const float rate = logf(float(rr) / float(s_pres)) / float(n - s_pstep);  // < 0
              // steps to the tolerance at that rate (a 25% margin measured
              // slower: 121k vs 124.7k GS/s on the 4x2 batch)
              const float need = logf(float(tl) / float(rr)) / rate;  // > 0 steps
              if (need < float(prm.check_every)) {
                const int p = n + ((need > 1.0f) ? int(ceilf(need)) : 1);
                if (p < nxt) nxt = p;
              }
            }
            s_next = nxt;
            s_pstep = n;
            s_pres = rr;
            s_theta = th;
            s_resid = rr;
            s_zwarm = 1;
            for (int i = n; i < kMaxM; ++i) s_z[i] = 0.0;
          }
        }
        __syncthreads();
        theta = s_theta;
        resid = s_resid;
        if (s_flag) {
          converged = true;
          break;
        }
      } else {
        unit_sync();
      }
      if (exhausted) break;
    }
    // Ritz vector x = sum z_i V_i (z of the last check, at size n)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rbase + tid + i * nthr;
      double xv = 0.0;
      if (r < N)
        for (int b = 0; b < n; ++b)
          xv = fma(s_z[b], widen(V[size_t(b) * vst + vo + i * nthr]), xv);
      x[i] = xv;
    }
    if (converged || cycle >= prm.maxiter) break;
    // restart from the Ritz vector
    double s2 = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) s2 = fma(x[i], x[i], s2);
    unit_sum(s2);
    const double xn = s_sum[1];
    // every CTA of the unit has formed its Ritz rows from the old basis
    unit_sync();
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rbase + tid + i * nthr;
      if (r < N) put_v(0, i, r, S(x[i] / xn));
    }
    unit_sync();
    ++restarts;
  }

  // FP64 finish: x normalised, y = H x in FP64, E = <x|y>, ||y - E x||
  double s2 = 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) s2 = fma(x[i], x[i], s2);
  unit_sum(s2);
  const double xn = s_sum[1];
  double* X = U.x;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rbase + tid + i * nthr;
    x[i] /= xn;
    if (r < N) X[r] = x[i];
  }
  unit_sync();
  double y[R];
  double ey = 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rbase + tid + i * nthr;
    y[i] = 0.0;
    if (r < N) {
      double acc = (U.cE * double(P.e2[r]) + U.cm * double(P.stag[r])) * X[r];
      bool done = false;
      if constexpr (kStage) {
        if (staged) {
          const uint32_t* l = s_list + rw[i];
          const int nh = rn[i] & 0xffff, n1 = rn[i] >> 16;
          double t[1];
          auto load = [&](uint32_t e, double(&v)[1]) { v[0] = X[e]; };
          int_sum<1, 8, true>(l, 0, nh, t, load);
          acc = fma(U.ch, t[0], acc);
          if (n1 > nh) {
            int_sum<1, 8, false>(l, nh, n1, t, load);
            acc = fma(U.cp, t[0], acc);
          }
          done = true;
        }
      }
      if (!done) {
        const int q1 = P.rowptr[r + 1];
        for (int q = P.rowptr[r]; q < q1; ++q) {
          const uint32_t e = __ldg(P.nbr + q);
          const uint32_t kind = e & 3u;
          const double c = (kind == kPlaq) ? U.cp : ((kind == kHopNeg) ? -U.ch : U.ch);
          acc = fma(c, X[e >> 2], acc);
        }
      }
      y[i] = acc;
    }
    ey = fma(x[i], y[i], ey);
  }
  const double Erq = unit_sum(ey);
  double rs = 0.0;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const double d = y[i] - Erq * x[i];
    rs = fma(d, d, rs);
  }
  unit_sum(rs);
  const double rnorm = s_sum[1];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rbase + tid + i * nthr;
    if (r < N) U.psi[size_t(r) * U.psi_stride] = x[i];
  }
  if (tid == 0 && cr == 0) {
    U.out[0] = fp32 ? Erq : theta;
    U.out[1] = rnorm;
    U.out[2] = double(steps);
    U.out[3] = double(restarts);
    U.out[4] = converged ? 1.0 : 0.0;
    U.out[5] = resid;
  }
  // no CTA of a split unit leaves while its peer may still access its
  // shared memory
  if constexpr (CL == 2) cooperative_groups::this_cluster().sync();
}

// Rows per thread R (a template case: the rows live in registers) and just
// enough whole warps for the largest sector: idle lanes still occupy the
// FP64 pipe in every warp instruction.  rows_per_thread = 0 takes the
// smallest R with maxN <= 512 R; a larger R means fewer threads.
// Environment switch (default `def`): "0" turns it off.
bool getenv_flag(const char* name, int def) {
  const char* e = getenv(name);
  if (!e || !e[0]) return def != 0;
  return e[0] != '0';
}

// Dynamic shared memory a CTA may take beside the kernel's static arrays.
constexpr int kCtaSmemMax = 200 * 1024;

// CL = 2 splits every unit over a cluster of two CTAs (cluster launch); the
// rows per thread then count half a sector.
template <typename S>
cudaError_t launch_cta(const SmallProblem* probs, const SmallUnit* units, int nunits, int maxN,
                       const SmallParams& prm_in, cudaStream_t s, int rows_per_thread,
                       int cl = 1) {
  const int rowsN = (cl == 2) ? (maxN + 1) / 2 : maxN;  // rows a CTA holds
  int R = (rowsN + kCta - 1) / kCta;
  if (rows_per_thread > R) R = rows_per_thread;
  auto threads_for = [&](int rr) {
    int t = ((rowsN + rr - 1) / rr + 31) / 32 * 32;
    return t < 64 ? 64 : t;  // the reduction of step j uses threads 0..j
  };
  // shared memory: a CTA's rows of the Krylov basis with the current vector,
  // and its neighbour lists (R <= 4), each when the largest sector's fit
  SmallParams prm = prm_in;
  const int mmax = (prm.m < maxN) ? prm.m : maxN;
  auto up = [](size_t b) { return (b + 15) / 16 * 16; };
  auto layout = [&](int rr) -> int {
    const size_t rows = size_t(threads_for(rr)) * rr;
    const size_t vb = up(size_t(mmax + 1) * rows * sizeof(S)), xb = up(size_t(maxN) * sizeof(S));
    const size_t lb =
        (rr <= 4 && prm.max_moves > 0)
            ? up(std::min(rows, size_t(maxN)) * size_t(prm.max_moves) * sizeof(uint32_t))
            : 0;
    size_t o = 0;
    prm.v_smem = getenv_flag("LGT_CTA_BASIS_SMEM", 1) && vb + xb <= size_t(kCtaSmemMax) ? 1 : 0;
    prm.x_off = int(vb);
    if (prm.v_smem) o = vb + xb;
    prm.list_cap = lb > 0 && o + lb <= size_t(kCtaSmemMax) ? 1 : 0;
    prm.list_off = int(o);
    return int(o + (prm.list_cap ? lb : 0));
  };
  auto go = [&](auto kern, int rr) -> cudaError_t {
    const int dyn = layout(rr);
    if (dyn > 0) {  // static + dynamic may pass 48 KB: opt in per device
      cudaError_t ea = lgt::raise_smem_limit(reinterpret_cast<const void*>(kern), kCtaSmemMax);
      if (ea != cudaSuccess) return ea;
    }
    if (cl == 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(unsigned(nunits) * 2u);
      cfg.blockDim = dim3(unsigned(threads_for(rr)));
      cfg.dynamicSmemBytes = size_t(dyn);
      cfg.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 2;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      cudaError_t e = cudaLaunchKernelEx(&cfg, kern, probs, units, prm);
      lgt::note_launch();
      if (e != cudaSuccess) return e;
      return cudaGetLastError();
    }
    kern<<<nunits, threads_for(rr), dyn, s>>>(probs, units, prm), lgt::note_launch();
    return cudaGetLastError();
  };
#define LGT_CTA_CASE(RR)                                                   \
  if (R <= RR) {                                                           \
    if (cl == 2) return go(k_lanczos_cta<S, RR, 2>, RR);                   \
    return go(k_lanczos_cta<S, RR, 1>, RR);                                \
  }
  LGT_CTA_CASE(1)
  LGT_CTA_CASE(2)
  LGT_CTA_CASE(3)
  LGT_CTA_CASE(4)
  LGT_CTA_CASE(8)
  LGT_CTA_CASE(16)
#undef LGT_CTA_CASE
  return cudaErrorInvalidValue;
}

}  // namespace

std::string build_pattern(const BasisDev& B, uint32_t model, Pattern* P, cudaStream_t s) {
  const int64_t N = B.dim;
  if (N > kSmallMaxN) return "sector too large for the per-CTA solver";
  P->N = int(N);
  P->model = model;
  P->max_moves = B.G.max_moves > 0 ? B.G.max_moves : 1;
  // Stream-ordered: the neighbour array is sized for the most moves a row can
  // have (at most kSmallMaxN rows, so a few MB at most) instead of reading
  // the exact count back; the fill kernel checks its bounds.
  const Geom& G = B.G;
  const size_t cap = size_t(N) * size_t(G.max_moves > 0 ? G.max_moves : 1);
  // one pool allocation for the row pointers, the diagonal features, the
  // neighbour entries and the scan's counts (256-byte aligned pieces)
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) & ~size_t(255);
    return o;
  };
  const size_t o_rowptr = take((size_t(N) + 1) * sizeof(int));
  const size_t o_e2 = take((size_t(N) + 1) * sizeof(int16_t));
  const size_t o_stag = take((size_t(N) + 1) * sizeof(int16_t));
  const size_t o_nbr = take((cap + 1) * sizeof(uint32_t));
  const size_t o_counts = take((size_t(N) + 1) * sizeof(int));
  SCK(dev_alloc(&P->block, at, s));
  char* base = static_cast<char*>(P->block);
  P->rowptr = reinterpret_cast<int*>(base + o_rowptr);
  P->e2 = reinterpret_cast<int16_t*>(base + o_e2);
  P->stag = reinterpret_cast<int16_t*>(base + o_stag);
  P->nbr = reinterpret_cast<uint32_t*>(base + o_nbr);
  int* counts = reinterpret_cast<int*>(base + o_counts);
  const unsigned blocks = unsigned((N + 255) / 256);
  const RankView R = B.view();
  const bool plaq = model & kModelPlaq, jw = model & kModelJW;
  if (plaq && jw) k_pattern_count<true, true><<<blocks, 256, 0, s>>>(G, R, N, counts), lgt::note_launch();
  else if (plaq) k_pattern_count<true, false><<<blocks, 256, 0, s>>>(G, R, N, counts), lgt::note_launch();
  else if (jw) k_pattern_count<false, true><<<blocks, 256, 0, s>>>(G, R, N, counts), lgt::note_launch();
  else k_pattern_count<false, false><<<blocks, 256, 0, s>>>(G, R, N, counts), lgt::note_launch();
  k_scan_rows<<<1, 1024, 0, s>>>(counts, N, P->rowptr), lgt::note_launch();
  P->nnz = -1;  // on the device (rowptr[N]); not needed on the host
  if (plaq && jw)
    k_pattern_fill<true, true><<<blocks, 256, 0, s>>>(G, R, N, P->rowptr, P->nbr, P->e2, P->stag, B.err), lgt::note_launch();
  else if (plaq)
    k_pattern_fill<true, false><<<blocks, 256, 0, s>>>(G, R, N, P->rowptr, P->nbr, P->e2, P->stag, B.err), lgt::note_launch();
  else if (jw)
    k_pattern_fill<false, true><<<blocks, 256, 0, s>>>(G, R, N, P->rowptr, P->nbr, P->e2, P->stag, B.err), lgt::note_launch();
  else
    k_pattern_fill<false, false><<<blocks, 256, 0, s>>>(G, R, N, P->rowptr, P->nbr, P->e2, P->stag, B.err), lgt::note_launch();
  SCK(cudaGetLastError());
  return std::string();
}

void free_small_work(SmallWork* w, cudaStream_t s) {
  dev_free(w->base, s);
  if (w->host) {
    cudaStreamSynchronize(s);  // a copy staged through it may still be in flight
    pinned_put(w->host, w->host_bytes);
  }
  event_put(w->ev[0]);
  event_put(w->ev[1]);
  *w = SmallWork();
}

void free_pattern(Pattern* P, cudaStream_t s) {
  dev_free(P->block, s);
  *P = Pattern();
}

std::string small_ground_states(const std::vector<SmallJob>& jobs, const SmallParams& prm_in,
                                int mixed, SmallWork* ws, cudaStream_t s, double* seconds,
                                const int* dev_err, int* err_out,
                                const std::function<cudaError_t()>& before_sync) {
  SmallParams prm = prm_in;
  for (const SmallJob& jb : jobs)
    prm.max_moves = std::max(prm.max_moves, jb.pattern->max_moves);
  // problems and units, the largest sectors first
  std::vector<SmallProblem> probs;
  std::vector<SmallUnit> units;
  std::vector<int> order(jobs.size());
  for (size_t i = 0; i < jobs.size(); ++i) order[i] = int(i);
  std::vector<std::pair<int, int>> sz;
  int maxN = 0;
  size_t vbytes = 0, xbytes = 0;
  const size_t es = mixed ? sizeof(float) : sizeof(double);
  for (size_t i = 0; i < jobs.size(); ++i) {
    const Pattern* P = jobs[i].pattern;
    SmallProblem q;
    q.N = P->N;
    q.rowptr = P->rowptr;
    q.nbr = P->nbr;
    q.e2 = P->e2;
    q.stag = P->stag;
    probs.push_back(q);
    if (P->N > maxN) maxN = P->N;
    const int m = (prm.m < P->N) ? prm.m : P->N;
    vbytes += size_t(jobs[i].K) * (size_t(m + 1) * P->N * es + 256);
    xbytes += size_t(jobs[i].K) * (size_t(P->N) * sizeof(double) + 256);
  }
  if (maxN > kSmallMaxN) return "sector too large for the per-CTA solver";
  if (prm.m > kMaxM - 1) return "krylovdim too large for the per-CTA solver";
  size_t nunits = 0;
  for (auto& j : jobs) nunits += size_t(j.K);
  const size_t need = vbytes + xbytes + nunits * (sizeof(SmallUnit) + 8 * sizeof(double)) +
                      probs.size() * sizeof(SmallProblem) + 4096;
  if (ws->bytes < need) {
    dev_free(ws->base, s);
    ws->base = nullptr;
    ws->bytes = 0;
    ws->up_bytes = 0;
    SCK(dev_alloc(&ws->base, need, s));
    ws->bytes = need;
  }
  char* base = static_cast<char*>(ws->base);
  size_t off = 0;
  auto take = [&](size_t b) {
    char* p = base + off;
    off += (b + 255) / 256 * 256;
    return p;
  };
  SmallProblem* d_probs = reinterpret_cast<SmallProblem*>(take(probs.size() * sizeof(SmallProblem)));
  SmallUnit* d_units = reinterpret_cast<SmallUnit*>(take(nunits * sizeof(SmallUnit)));
  double* d_out = reinterpret_cast<double*>(take(nunits * 8 * sizeof(double)));
  // units sorted by sector size, descending
  std::vector<std::pair<int, size_t>> jorder;
  for (size_t i = 0; i < jobs.size(); ++i) jorder.push_back({-jobs[i].pattern->N, i});
  std::sort(jorder.begin(), jorder.end());
  std::vector<std::pair<size_t, int>> unit_src;  // (job, k)
  for (auto& jo : jorder) {
    const SmallJob& J = jobs[jo.second];
    const int N = J.pattern->N;
    const int m = (prm.m < N) ? prm.m : N;
    for (int k = 0; k < J.K; ++k) {
      SmallUnit u;
      u.prob = int(jo.second);
      u.k = k;
      u.cE = J.cE[k];
      u.cm = J.cm[k];
      u.ch = J.ch[k];
      u.cp = J.cp[k];
      u.psi = J.psi + k;
      u.psi_stride = J.K;
      u.V = take(size_t(m + 1) * N * es);
      u.x = reinterpret_cast<double*>(take(size_t(N) * sizeof(double)));
      u.out = d_out + units.size() * 8;
      units.push_back(u);
      unit_src.push_back({jo.second, k});
    }
  }
  // the tables through the pinned staging buffer, uploaded only when they
  // differ from the copy the device buffer already holds (a repeated solve
  // of the same batch); the outputs come back through it as well
  const size_t pb = sizeof(SmallProblem) * probs.size(), ub = sizeof(SmallUnit) * units.size();
  const size_t tb = (pb + ub + 15) / 16 * 16, ob = sizeof(double) * nunits * 8 + 16;
  if (ws->host_bytes < tb + ob) {
    if (ws->host) {
      SCK(cudaStreamSynchronize(s));
      pinned_put(ws->host, ws->host_bytes);
    }
    ws->host = nullptr;
    ws->host_bytes = 0;
    ws->up_bytes = 0;
    SCK(pinned_get(tb + ob, &ws->host, &ws->host_bytes));
  }
  char* hst = static_cast<char*>(ws->host);
  const bool same = ws->up_bytes == pb + ub && memcmp(hst, probs.data(), pb) == 0 &&
                    memcmp(hst + pb, units.data(), ub) == 0;
  if (!same) {
    memcpy(hst, probs.data(), pb);
    memcpy(hst + pb, units.data(), ub);
    SCK(cudaMemcpyAsync(d_probs, hst, pb, cudaMemcpyHostToDevice, s));
    SCK(cudaMemcpyAsync(d_units, hst + pb, ub, cudaMemcpyHostToDevice, s));
    ws->up_bytes = pb + ub;
  }
  double* h_out = reinterpret_cast<double*>(hst + tb);
  if (!ws->ev[0]) SCK(event_get(&ws->ev[0]));
  if (!ws->ev[1]) SCK(event_get(&ws->ev[1]));
  cudaEvent_t e0 = ws->ev[0], e1 = ws->ev[1];
  auto launch = [&](int rows, int cl) {
    return mixed ? launch_cta<float>(d_probs, d_units, int(nunits), maxN, prm, s, rows, cl)
                 : launch_cta<double>(d_probs, d_units, int(nunits), maxN, prm, s, rows, cl);
  };
  // LGT_CTA_CLUSTER=1 or 2 fixes the CTAs per unit; unset, the tuner decides
  int cl_env = 0;
  if (const char* ce = getenv("LGT_CTA_CLUSTER")) cl_env = (ce[0] == '2') ? 2 : (ce[0] == '1' ? 1 : 0);
  int rows = prm.rows_per_thread;
  int cl = cl_env ? cl_env : 1;
  static std::mutex mu;
  // by what a shape's time depends on: the batch, the models' moves and the
  // Krylov dimension (whether lists and basis fit the shared memory), the device
  int dev = 0;
  SCK(cudaGetDevice(&dev));
  uint32_t models = 0;
  for (const SmallJob& jb : jobs) models |= 1u << (jb.pattern->model & 31u);
  using Key = std::tuple<int, int, int, int, int, uint32_t, int, int>;
  static std::map<Key, std::pair<int, int>> cache;
  const Key key(maxN, int(nunits), mixed ? 1 : 0, cl_env, dev, models, prm.max_moves, prm.m);
  if (rows == 0) {
    // Autotuner over the launch shape: CTAs per unit (1, or a cluster of 2
    // holding half the rows each) and rows per thread R0 (the fewest that
    // fit 512 threads), R0 + 1 or 2 R0 (fewer warps: fewer instructions per
    // basis vector, less latency hiding); timed on this batch once per key,
    // the solve then runs with the fastest.  A solve from a given start vector
    // takes the tuned shape when there is one (else that of another Krylov
    // dimension), else the smallest.
    std::unique_lock<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it == cache.end() && prm.start_given) {
      Key first = key;
      std::get<7>(first) = 0;
      const auto at = cache.lower_bound(first);
      if (at != cache.end()) {
        Key k = at->first;
        std::get<7>(k) = prm.m;
        if (k == key) it = at;
      }
    }
    if (it != cache.end()) {
      rows = it->second.first;
      cl = it->second.second;
    } else if (!prm.start_given) {
      const char* en = getenv("LGT_AUTOTUNE");
      // candidates: for each CTAs-per-unit count, the rows-per-thread cases
      // R0, R0 + 1 and 2 R0 (rounded up to an instantiated case), each with
      // at least 64 threads
      auto round_case = [](int r) { return r <= 3 ? r : (r <= 4 ? 4 : (r <= 8 ? 8 : 16)); };
      std::vector<std::pair<int, int>> cand;
      for (int cc : {1, 2}) {
        if (cl_env && cc != cl_env) continue;
        const int rowsN = (cc == 2) ? (maxN + 1) / 2 : maxN;
        const int r0 = (rowsN + 511) / 512;
        for (int r : {r0, r0 + 1, 2 * r0}) {
          const int rc = round_case(r);
          const auto cp = std::make_pair(rc, cc);
          if (rc <= 16 && (rowsN + rc - 1) / rc >= 64 &&
              std::find(cand.begin(), cand.end(), cp) == cand.end())
            cand.push_back(cp);
        }
        if (cand.empty() || cand.back().second != cc) cand.push_back({r0, cc});
      }
      rows = cand[0].first;
      cl = cand[0].second;
      if (!(en && en[0] == '0') && cand.size() > 1) {
        float best = 3e38f;
        // each candidate twice, the second run counts (a first run pays
        // the kernel's load and cold caches)
        for (int rep = 0; rep < 2; ++rep)
          for (auto& cc : cand) {
            cudaEventRecord(e0, s);
            cudaError_t ce = launch(cc.first, cc.second);
            cudaEventRecord(e1, s);
            if (ce != cudaSuccess && cc.second == 2) {  // no room for the cluster: skip it
              cudaGetLastError();
              SCK(cudaEventSynchronize(e1));
              continue;
            }
            if (ce != cudaSuccess) return std::string("k_lanczos_cta: ") + cudaGetErrorString(ce);
            SCK(cudaEventSynchronize(e1));
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (rep == 1 && ms < best) {
              best = ms;
              rows = cc.first;
              cl = cc.second;
            }
          }
      }
      cache[key] = std::make_pair(rows, cl);
    }
  }
  cudaEventRecord(e0, s);
  cudaError_t e = launch(rows, cl);
  cudaEventRecord(e1, s);
  if (e != cudaSuccess) return std::string("k_lanczos_cta: ") + cudaGetErrorString(e);
  SCK(cudaMemcpyAsync(h_out, d_out, sizeof(double) * nunits * 8, cudaMemcpyDeviceToHost, s));
  int* h_err = reinterpret_cast<int*>(h_out + nunits * 8);
  if (dev_err) SCK(cudaMemcpyAsync(h_err, dev_err, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (before_sync) SCK(before_sync());
  SCK(cudaStreamSynchronize(s));
  if (dev_err && err_out) *err_out |= *h_err;
  const double* out = h_out;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  if (seconds) *seconds = ms * 1e-3;
  for (size_t u = 0; u < nunits; ++u) {
    const SmallJob& J = jobs[unit_src[u].first];
    const int k = unit_src[u].second;
    J.E0[k] = out[u * 8 + 0];
    if (J.resid) J.resid[k] = out[u * 8 + 1];
    if (J.steps) J.steps[k] = int(out[u * 8 + 2]);
    if (J.restarts) J.restarts[k] = int(out[u * 8 + 3]);
    if (J.converged) J.converged[k] = out[u * 8 + 4] != 0.0;
  }
  return std::string();
}

}  // namespace lgt
