// lanczos_grid.cu -- a whole Lanczos cycle of the panel solver
// (find_ground_state, finite_ed.jl:333-341) in one cooperative launch.
//
// The multi-launch driver (krylov.cu) spends eleven dependent launches a
// step.  For sectors whose residual panel W fits the shared memory of the
// chip (4x3 with K = 16: 30 KB an SM) those launches, their short reductions
// and the read-backs of the convergence checks outweigh the work: the 4x3
// K = 1 mixed solve took 0.1 ms a step for 7 MB of basis vectors.  Here one
// block per SM owns a contiguous row range for the whole cycle:
//
//   W = H V_j        neighbour lists and W in shared memory, V_j from L2
//   h = V^T W        per-block partials, one grid barrier, one warp per
//                    output adds them in block order, one barrier
//   W -= V h, |W|    another barrier; every block adds the norms itself
//   V_{j+1} = W / b  a last barrier orders the vector before its gathers
//
// and the convergence checks run in the same launch (one warp per point).
// Columns that have converged or are exhausted leave the active list, so the
// remaining ones get all threads.  Arithmetic as in the multi-launch driver:
// FP32 panels with double-float dots and updates, FP64 panels in FP64; a
// further Gram-Schmidt pass runs for the columns that cancelled more than
// two digits.  All sums have a fixed order, and every block derives the same
// decisions from the same values.
//
// The grid barrier counts arrivals in one word; its wait is bounded by the
// SM clock (GridArgs::spin).  Where it runs out, the blocks leave and no step
// count is written; the driver then takes the multi-launch steps.
#include <type_traits>

#include "lgt_dfloat.cuh"
#include "lgt_internal.h"
#include "lgt_intsum.cuh"
#include "lgt_lanczos_grid.h"
#include "lgt_tridiag.cuh"

namespace lgt {

namespace {

// 512 threads: the block sums of the dots cost threads x slots additions,
// and 16 warps with 16 to 32 loads each already cover the L2 latency (1024
// threads with 4-vector chunks: dots 122k cycles a step at 4x3 K = 16 and
// 66k at K = 1, most of it those sums).
template <typename S>
struct Threads {
  // FP64: 168 registers a thread, so that the loads ahead do not spill (L1 has
  // what shared memory leaves)
  static constexpr int n = sizeof(S) == 4 ? 512 : 384;
};
constexpr int kQ = 8;               // basis vectors per dot chunk
constexpr int kSmemMax = 214 * 1024;  // beside the static arrays

enum : int { kActive = 0, kExhausted = 1, kConverged = 2 };  // as krylov.cu

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ float flip(float v, uint32_t ent) {
  return __uint_as_float(__float_as_uint(v) ^ (ent & 0x80000000u));
}

// Shared-memory layout of a block.
struct Layout {
  int W, list, meta, loff, h, red, coef, cols, total;
};
template <typename S>
__host__ __device__ inline Layout layout(int rpb, int C, int m, int mm, int list_smem) {
  constexpr int kNT = Threads<S>::n;
  auto up = [](int b) { return (b + 15) / 16 * 16; };
  Layout L;
  int o = 0;
  L.W = o;
  o += up(rpb * C * 8);  // FP32: the leading parts, then the trailing ones
  L.list = o;
  o += list_smem ? up(rpb * mm * 4) : 0;
  L.meta = o;
  o += up(rpb * 4);
  L.loff = o;
  o += up(rpb * 4);
  L.h = o;  // [m][C] coefficients: doubles, or float pairs hi, lo
  o += up(m * C * 8);
  L.red = o;  // [kQ + 1][kNT] doubles
  o += (kQ + 1) * kNT * 8;
  L.coef = o;  // [4][C]
  o += up(4 * C * int(sizeof(S)));
  L.cols = o;  // doubles nb, nrm, alpha, beta_prev; ints act, need, status
  o += up(C * (4 * 8 + 3 * 4));
  L.total = o;
  return L;
}

template <typename S>
__global__ void __launch_bounds__(Threads<S>::n, 1) k_lanczos_grid(GridArgs<S> a) {
  constexpr int kNT = Threads<S>::n, kNW = kNT / 32;
  constexpr bool kDF = sizeof(S) == 4;
  constexpr int kU = kDF ? 2 : 1;  // rows per trip
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_n, s_bad;
  __shared__ S s_int[256], s_stag[256];  // small integers: conversions to FP64 are slow
  __shared__ double s_ta[kTriMax], s_tb[kTriMax], s_tz[kTriMax];
  __shared__ __align__(16) double s_work[3 * kTriMax];
  const Layout L = layout<S>(a.rpb, a.C, a.m, a.mm, a.list_smem);
  S* s_W = reinterpret_cast<S*>(smem + L.W);
  S* s_lo = s_W + a.rpb * a.C;  // (FP32 only)
  uint32_t* s_list = reinterpret_cast<uint32_t*>(smem + L.list);
  uint32_t* s_meta = reinterpret_cast<uint32_t*>(smem + L.meta);
  uint32_t* s_loff = reinterpret_cast<uint32_t*>(smem + L.loff);
  double* s_h = reinterpret_cast<double*>(smem + L.h);
  float* s_hh = reinterpret_cast<float*>(smem + L.h);
  const int C = a.C, m = a.m;
  const uint32_t vs = uint32_t(a.vstride);  // (m + 1) N C < 2^32: the plan checks it
  float* s_hl = s_hh + m * C;
  using Acc = typename std::conditional<kDF, df, double>::type;  // running sums
  Acc* s_red = reinterpret_cast<Acc*>(smem + L.red);
  auto add = [](Acc x, Acc y) -> Acc {
    if constexpr (kDF) return df_add(x, y);
    else return x + y;
  };
  auto zero = []() -> Acc {
    if constexpr (kDF) return df{0.f, 0.f};
    else return 0.0;
  };
  S* s_coef = reinterpret_cast<S*>(smem + L.coef);
  double* s_nb = reinterpret_cast<double*>(smem + L.cols);
  double* s_nrm = s_nb + C;
  double* s_al = s_nrm + C;
  double* s_bp = s_al + C;
  int* s_act = reinterpret_cast<int*>(s_bp + C);
  int* s_need = s_act + C;
  int* s_st = s_need + C;

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int blk = blockIdx.x, G = a.nblk;
  const int64_t r0 = int64_t(blk) * a.rpb;
  const int nr = (a.N - r0 < a.rpb) ? int(a.N - r0) : a.rpb;
  unsigned target = 0;

  // false when the wait ran out (the block then leaves)
  auto grid_barrier = [&]() -> bool {
    __syncthreads();
    if (tid == 0) {
      target += unsigned(G);
      __threadfence();
      atomicAdd(a.bar, 1u);
      const long long t0 = clock64();
      while (int(ld_acquire(a.bar) - target) < 0)
        if (clock64() - t0 > a.spin) {
          s_bad = 1;
          break;
        }
      __threadfence();
    }
    __syncthreads();
    return s_bad == 0;
  };
  // the columns c with pred(c), in order, into list; returns their number
  auto compact = [&](int* list, auto pred) -> int {
    __syncthreads();
    if (wid == 0) {
      int n = 0;
      for (int c0 = 0; c0 < C; c0 += 32) {
        const int c = c0 + lane;
        const bool f = c < C && pred(c);
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        if (f) list[n + __popc(bal & ((1u << lane) - 1u))] = c;
        n += __popc(bal);
      }
      if (lane == 0) s_n = n;
    }
    __syncthreads();
    return s_n;
  };
  // sums red[q][g * nl + ci] over the row groups g for q < nq, ci < nl, in a
  // fixed order, and hands each sum to put(q, ci)
  auto group_sums = [&](int nq, int nl, int RG, auto put) {
    __syncthreads();
    const int nout = nq * nl;
    int LN = 32;
    while (LN > 1 && nout * LN > kNT) LN >>= 1;  // (LN divides a warp)
    for (int o0 = 0; o0 < nout; o0 += kNT / LN) {
      const int o = o0 + tid / LN;
      const int q = o / nl, ci = o - q * nl;
      Acc v = zero();
      if (o < nout)
        for (int g = tid % LN; g < RG; g += LN) v = add(v, s_red[q * kNT + g * nl + ci]);
      for (int d = LN >> 1; d > 0; d >>= 1) {
        if constexpr (kDF)
          v = df_add(v, df{__shfl_xor_sync(0xffffffffu, v.hi, d),
                           __shfl_xor_sync(0xffffffffu, v.lo, d)});
        else
          v += __shfl_xor_sync(0xffffffffu, v, d);
      }
      if (o < nout && tid % LN == 0) {
        if constexpr (kDF) put(q, ci, widen(v.hi) + widen(v.lo));
        else put(q, ci, v);
      }
    }
    __syncthreads();
  };

  if (tid == 0) s_bad = 0;
  for (int i = tid; i < 256; i += kNT) {
    s_int[i] = S(i);
    s_stag[i] = S(i - 128);
  }
  for (int i = tid; i < C; i += kNT) {
    s_coef[i] = a.cE[i];
    s_coef[C + i] = a.cm[i];
    s_coef[2 * C + i] = a.ch[i];
    s_coef[3 * C + i] = a.cp[i];
    s_st[i] = a.status[i];
    s_bp[i] = 0.0;
  }
  const uint32_t lbase = nr > 0 ? a.off[r0 >> 5] : 0u;
  for (int t = wid; t * 32 < nr; t += kNW) {
    const int r = t * 32 + lane;
    const uint32_t mw = (r < nr) ? a.meta[r0 + r] : 0u;
    const int cnt = int(mw & 255u);
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    if (r < nr) {
      s_meta[r] = mw;
      s_loff[r] = a.off[(r0 >> 5) + t] - lbase + uint32_t(incl - cnt);
    }
  }
  if (a.list_smem && nr > 0) {
    const uint32_t total = a.off[(r0 + nr + 31) >> 5] - lbase;
    for (uint32_t i = tid; i < total; i += kNT) s_list[i] = a.nbr[lbase + i];
  }
  const uint32_t* list = a.list_smem ? s_list : a.nbr + lbase;

  int nact = compact(s_act, [&](int c) { return s_st[c] == kActive; });
  int j = 0;
  while (j < m && nact > 0) {
    const S* Vj = a.V + size_t(j) * a.vstride;
    // ---- W = H V_j on the active columns
    {
      const int RG = kNT / nact, ci = tid % nact, rg = tid / nact;
      if (rg < RG) {
        const int c = s_act[ci];
        const S cE = s_coef[c], cm = s_coef[C + c], ch = s_coef[2 * C + c], cp = s_coef[3 * C + c];
        for (int r = rg; r < nr; r += RG) {
          const uint32_t mw = s_meta[r];
          const int n1 = int(mw & 255u), nh = int((mw >> 8) & 255u);
          const uint32_t* l = list + s_loff[r];
          const S xd = Vj[size_t(r0 + r) * C + c];
          S sh = S(0), sp = S(0);
          if constexpr (!kDF) {
            double t[1];
            auto load = [&](uint32_t i, double(&v)[1]) { v[0] = Vj[size_t(i) * C + c]; };
            int_sum<1, 8, true>(l, 0, nh, t, load);
            sh = t[0];
            if (n1 > nh) {
              int_sum<1, 8, false>(l, nh, n1, t, load);
              sp = t[0];
            }
          } else {
            for (int n = 0; n < n1; n += 8) {
              S v[8];
              uint32_t ent[8];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (n + u < n1) {
                  ent[u] = l[n + u];
                  v[u] = Vj[size_t(ent[u] & 0x7fffffffu) * C + c];
                }
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (n + u < n1) {
                  if (n + u < nh) sh += flip(v[u], ent[u]);
                  else sp += v[u];
                }
            }
          }
          const S cd = fma(cE, s_int[(mw >> 16) & 255u], cm * s_stag[mw >> 24]);
          S y = fma(ch, sh, cd * xd);
          if (n1 > nh) y = fma(cp, sp, y);
          s_W[r * C + c] = y;
        }
      }
      __syncthreads();
    }
    const int J = j + 1;
    const int* lst = s_act;
    int nl = nact;
    for (int pass = 0;; ++pass) {
      const int RG = kNT / nl, ci = tid % nl, rg = tid / nl;
      const bool on = rg < RG;
      const int c = on ? lst[ci] : 0;
      const S* Vc = a.V + size_t(r0) * C + c;
      // ---- dots against V_0 .. V_j (and W itself in the first pass)
      for (int i0 = 0; i0 < J; i0 += kQ) {
        const bool self = pass == 0 && i0 == 0;
        if (on) {
          Acc acc[kQ], ss = zero();
#pragma unroll
          for (int q = 0; q < kQ; ++q) acc[q] = zero();
          // rows r, r + RG, ... (kU at once); those past the block's count as
          // zeros
          auto load = [&](int r, S(&v)[kQ][kU]) {
#pragma unroll
            for (int q = 0; q < kQ; ++q)
#pragma unroll
              for (int u = 0; u < kU; ++u)
                v[q][u] = (i0 + q < J && r + u * RG < nr)
                              ? Vc[uint32_t(i0 + q) * vs + uint32_t((r + u * RG) * C)]
                              : S(0);
          };
          auto use = [&](int r, const S(&v)[kQ][kU]) {
            S w[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) w[u] = r + u * RG < nr ? s_W[(r + u * RG) * C + c] : S(0);
#pragma unroll
            for (int q = 0; q < kQ; ++q)
              if (i0 + q < J) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                  if constexpr (kDF) df_fma(acc[q], v[q][u], w[u]);
                  else acc[q] = fma(v[q][u], w[u], acc[q]);
                }
              }
            if (self) {
#pragma unroll
              for (int u = 0; u < kU; ++u) {
                if constexpr (kDF) df_fma(ss, w[u], w[u]);
                else ss = fma(w[u], w[u], ss);
              }
            }
          };
          // the next rows' loads are issued before the current rows'
          // arithmetic: the warps of a block run in step, so nothing else
          // covers their latency
          S va[kQ][kU], vb[kQ][kU];
          int r = rg;
          if (r < nr) load(r, va);
          while (r < nr) {
            const int r2 = r + kU * RG, r3 = r2 + kU * RG;
            if (r2 < nr) load(r2, vb);
            use(r, va);
            if (r2 >= nr) break;
            if (r3 < nr) load(r3, va);
            use(r2, vb);
            r = r3;
          }
#pragma unroll
          for (int q = 0; q < kQ; ++q) s_red[q * kNT + tid] = acc[q];
          if (self) s_red[kQ * kNT + tid] = ss;
        }
        // slot kQ (the self-dot) goes to row J of the partials
        const int nv = J - i0 < kQ ? J - i0 : kQ;
        group_sums(self ? kQ + 1 : nv, nl, RG, [&](int q, int cj, double v) {
          const int i = q == kQ ? J : i0 + q;
          if (q == kQ || q < nv) a.part[(size_t(i) * C + lst[cj]) * G + blk] = v;
        });
      }
      if (!grid_barrier()) return;
      // ---- one warp per output over the blocks' partials
      const int Jd = J + (pass == 0 ? 1 : 0);
      for (int o = blk * kNW + wid; o < Jd * nl; o += G * kNW) {
        const int i = o / nl, cc = lst[o - i * nl];
        const double* p = a.part + (size_t(i) * C + cc) * G;
        double v = 0.0;
        for (int b = lane; b < G; b += 32) v += __ldcg(p + b);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        if (lane == 0) a.h[size_t(i) * C + cc] = v;
      }
      if (!grid_barrier()) return;
      for (int o = tid; o < Jd * nl; o += kNT) {
        const int i = o / nl, cc = lst[o - i * nl];
        const double v = __ldcg(a.h + size_t(i) * C + cc);
        if (i == J) {
          s_nb[cc] = v;
        } else {
          if constexpr (kDF) {
            const float hh = narrow(v);
            s_hh[i * C + cc] = hh;
            s_hl[i * C + cc] = narrow(v - widen(hh));
          } else {
            s_h[i * C + cc] = v;
          }
          if (i == j) s_al[cc] = pass == 0 ? v : s_al[cc] + v;
        }
      }
      __syncthreads();
      // ---- W -= sum_i h_i V_i, and |W|^2
      if (on) {
        Acc n2 = zero();
        // eight vectors at a time, the latest first (the dots read them last,
        // so they are what L2 still holds), W in shared memory between the
        // groups -- with its trailing part in FP32
        for (int i = (J - 1) / 8 * 8; i >= 0; i -= 8) {
          const bool first = i + 8 >= J, last = i == 0;
          auto load = [&](int r, S(&x)[8][kU]) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
              for (int u = 0; u < kU; ++u)
                x[q][u] = (i + q < J && r + u * RG < nr)
                              ? Vc[uint32_t(i + q) * vs + uint32_t((r + u * RG) * C)]
                              : S(0);
          };
          auto use = [&](int r, const S(&x)[8][kU]) {
            S hi[kU], lo[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
              const int at = (r + u * RG) * C + c;
              const bool in = r + u * RG < nr;
              hi[u] = in ? s_W[at] : S(0);
              lo[u] = S(0);
              if (kDF && in && !first) lo[u] = s_lo[at];
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (i + q < J) {
                if constexpr (kDF) {
                  const float hh = s_hh[(i + q) * C + c], hl = s_hl[(i + q) * C + c];
#pragma unroll
                  for (int u = 0; u < kU; ++u) {
                    float p, e, t;
                    two_prod(hh, x[q][u], p, e);
                    e = df_fma_rn(hl, x[q][u], e);
                    two_sum(hi[u], -p, hi[u], t);
                    lo[u] = df_add_rn(lo[u], df_sub_rn(t, e));
                  }
                } else {  // two chains: even and odd vectors
                  const double h = s_h[(i + q) * C + c];
#pragma unroll
                  for (int u = 0; u < kU; ++u) {
                    if (q & 1) lo[u] = fma(-h, x[q][u], lo[u]);
                    else hi[u] = fma(-h, x[q][u], hi[u]);
                  }
                }
              }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
              const int at = (r + u * RG) * C + c;
              S w = hi[u];
              if (!kDF || last) w = hi[u] + lo[u];
              if (r + u * RG < nr) {
                s_W[at] = w;
                if (kDF && !last) s_lo[at] = lo[u];
              }
              if (last) {
                if constexpr (kDF) df_fma(n2, w, w);
                else n2 = fma(w, w, n2);
              }
            }
          };
          S xa[8][kU], xb[8][kU];
          int r = rg;
          if (r < nr) load(r, xa);
          while (r < nr) {
            const int r2 = r + kU * RG, r3 = r2 + kU * RG;
            if (r2 < nr) load(r2, xb);
            use(r, xa);
            if (r2 >= nr) break;
            if (r3 < nr) load(r3, xa);
            use(r2, xb);
            r = r3;
          }
        }
        s_red[tid] = n2;
      }
      group_sums(1, nl, RG, [&](int, int cj, double v) {
        a.npart[size_t(lst[cj]) * G + blk] = v;
      });
      if (!grid_barrier()) return;
      for (int q = wid; q < nl; q += kNW) {
        const double* p = a.npart + size_t(lst[q]) * G;
        double v = 0.0;
        for (int b = lane; b < G; b += 32) v += __ldcg(p + b);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        if (lane == 0) s_nrm[lst[q]] = v;
      }
      if (pass + 1 >= a.reorth) break;
      // a further pass for the columns that cancelled more than two digits;
      // the entries of s_need are read before they are overwritten
      const int cnt = nl;
      __syncthreads();
      bool mine = false;
      int my = 0;
      if (tid < cnt) {
        my = lst[tid];
        mine = s_nrm[my] < 1e-4 * s_nb[my];
      }
      __syncthreads();
      int* mark = reinterpret_cast<int*>(s_red);
      if (tid < C) mark[tid] = 0;
      __syncthreads();
      if (mine) mark[my] = 1;
      __syncthreads();
      if (tid < cnt) s_nb[my] = s_nrm[my];
      const int nn = compact(s_need, [&](int c2) { return mark[c2] != 0; });
      if (nn == 0) break;
      lst = s_need;
      nl = nn;
    }
    __syncthreads();
    // ---- beta, exhaustion, and the new vector
    bool gone = false;
    if (tid < nact) {
      const int c = s_act[tid];
      const double b = sqrt(s_nrm[c]);
      double scale = fabs(s_al[c]);
      if (j > 0) scale = fmax(scale, s_bp[c]);
      gone = !(b > a.tiny_rel * fmax(scale, 1.0));
      s_bp[c] = b;
      s_nrm[c] = (b > 0.0) ? 1.0 / b : 0.0;
      if (gone) s_st[c] = kExhausted;
      if (blk == 0) {
        a.alpha[size_t(c) * a.ldT + j] = s_al[c];
        a.beta[size_t(c) * a.ldT + j] = b;
        a.len[c] = j + 1;
        if (gone) a.status[c] = kExhausted;
      }
    }
    const bool any_gone = __syncthreads_or(gone ? 1 : 0);
    {
      const int RG = kNT / nact, ci = tid % nact, rg = tid / nact;
      if (rg < RG && s_st[s_act[ci]] == kActive) {
        const int c = s_act[ci];
        S* out = a.V + size_t(j + 1) * a.vstride + size_t(r0) * C + c;
        const S inv = S(s_nrm[c]);
        for (int r = rg; r < nr; r += RG) out[r * C] = s_W[r * C + c] * inv;
      }
    }
    if (any_gone) nact = compact(s_act, [&](int c) { return s_st[c] == kActive; });
    ++j;
    if (!grid_barrier()) return;
    // ---- convergence checks, one warp per point over the blocks
    if (j % a.check_every == 0 || j == m || nact == 0) {
      for (int k = blk; k < C; k += G) {
        if (wid == 0) {
          const int st = __ldcg(a.status + k);
          const int n = __ldcg(a.len + k);
          if (st < kConverged && n > 0) {
            for (int i = lane; i < n; i += 32) {
              s_ta[i] = __ldcg(a.alpha + size_t(k) * a.ldT + i);
              s_tb[i] = __ldcg(a.beta + size_t(k) * a.ldT + i);
            }
            __syncwarp();
            const double bn = s_tb[n - 1];
            __syncwarp();
            if (lane == 0) s_tb[n - 1] = 0.0;
            __syncwarp();
            const double tp = __ldcg(a.theta + k), rp = __ldcg(a.resid + k);
            const bool warm = isfinite(tp) && isfinite(rp);
            double th, r;
            bool conv, vec = true;  // vec: s_tz holds the vector
            if constexpr (kDF) {
              th = warp_lowest_eig_f32(s_ta, s_tb, n, s_tz, s_work, warm, tp, rp);
              r = fabs(bn * s_tz[n - 1]);
              conv = r <= a.tol;
            } else {
              const bool need = j == m || st == kExhausted;
              conv = warp_check_lowest(s_ta, s_tb, n, bn, a.tol, need, warm, tp, rp, s_tz, s_work, &th,
                                       &r);
              vec = conv || need;
            }
            for (int i = lane; i < a.ldT && vec; i += 32) {
              a.coef[(size_t(k) * a.ldT + i) * 2 + 0] = (i < n) ? s_tz[i] : 0.0;
              a.coef[(size_t(k) * a.ldT + i) * 2 + 1] = 0.0;
            }
            if (lane == 0) {
              a.theta[k] = th;
              a.resid[k] = (st == kExhausted) ? 0.0 : r;
              if (st == kExhausted || conv) a.status[k] = kConverged;
            }
            __syncwarp();
          }
        }
      }
      if (!grid_barrier()) return;
      for (int c = tid; c < C; c += kNT) s_st[c] = __ldcg(a.status + c);
      nact = compact(s_act, [&](int c) { return s_st[c] == kActive; });
    }
  }
  if (blk == 0 && tid == 0) *a.steps = j;
}

}  // namespace

template <typename S>
bool lanczos_grid_plan(int64_t N, int C, int m, int mm, int* rpb, int* nblk, int* list_smem,
                       int* bytes) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return false;
  if (N < 1 || C < 1 || C > 256 || m < 1 || m >= kTriMax) return false;
  const int64_t rows = ((N + sms - 1) / sms + 31) / 32 * 32;
  if ((m + 1) * N * C >= (int64_t(1) << 32)) return false;
  if (rows * C > kSmemMax / 8 || rows > kSmemMax / 8) return false;
  for (int ls = 1; ls >= 0; --ls) {
    if (ls && rows * mm > kSmemMax / 4) continue;
    const Layout L = layout<S>(int(rows), C, m, mm, ls);
    if (L.total > kSmemMax) continue;
    *rpb = int(rows);
    *nblk = int((N + rows - 1) / rows);
    *list_smem = ls;
    *bytes = L.total;
    return true;
  }
  return false;
}

template <typename S>
cudaError_t launch_lanczos_grid(const GridArgs<S>& a, int bytes, cudaStream_t s) {
  auto kern = k_lanczos_grid<S>;
  // (the static arrays count towards the 48 KB that need no opt-in)
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kern),
                                         bytes > 32 * 1024 ? kSmemMax : bytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(a.nblk));
  cfg.blockDim = dim3(Threads<S>::n);
  cfg.dynamicSmemBytes = size_t(bytes);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, a);
  note_launch();
  if (le != cudaSuccess) return le;
  return cudaGetLastError();
}

template bool lanczos_grid_plan<float>(int64_t, int, int, int, int*, int*, int*, int*);
template bool lanczos_grid_plan<double>(int64_t, int, int, int, int*, int*, int*, int*);
template cudaError_t launch_lanczos_grid<float>(const GridArgs<float>&, int, cudaStream_t);
template cudaError_t launch_lanczos_grid<double>(const GridArgs<double>&, int, cudaStream_t);

}  // namespace lgt
