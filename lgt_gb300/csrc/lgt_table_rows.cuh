// lgt_table_rows.cuh -- the products of the Chebyshev expansion (cheb.cu) from
// the stored neighbour table:
//
//   y = scale ((H + shift) x), minus `prev` where it is given,
//   H x = (cE e2 + cm stag) x + ch sum_hops (+-) x_j + cp sum_plaq x_j
// (T_{n+1} = 2 H~ T_n - T_{n-1}; finite_ed.jl:265-318,
// matter_gauge_entanglement_pjw.jl:82-147).  A panel row holds (re, im) of K
// points.
//
// A warp copies the meta words and entries of its 32 rows into shared memory
// (coalesced, evict-first) and runs its lanes over (row, W-column slice): a
// lane sums the slices of the row's neighbours and applies the couplings
// once.  A slice is one 8-, 16- or 32-byte access.
//
// FP32 panels: A x + B sum_hops + C sum_plaq - prev with the scale folded into
// the couplings, these as pairs of FP32 numbers (PairCoef below), and the
// neighbours added pairwise, so that a new entry sees about three roundings
// of its own size (errors: cheb.cu).  The 4x4 quench takes 35.0 ms a run with
// them for K = 8, 27.2 for K = 5 and 54.3 for K = 8 with plaquettes (with FP32
// couplings, one chain of sums and the scale apart 35.2, 26.6 and 51.8); with
// every error carried by TwoSum and TwoProduct 48.0 for K = 8 (and two thirds
// of the state's error).  Where `low` is given, an entry's products and their sum
// carry their errors and what its rounding drops is stored.
#pragma once

#include "lgt_cheb.h"
#include "lgt_dfloat.cuh"
#include "lgt_hpsi_gather.cuh"
#include "lgt_intsum.cuh"

namespace lgt {
namespace rows {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

template <typename T>
struct Args {
  const uint32_t* meta;   // the table (NbrTable)
  const uint32_t* off;
  const uint32_t* nbr;
  int mm;
  int64_t N;
  int K;
  const T* x;
  T* y;
  const T* prev;          // subtracted when not null
  T* low;                 // FP32: the dropped part of y when not null
  const T* coef;          // FP64: [6][K] cE, cm, ch, cp, shift, scale; FP32: PairCoef
};

template <typename T, int W>
__device__ __forceinline__ void ld_cols(const T* p, T (&r)[W]) {
  constexpr int B = W * int(sizeof(T));
  if constexpr (B == 32) {
    gather::ld32(p, r);
  } else if constexpr (B == 16 && sizeof(T) == 4) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    r[0] = v.x, r[1] = v.y, r[2] = v.z, r[3] = v.w;
  } else if constexpr (B == 16) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    r[0] = v.x, r[1] = v.y;
  } else {
    static_assert(B == 8 && sizeof(T) == 4, "slices of 8, 16 or 32 bytes");
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    r[0] = v.x, r[1] = v.y;
  }
}

template <typename T, int W>
__device__ __forceinline__ void st_cols(T* p, const T (&r)[W]) {
  constexpr int B = W * int(sizeof(T));
  if constexpr (B == 32) {
    gather::st32(p, r);
  } else if constexpr (B == 16 && sizeof(T) == 4) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(r[0], r[1], r[2], r[3]));
  } else if constexpr (B == 16) {
    __stcs(reinterpret_cast<double2*>(p), make_double2(r[0], r[1]));
  } else {
    static_assert(B == 8 && sizeof(T) == 4, "slices of 8, 16 or 32 bytes");
    __stcs(reinterpret_cast<float2*>(p), make_float2(r[0], r[1]));
  }
}

// s = the sum of the slices of entries lst[n0 .. n1), eight of them in flight
// and added pairwise (the last trip adds zeros for the entries it lacks); SGN:
// bit 31 of an entry flips the sign.
template <int W, bool SGN>
__device__ __forceinline__ void sum_slices(const float* x, int C, int col0, const uint32_t* lst,
                                           int n0, int n1, float (&s)[W]) {
#pragma unroll
  for (int e = 0; e < W; ++e) s[e] = 0.f;
  for (int n = n0; n < n1; n += 8) {
    float v[8][W];
    uint32_t ent[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (n + u < n1) {
        ent[u] = lst[n + u];
        ld_cols<float, W>(x + size_t(ent[u] & 0x7fffffffu) * C + col0, v[u]);
      } else {
        ent[u] = 0u;
#pragma unroll
        for (int e = 0; e < W; ++e) v[u][e] = 0.f;
      }
    }
    float sg[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) sg[u] = (ent[u] >> 31) ? -1.f : 1.f;
#pragma unroll
    for (int e = 0; e < W; ++e) {
      float t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        t[u] = SGN ? fmaf(sg[2 * u], v[2 * u][e], sg[2 * u + 1] * v[2 * u + 1][e])
                   : v[2 * u][e] + v[2 * u + 1][e];
      s[e] += (t[0] + t[1]) + (t[2] + t[3]);
    }
  }
}

// h + l += (c + d) s
__device__ __forceinline__ void add_prod(float c, float d, float s, float& h, float& l) {
  float p, e, q;
  two_prod(c, s, p, e);
  e = df_fma_rn(d, s, e);
  two_sum(h, p, h, q);
  l = df_add_rn(l, df_add_rn(q, e));
}

template <typename T>
__host__ __device__ constexpr int coef_rows() { return sizeof(T) == 4 ? kPairCoefs : 6; }

template <typename T>
__host__ __device__ inline int smem_bytes(int K, int mm) {
  return (coef_rows<T>() * K * int(sizeof(T)) + 15) / 16 * 16 + 2 * kThreads * 4 +
         kThreads * mm * 4;
}

__device__ __forceinline__ int incl_scan(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += u;
  }
  return v;
}

// The scaled and shifted diagonal of a row: the leading parts are multiples of
// one unit, so their sum is exact (cheb.cu).
__device__ __forceinline__ float diag_hi(const float* c, int K, float e2, float stag) {
  return fmaf(c[kElHi * K], e2, fmaf(c[kMassHi * K], stag, c[kShiftHi * K]));
}
__device__ __forceinline__ float diag_lo(const float* c, int K, float e2, float stag) {
  return fmaf(c[kElLo * K], e2, fmaf(c[kMassLo * K], stag, c[kShiftLo * K]));
}

// U: entries in flight (FP64; FP32 has eight).
template <typename T, int W, int U, bool PLAQ, bool JW>
__global__ void __launch_bounds__(kThreads, PLAQ || JW || W * sizeof(T) != 8 ? 4 : 5)
    k_cheb_product(Args<T> a) {
  static_assert(W % 2 == 0, "a slice holds whole points");
  extern __shared__ __align__(16) unsigned char smem[];
  const int K = a.K, C = 2 * K;
  T* s_coef = reinterpret_cast<T*>(smem);
  uint32_t* s_meta =
      reinterpret_cast<uint32_t*>(smem + (coef_rows<T>() * K * int(sizeof(T)) + 15) / 16 * 16);
  uint32_t* s_off = s_meta + kThreads;
  uint32_t* s_list = s_off + kThreads;
  for (int i = threadIdx.x; i < coef_rows<T>() * K; i += kThreads) s_coef[i] = a.coef[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t row0 = (int64_t(blockIdx.x) * kWarps + wid) * 32;
  if (row0 >= a.N) return;
  const uint32_t m = (row0 + lane < a.N) ? __ldcs(a.meta + row0 + lane) : 0u;
  const int cnt = int(m & 255u);
  const int incl = incl_scan(cnt, lane);
  s_meta[wid * 32 + lane] = m;
  s_off[wid * 32 + lane] = uint32_t(incl - cnt);
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t* src = a.nbr + __ldg(a.off + (row0 >> 5));
  uint32_t* lst = s_list + wid * 32 * a.mm;
  for (int i = lane; i < total; i += 32) lst[i] = __ldcs(src + i);
  __syncwarp();

  const T* __restrict__ x = a.x;
  const int lpr = C / W;
  const int items = 32 * lpr;
  for (int it = lane; it < items; it += 32) {
    const int rl = it / lpr;
    const int64_t row = row0 + rl;
    if (row >= a.N) break;  // rows only grow with it
    const int col0 = (it - rl * lpr) * W;
    const uint32_t mw = s_meta[wid * 32 + rl];
    const int n1 = int(mw & 255u), nh = int((mw >> 8) & 255u);
    const T e2 = T(int((mw >> 16) & 255u)), stag = T(int(mw >> 24) - 128);
    const uint32_t* l = lst + s_off[wid * 32 + rl];
    const size_t at = size_t(row) * C + col0;
    const T* cf = s_coef + (col0 >> 1);  // the slice's points
    T xd[W], out[W];
    ld_cols<T, W>(x + at, xd);
    if constexpr (sizeof(T) == 8) {
      T ah[W];
      auto load = [&](uint32_t j, double(&v)[W]) {
        ld_cols<double, W>(x + size_t(j) * C + col0, v);
      };
      int_sum<W, U, JW>(l, 0, nh, ah, load);
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const int k = e >> 1;
        const T cd = fma(cf[k], e2, fma(cf[K + k], stag, cf[4 * K + k]));
        out[e] = fma(cf[2 * K + k], ah[e], cd * xd[e]);
      }
      if (PLAQ) {
        int_sum<W, U, false>(l, nh, n1, ah, load);
#pragma unroll
        for (int e = 0; e < W; ++e) out[e] = fma(cf[3 * K + (e >> 1)], ah[e], out[e]);
      }
#pragma unroll
      for (int e = 0; e < W; ++e) ah[e] = T(0);
      if (a.prev) ld_cols<T, W>(a.prev + at, ah);
#pragma unroll
      for (int e = 0; e < W; ++e) out[e] = fma(cf[5 * K + (e >> 1)], out[e], -ah[e]);
    } else {
      // T_{n-1} is loaded ahead of the gathers where the 64 registers of four
      // blocks have room (the same quench, K = 8: 35.0 ms against 36.4; at five
      // blocks 39.5; with plaquettes 56.2 against 53.1, so not there)
      constexpr bool kAhead = W == 4 && !PLAQ && !JW;
      T ah[W], ap[W], pv[W];
      auto load_prev = [&] {
#pragma unroll
        for (int e = 0; e < W; ++e) pv[e] = 0.f;
        if (a.prev) ld_cols<T, W>(a.prev + at, pv);
      };
      if (kAhead) load_prev();
      sum_slices<W, JW>(x, C, col0, l, 0, nh, ah);
      if (PLAQ) sum_slices<W, false>(x, C, col0, l, nh, n1, ap);
      if (!kAhead) load_prev();
      if (a.low) {
        T low[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          const float* c = cf + (e >> 1);
          out[e] = -pv[e];
          low[e] = 0.f;
          add_prod(diag_hi(c, K, e2, stag), diag_lo(c, K, e2, stag), xd[e], out[e], low[e]);
          add_prod(c[kHopHi * K], c[kHopLo * K], ah[e], out[e], low[e]);
          if (PLAQ) add_prod(c[kPlaqHi * K], c[kPlaqLo * K], ap[e], out[e], low[e]);
          fast_two_sum(out[e], low[e], out[e], low[e]);
        }
        st_cols<T, W>(a.low + at, low);
      } else {
#pragma unroll
        for (int p = 0; p < W / 2; ++p) {
          const float* c = cf + p;
          const float dh = diag_hi(c, K, e2, stag), dl = diag_lo(c, K, e2, stag);
#pragma unroll
          for (int e = 2 * p; e < 2 * p + 2; ++e) {
            // the small terms first, T_{n-1} last
            float t = fmaf(dl, xd[e], c[kHopLo * K] * ah[e]);
            if (PLAQ) t = fmaf(c[kPlaqHi * K], ap[e], fmaf(c[kPlaqLo * K], ap[e], t));
            t = fmaf(c[kHopHi * K], ah[e], t);
            out[e] = fmaf(dh, xd[e], t) - pv[e];
          }
        }
      }
    }
    st_cols<T, W>(a.y + at, out);
  }
}

template <typename T, int W, int U, bool PLAQ, bool JW>
cudaError_t launch(const Args<T>& a, cudaStream_t s) {
  auto kern = k_cheb_product<T, W, U, PLAQ, JW>;
  const int bytes = smem_bytes<T>(a.K, a.mm);
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kern), bytes);
  if (e != cudaSuccess) return e;
  const int64_t blocks = (a.N + kThreads - 1) / kThreads;
  if (blocks <= 0) return cudaSuccess;
  kern<<<unsigned(blocks), kThreads, bytes, s>>>(a), lgt::note_launch();
  return cudaGetLastError();
}

template <typename T, int W, int U>
cudaError_t launch_model(const Args<T>& a, uint32_t model, cudaStream_t s) {
  const bool plaq = model & kModelPlaq, jw = model & kModelJW;
  if (plaq && jw) return launch<T, W, U, true, true>(a, s);
  if (plaq) return launch<T, W, U, true, false>(a, s);
  if (jw) return launch<T, W, U, false, true>(a, s);
  return launch<T, W, U, false, false>(a, s);
}

template <typename T>
Args<T> args(const NbrTable& t, int64_t N, int K, const T* x, T* y, const T* prev, T* low,
             const T* coef) {
  Args<T> a = {};
  a.meta = t.meta;
  a.off = t.tile_off;
  a.nbr = t.nbr;
  a.mm = t.mm;
  a.N = N;
  a.K = K;
  a.x = x;
  a.y = y;
  a.prev = prev;
  a.low = low;
  a.coef = coef;
  return a;
}

}  // namespace rows
}  // namespace lgt
