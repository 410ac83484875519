// lgt_table_rows.cuh -- row-pull products from the stored neighbour table
// for any panel width, with an optional three-term epilogue.
//
// A warp copies the meta words and entries of its 32 rows into shared memory
// (coalesced, evict-first) and runs its lanes over (row, W-column slice): a
// lane sums the slices of the row's neighbours and applies the couplings
// once.  W columns of T are one 4-, 8-, 16- or 32-byte access, so every
// width divides into slices (W = 1 where C is odd).
//
//   plain  y = (cE e2 + cm stag) x + ch sum_hops (+-) x_j + cp sum_plaq x_j
//   Cheb   y = scale ((H + shift) x), minus `prev` where it is given:
//          T_{n+1} = 2 H~ T_n - T_{n-1}  (cheb.cu)
// (finite_ed.jl:265-318; matter_gauge_entanglement_pjw.jl:82-147).
#pragma once

#include "lgt_hpsi.h"
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
  int C, ncomp, K;
  const T* x;
  T* y;
  const T* prev;          // Cheb: subtracted when not null
  const T* coef;          // Cheb: [6][K] cE, cm, ch, cp, shift, scale
  const T* cE;            // plain: the four coupling arrays
  const T* cm;
  const T* ch;
  const T* cp;
  const int* xsel;        // x + *xsel * xstride when not null
  size_t xstride;
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
  } else if constexpr (B == 8 && sizeof(T) == 4) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    r[0] = v.x, r[1] = v.y;
  } else {
    r[0] = __ldg(p);
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
  } else if constexpr (B == 8 && sizeof(T) == 4) {
    __stcs(reinterpret_cast<float2*>(p), make_float2(r[0], r[1]));
  } else {
    __stcs(p, r[0]);
  }
}

// s = the sum of the slices of entries lst[n0 .. n1), U of them in flight (the
// last trip adds zeros for the entries it lacks); SGN: bit 31 of an entry
// flips the sign.
template <typename T, int W, int U, bool SGN>
__device__ __forceinline__ void sum_slices(const T* x, int C, int col0, const uint32_t* lst,
                                           int n0, int n1, T (&s)[W]) {
#pragma unroll
  for (int e = 0; e < W; ++e) s[e] = T(0);
  for (int n = n0; n < n1; n += U) {
    T v[U][W];
    uint32_t ent[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (n + u < n1) {
        ent[u] = lst[n + u];
        ld_cols<T, W>(x + size_t(ent[u] & 0x7fffffffu) * C + col0, v[u]);
      } else {
        ent[u] = 0u;
#pragma unroll
        for (int e = 0; e < W; ++e) v[u][e] = T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int e = 0; e < W; ++e)
        s[e] = SGN ? fma((ent[u] >> 31) ? T(-1) : T(1), v[u][e], s[e]) : s[e] + v[u][e];
  }
}

// A row's sum over entries lst[n0 .. n1) in T: FP64 by integers.
template <typename T, int W, int U, bool SGN>
__device__ __forceinline__ void sum_entries(const T* x, int C, int col0, const uint32_t* lst,
                                            int n0, int n1, T (&s)[W]) {
  if constexpr (sizeof(T) == 8)
    int_sum<W, U, SGN>(lst, n0, n1, s, [&](uint32_t j, double(&v)[W]) {
      ld_cols<double, W>(x + size_t(j) * C + col0, v);
    });
  else
    sum_slices<T, W, U, SGN>(x, C, col0, lst, n0, n1, s);
}

__host__ __device__ inline int coef_words(bool cheb, int K) { return (cheb ? 6 : 4) * K; }

template <typename T>
__host__ __device__ inline int smem_bytes(bool cheb, int K, int mm) {
  return (coef_words(cheb, K) * int(sizeof(T)) + 15) / 16 * 16 + 2 * kThreads * 4 +
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

template <typename T, int W, int U, bool PLAQ, bool JW, bool CHEB>
__global__ void __launch_bounds__(kThreads, PLAQ || JW || sizeof(T) == 8 ? 4 : 5)
    k_table_rows(Args<T> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int K = a.K, C = a.C;
  T* s_coef = reinterpret_cast<T*>(smem);
  uint32_t* s_meta =
      reinterpret_cast<uint32_t*>(smem + (coef_words(CHEB, K) * int(sizeof(T)) + 15) / 16 * 16);
  uint32_t* s_off = s_meta + kThreads;
  uint32_t* s_list = s_off + kThreads;
  if constexpr (CHEB) {
    for (int i = threadIdx.x; i < 6 * K; i += kThreads) s_coef[i] = a.coef[i];
  } else {
    for (int i = threadIdx.x; i < K; i += kThreads) {
      s_coef[i] = a.cE[i];
      s_coef[K + i] = a.cm[i];
      s_coef[2 * K + i] = a.ch[i];
      s_coef[3 * K + i] = a.cp[i];
    }
  }
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

  const T* __restrict__ x = a.xsel ? a.x + size_t(*a.xsel) * a.xstride : a.x;
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
    T xd[W], ah[W], out[W];
    ld_cols<T, W>(x + at, xd);
    sum_entries<T, W, U, JW>(x, C, col0, l, 0, nh, ah);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const int k = a.ncomp == 2 ? (col0 + e) >> 1 : col0 + e;
      const T cd = CHEB ? fma(s_coef[k], e2, fma(s_coef[K + k], stag, s_coef[4 * K + k]))
                        : fma(s_coef[k], e2, s_coef[K + k] * stag);
      out[e] = fma(s_coef[2 * K + k], ah[e], cd * xd[e]);
    }
    if (PLAQ) {
      sum_entries<T, W, U, false>(x, C, col0, l, nh, n1, ah);
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const int k = a.ncomp == 2 ? (col0 + e) >> 1 : col0 + e;
        out[e] = fma(s_coef[3 * K + k], ah[e], out[e]);
      }
    }
    if (CHEB) {
#pragma unroll
      for (int e = 0; e < W; ++e) ah[e] = T(0);
      if (a.prev) ld_cols<T, W>(a.prev + at, ah);
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const int k = a.ncomp == 2 ? (col0 + e) >> 1 : col0 + e;
        out[e] = fma(s_coef[5 * K + k], out[e], -ah[e]);
      }
    }
    st_cols<T, W>(a.y + at, out);
  }
}

template <typename T, int W, int U, bool PLAQ, bool JW, bool CHEB>
cudaError_t launch(const Args<T>& a, cudaStream_t s) {
  auto kern = k_table_rows<T, W, U, PLAQ, JW, CHEB>;
  const int bytes = smem_bytes<T>(CHEB, a.K, a.mm);
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(kern), bytes);
  if (e != cudaSuccess) return e;
  const int64_t blocks = (a.N + kThreads - 1) / kThreads;
  if (blocks <= 0) return cudaSuccess;
  kern<<<unsigned(blocks), kThreads, bytes, s>>>(a), lgt::note_launch();
  return cudaGetLastError();
}

template <typename T, int W, int U, bool CHEB>
cudaError_t launch_model(const Args<T>& a, uint32_t model, cudaStream_t s) {
  const bool plaq = model & kModelPlaq, jw = model & kModelJW;
  if (plaq && jw) return launch<T, W, U, true, true, CHEB>(a, s);
  if (plaq) return launch<T, W, U, true, false, CHEB>(a, s);
  if (jw) return launch<T, W, U, false, true, CHEB>(a, s);
  return launch<T, W, U, false, false, CHEB>(a, s);
}

}  // namespace rows
}  // namespace lgt
