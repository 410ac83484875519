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
#pragma once

#include "lgt_cheb.h"
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
  const T* coef;          // [6][K] cE, cm, ch, cp, shift, scale
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

template <typename T>
__host__ __device__ inline int smem_bytes(int K, int mm) {
  return (6 * K * int(sizeof(T)) + 15) / 16 * 16 + 2 * kThreads * 4 + kThreads * mm * 4;
}

__device__ __forceinline__ int incl_scan(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += u;
  }
  return v;
}

template <typename T, int W, int U, bool PLAQ, bool JW>
__global__ void __launch_bounds__(kThreads, PLAQ || JW || sizeof(T) == 8 ? 4 : 5)
    k_cheb_product(Args<T> a) {
  static_assert(W % 2 == 0, "a slice holds whole points");
  extern __shared__ __align__(16) unsigned char smem[];
  const int K = a.K, C = 2 * K;
  T* s_coef = reinterpret_cast<T*>(smem);
  uint32_t* s_meta =
      reinterpret_cast<uint32_t*>(smem + (6 * K * int(sizeof(T)) + 15) / 16 * 16);
  uint32_t* s_off = s_meta + kThreads;
  uint32_t* s_list = s_off + kThreads;
  for (int i = threadIdx.x; i < 6 * K; i += kThreads) s_coef[i] = a.coef[i];
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
    T xd[W], ah[W], out[W];
    ld_cols<T, W>(x + at, xd);
    sum_entries<T, W, U, JW>(x, C, col0, l, 0, nh, ah);
#pragma unroll
    for (int e = 0; e < W; ++e) {
      const int k = e >> 1;
      const T cd = fma(cf[k], e2, fma(cf[K + k], stag, cf[4 * K + k]));
      out[e] = fma(cf[2 * K + k], ah[e], cd * xd[e]);
    }
    if (PLAQ) {
      sum_entries<T, W, U, false>(x, C, col0, l, nh, n1, ah);
#pragma unroll
      for (int e = 0; e < W; ++e) out[e] = fma(cf[3 * K + (e >> 1)], ah[e], out[e]);
    }
#pragma unroll
    for (int e = 0; e < W; ++e) ah[e] = T(0);
    if (a.prev) ld_cols<T, W>(a.prev + at, ah);
#pragma unroll
    for (int e = 0; e < W; ++e) out[e] = fma(cf[5 * K + (e >> 1)], out[e], -ah[e]);
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
Args<T> args(const NbrTable& t, int64_t N, int K, const T* x, T* y, const T* prev,
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
  a.coef = coef;
  return a;
}

}  // namespace rows
}  // namespace lgt
