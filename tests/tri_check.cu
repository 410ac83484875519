// Runs the mixed path's convergence check (lgt_tridiag.cuh) on a batch of
// tridiagonals: one warp a matrix, out = (theta, residual, z_{n-1}).
#include "../lgt_gb300/csrc/lgt_tridiag.cuh"

namespace {
__global__ void k(const double* a, const double* b, int n, double* out) {
  __shared__ double sa[lgt::kTriMax], sb[lgt::kTriMax], sz[lgt::kTriMax];
  __shared__ __align__(16) double work[3 * lgt::kTriMax];
  const int lane = threadIdx.x;
  for (int i = lane; i < n; i += 32) {
    sa[i] = a[size_t(blockIdx.x) * n + i];
    sb[i] = b[size_t(blockIdx.x) * n + i];
  }
  __syncwarp();
  double r = 0.0;
  const double th =
      lgt::warp_check_lowest_f32(sa, sb, n, sb[n - 1], false, 0.0, 0.0, sz, work, &r);
  if (lane == 0) {
    out[3 * blockIdx.x] = th;
    out[3 * blockIdx.x + 1] = r;
    out[3 * blockIdx.x + 2] = sz[n - 1];
  }
}
}  // namespace

// a, b, out: device pointers, `count` matrices of n <= kTriMax rows.
extern "C" int tri_check(const double* a, const double* b, int n, int count, double* out) {
  if (n < 1 || n > lgt::kTriMax || count < 1) return -1;
  k<<<count, 32>>>(a, b, n, out);
  return int(cudaDeviceSynchronize());
}
