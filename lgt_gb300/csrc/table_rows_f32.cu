// table_rows_f32.cu -- FP32 instances of the expansion's products
// (lgt_table_rows.cuh).
#include "lgt_table_rows.cuh"

namespace lgt {

// Slices of 16 bytes where they divide the panel row, else of 8.  (32-byte
// ones take half the instructions, but the lanes wait on L2 and have more rows
// in flight with the smaller ones: 4x4 K = 8 quench, FP32-mixed, 35.9 ms a run
// with 32-byte slices, 35.1 with 16, 40.5 with 8, all with one chain of sums.)
cudaError_t launch_cheb_product(const NbrTable& T, uint32_t model, int64_t N, int K, const float* x,
                                float* y, const float* prev, float* low, const float* coef,
                                cudaStream_t s) {
  const rows::Args<float> a = rows::args(T, N, K, x, y, prev, low, coef);
  if (K % 2 == 0) return rows::launch_model<float, 4, 8>(a, model, s);
  return rows::launch_model<float, 2, 8>(a, model, s);
}

}  // namespace lgt
