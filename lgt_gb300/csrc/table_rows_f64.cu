// table_rows_f64.cu -- FP64 instances of the expansion's products
// (lgt_table_rows.cuh).
#include "lgt_table_rows.cuh"

namespace lgt {

// Slices of 32 or 16 bytes.
cudaError_t launch_cheb_product(const NbrTable& T, uint32_t model, int64_t N, int K,
                                const double* x, double* y, const double* prev,
                                const double* coef, cudaStream_t s) {
  const rows::Args<double> a = rows::args<double>(T, N, K, x, y, prev, nullptr, coef);
  if (K % 2 == 0) return rows::launch_model<double, 4, 2>(a, model, s);
  return rows::launch_model<double, 2, 4>(a, model, s);
}

}  // namespace lgt
