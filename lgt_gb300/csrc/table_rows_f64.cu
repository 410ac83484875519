// table_rows_f64.cu -- FP64 instances of the table products of
// lgt_table_rows.cuh.
#include "lgt_cheb.h"
#include "lgt_table_rows.cuh"

namespace lgt {

// Slices of 32 or 16 bytes.
cudaError_t launch_cheb_product(const NbrTable& T, uint32_t model, int64_t N, int K,
                                const double* x, double* y, const double* prev,
                                const double* coef, cudaStream_t s) {
  rows::Args<double> a = {};
  a.meta = T.meta;
  a.off = T.tile_off;
  a.nbr = T.nbr;
  a.mm = T.mm;
  a.N = N;
  a.C = 2 * K;
  a.ncomp = 2;
  a.K = K;
  a.x = x;
  a.y = y;
  a.prev = prev;
  a.coef = coef;
  if (a.C % 4 == 0) return rows::launch_model<double, 4, 2, true>(a, model, s);
  return rows::launch_model<double, 2, 4, true>(a, model, s);
}

}  // namespace lgt
