// lgt_lanczos_grid.h -- a Lanczos cycle of the panel solver in one launch
// (lanczos_grid.cu).
#pragma once

#include "lgt_hpsi.h"

namespace lgt {

template <typename S>
struct GridArgs {
  const uint32_t* meta;   // the stored neighbour table
  const uint32_t* off;
  const uint32_t* nbr;
  int mm;
  int64_t N;
  int C;                  // real columns, one per coupling point
  int rpb, nblk;          // rows per block (a multiple of 32), blocks
  int m, reorth, check_every;
  double tol, tiny_rel;
  const S *cE, *cm, *ch, *cp;  // [C]
  S* V;                   // m + 1 panels; panel 0 holds the start vectors
  size_t vstride;
  double *alpha, *beta;   // [C][ldT]
  int ldT;
  int *status, *len;      // [C]
  double *theta, *resid, *coef;
  double* part;           // [m + 1][C][nblk] dot partials
  double* h;              // [m + 1][C]
  double* npart;          // [C][nblk]
  unsigned* bar;          // zero at launch
  int* steps;             // steps taken; untouched where a wait ran out
  long long spin;         // SM cycles that a barrier waits at the most
  int list_smem;          // the blocks' neighbour lists sit in shared memory
};

// Rows per block, blocks and bytes of dynamic shared memory for N rows of C
// columns; false where a block's rows do not fit.
template <typename S>
bool lanczos_grid_plan(int64_t N, int C, int m, int mm, int* rpb, int* nblk, int* list_smem,
                       int* bytes);

// Runs the cycle (cooperative launch; all blocks resident).
template <typename S>
cudaError_t launch_lanczos_grid(const GridArgs<S>& a, int bytes, cudaStream_t s);

}  // namespace lgt
