// lgt_cheb.h -- exp(-iHt) steps by Chebyshev expansion (cheb.cu).
#pragma once

#include <string>
#include <vector>

#include "lgt_krylov.h"

namespace lgt {

// Device workspace of the expansion in one storage precision, kept with the
// Hamiltonian (pool memory, stream-ordered).
struct ChebWork {
  void* V = nullptr;      // polynomial panels T_0 .. T_{terms-1}
  size_t v_bytes = 0;
  void* aux = nullptr;    // bounds, coefficients, norms, partial sums
  size_t aux_bytes = 0;
  void release(cudaStream_t s);
};

// psi <- exp(-i H dt) psi, n_steps times with renormalisation after each, on
// the complex panel X (as krylov_expm).  Runs when the table of `op` is
// built, dt > 0, the expansion needs at most p.krylovdim products a step and
// its panels can be allocated; otherwise *done stays false and nothing was
// changed.
std::string cheb_expm(const OpDev& op, const KrylovParams& p, ChebWork* w, double dt, int n_steps,
                      double* X, double* drift, StepObserver* obs, cudaStream_t s,
                      KrylovReport* rep, bool* done);

// Expansion coefficients J_0(z) .. J_n(z) with the shortest n whose tail
// 2 sum_{m > n} |J_m(z)| is below eps; empty when n would pass nmax.
std::vector<double> cheb_bessel(double z, double eps, int nmax);

// Rows of the FP32 products' coefficients: the couplings times the scale, each
// as a leading and a trailing FP32 number (cheb.cu).
enum PairCoef : int {
  kElHi, kElLo, kMassHi, kMassLo, kShiftHi, kShiftLo, kHopHi, kHopLo, kPlaqHi, kPlaqLo,
  kPairCoefs
};

// The products of the expansion from the stored table (one translation unit
// per precision): y = scale (H + shift) x (- prev).  FP64: coef = [6][K].
// FP32: coef = [kPairCoefs][K]; the part of y that its rounding drops goes to
// `low` when that is given.
cudaError_t launch_cheb_product(const NbrTable& T, uint32_t model, int64_t N, int K, const float* x,
                                float* y, const float* prev, float* low, const float* coef,
                                cudaStream_t s);
cudaError_t launch_cheb_product(const NbrTable& T, uint32_t model, int64_t N, int K,
                                const double* x, double* y, const double* prev,
                                const double* coef, cudaStream_t s);

}  // namespace lgt
