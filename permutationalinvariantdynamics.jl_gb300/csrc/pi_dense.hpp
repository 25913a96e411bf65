// Small dense complex linear algebra for the projected Krylov problems (host, FP64):
// the matrix exponential of the (m+1) x (m+1) Hessenberg matrix used by expv
// (krylov_extensions.jl:1412, Julia's LinearAlgebra.exp) and helpers.
#pragma once

#include <cmath>
#include <complex>
#include <vector>

namespace picuda {

using cd = std::complex<double>;

struct CMat {
  int n = 0;
  std::vector<cd> a;  // row-major
  CMat() = default;
  explicit CMat(int n_) : n(n_), a((size_t)n_ * n_, cd(0, 0)) {}
  cd& operator()(int i, int j) { return a[(size_t)i * n + j]; }
  const cd& operator()(int i, int j) const { return a[(size_t)i * n + j]; }
};

// First column of exp(A) by the scaling-and-squaring algorithm with [m/m] Pade approximants of
// N. J. Higham, "The scaling and squaring method for the matrix exponential revisited", SIAM
// J. Matrix Anal. Appl. 26 (2005) 1179-1193, Algorithm 2.3: degrees 3, 5, 7, 9, 13 chosen by
// the 1-norm against the published theta_m bounds.  Not a number in every entry when A is not
// finite (pi_dense.cpp).
std::vector<cd> expm_column(const CMat& A);

// Complex Givens rotation (krylov.jl:710-716).
inline void complex_givens(cd a, cd b, double* c, cd* s) {
  if (b == cd(0, 0)) {
    *c = 1.0;
    *s = cd(0, 0);
    return;
  }
  if (a == cd(0, 0)) {
    *c = 0.0;
    *s = cd(1, 0);
    return;
  }
  const double scale = std::abs(a) + std::abs(b);
  const double normab = scale * std::sqrt(std::norm(a / scale) + std::norm(b / scale));
  const cd alpha = a / std::abs(a);
  *c = std::abs(a) / normab;
  *s = alpha * std::conj(b) / normab;
}

}  // namespace picuda
