// First column of the exponential of a small dense complex matrix (see pi_dense.hpp).
//
// Matrices are kept as split real and imaginary arrays with padded rows: products through
// std::complex go through the checked complex multiply (a test per product, no vector code) and
// took most of a mixed-precision interval.  Only the first column of the exponential is used
// by the callers, so the scaled approximant r(A / 2^s) = D^-1 N is applied 2^s times to e_1 through one
// LU factorisation of D instead of being formed (a solve with n right-hand sides) and squared s
// times.  31 x 31, 1-norms of 4 to 40, on one Grace core: 130-200 -> 65-85 us.
#pragma GCC optimize("O3")

#include "pi_dense.hpp"

#include <algorithm>
#include <cmath>
#include <limits>
#include <stdexcept>

namespace picuda {
namespace {

typedef double v2 __attribute__((vector_size(16)));

constexpr int kBlk = 8;  // columns per register block

struct Split {
  int n, ld;
  std::vector<double> re, im;
  explicit Split(int n_) : n(n_), ld((n_ + kBlk - 1) / kBlk * kBlk), re((size_t)n_ * ld), im((size_t)n_ * ld) {}
};

inline v2 load(const double* p) { return v2{p[0], p[1]}; }
inline void store(double* p, v2 v) {
  p[0] = v[0];
  p[1] = v[1];
}

// R rows of c = x y, eight columns at a time with the sums in registers.
template <int R>
void rows(const Split& x, const Split& y, Split& c, int i0) {
  const int n = x.n, ld = x.ld;
  for (int j0 = 0; j0 < n; j0 += kBlk) {
    v2 cr[R][4], ci[R][4];
    for (int r = 0; r < R; ++r)
      for (int q = 0; q < 4; ++q) cr[r][q] = ci[r][q] = v2{0, 0};
    for (int k = 0; k < n; ++k) {
      const double* yr = y.re.data() + (size_t)k * ld + j0;
      const double* yi = y.im.data() + (size_t)k * ld + j0;
      v2 br[4], bi[4];
      for (int q = 0; q < 4; ++q) br[q] = load(yr + 2 * q), bi[q] = load(yi + 2 * q);
      for (int r = 0; r < R; ++r) {
        const double a = x.re[(size_t)(i0 + r) * ld + k], b = x.im[(size_t)(i0 + r) * ld + k];
        const v2 av = {a, a}, bv = {b, b};
        for (int q = 0; q < 4; ++q) {
          cr[r][q] += av * br[q];
          cr[r][q] -= bv * bi[q];
          ci[r][q] += av * bi[q];
          ci[r][q] += bv * br[q];
        }
      }
    }
    for (int r = 0; r < R; ++r)
      for (int q = 0; q < 4; ++q) {
        store(c.re.data() + (size_t)(i0 + r) * ld + j0 + 2 * q, cr[r][q]);
        store(c.im.data() + (size_t)(i0 + r) * ld + j0 + 2 * q, ci[r][q]);
      }
  }
}

Split matmul(const Split& x, const Split& y) {
  Split c(x.n);
  int i = 0;
  for (; i + 2 <= x.n; i += 2) rows<2>(x, y, c, i);
  if (i < x.n) rows<1>(x, y, c, i);
  return c;
}

// a x + b y + c z
Split combine(double a, const Split& x, double b, const Split& y, double c, const Split& z) {
  Split r(x.n);
  for (size_t i = 0; i < r.re.size(); ++i) {
    r.re[i] = a * x.re[i] + b * y.re[i] + c * z.re[i];
    r.im[i] = a * x.im[i] + b * y.im[i] + c * z.im[i];
  }
  return r;
}
void add(Split& r, double a, const Split& x) {
  for (size_t i = 0; i < r.re.size(); ++i) {
    r.re[i] += a * x.re[i];
    r.im[i] += a * x.im[i];
  }
}
void add_identity(Split& r, double a) {
  for (int i = 0; i < r.n; ++i) r.re[(size_t)i * r.ld + i] += a;
}

// Numerator and denominator V + U, V - U of the degree-m approximant.
void pade(const Split& A, int m, Split& U, Split& V) {
  std::vector<double> b(m + 1);
  // b_j = (2m-j)! m! / ((2m)! j! (m-j)!) evaluated as a running product
  b[0] = 1.0;
  for (int j = 1; j <= m; ++j) b[j] = b[j - 1] * (double)(m - j + 1) / ((double)j * (double)(2 * m - j + 1));
  const Split A2 = matmul(A, A);
  if (m == 13) {
    const Split A4 = matmul(A2, A2), A6 = matmul(A4, A2);
    U = matmul(A6, combine(b[13], A6, b[11], A4, b[9], A2));
    V = matmul(A6, combine(b[12], A6, b[10], A4, b[8], A2));
    add(U, 1.0, combine(b[7], A6, b[5], A4, b[3], A2));
    add(V, 1.0, combine(b[6], A6, b[4], A4, b[2], A2));
  } else {
    std::fill(U.re.begin(), U.re.end(), 0.0);
    std::fill(U.im.begin(), U.im.end(), 0.0);
    V = U;
    Split P = A2;
    for (int k = 2; k <= m; k += 2) {
      if (k > 2) P = matmul(P, A2);
      add(U, b[k + 1], P);
      add(V, b[k], P);
    }
  }
  add_identity(U, b[1]);
  add_identity(V, b[0]);
  U = matmul(A, U);
}

// LU factors of D by partial pivoting, in place; perm[k]: the row exchanged with k.
void factorize(Split& D, std::vector<int>& perm) {
  const int n = D.n, ld = D.ld;
  perm.resize(n);
  for (int k = 0; k < n; ++k) {
    int piv = k;
    double best = -1.0;
    for (int i = k; i < n; ++i) {
      const double a = D.re[(size_t)i * ld + k], b = D.im[(size_t)i * ld + k], v = a * a + b * b;
      if (v > best) best = v, piv = i;
    }
    if (best == 0.0) throw std::runtime_error("singular Pade denominator");
    perm[k] = piv;
    double* pr = D.re.data() + (size_t)k * ld;
    double* pi = D.im.data() + (size_t)k * ld;
    if (piv != k) {
      std::swap_ranges(pr, pr + n, D.re.data() + (size_t)piv * ld);
      std::swap_ranges(pi, pi + n, D.im.data() + (size_t)piv * ld);
    }
    const double den = pr[k] * pr[k] + pi[k] * pi[k], ir = pr[k] / den, ii = -pi[k] / den;
    for (int i = k + 1; i < n; ++i) {
      double* qr = D.re.data() + (size_t)i * ld;
      double* qi = D.im.data() + (size_t)i * ld;
      const double fr = qr[k] * ir - qi[k] * ii, fi = qr[k] * ii + qi[k] * ir;
      qr[k] = fr;
      qi[k] = fi;
      for (int j = k + 1; j < n; ++j) {
        qr[j] -= fr * pr[j] - fi * pi[j];
        qi[j] -= fr * pi[j] + fi * pr[j];
      }
    }
  }
}

using Vec = std::vector<double>;

void matvec(const Split& M, const Vec& xr, const Vec& xi, Vec& yr, Vec& yi) {
  for (int i = 0; i < M.n; ++i) {
    const double* mr = M.re.data() + (size_t)i * M.ld;
    const double* mi = M.im.data() + (size_t)i * M.ld;
    double sr = 0, si = 0;
    for (int j = 0; j < M.n; ++j) {
      sr += mr[j] * xr[j] - mi[j] * xi[j];
      si += mr[j] * xi[j] + mi[j] * xr[j];
    }
    yr[i] = sr;
    yi[i] = si;
  }
}

void solve(const Split& LU, const std::vector<int>& perm, Vec& xr, Vec& xi) {
  const int n = LU.n, ld = LU.ld;
  for (int k = 0; k < n; ++k)
    if (perm[k] != k) std::swap(xr[k], xr[perm[k]]), std::swap(xi[k], xi[perm[k]]);
  for (int i = 1; i < n; ++i) {
    const double* lr = LU.re.data() + (size_t)i * ld;
    const double* li = LU.im.data() + (size_t)i * ld;
    double sr = xr[i], si = xi[i];
    for (int j = 0; j < i; ++j) {
      sr -= lr[j] * xr[j] - li[j] * xi[j];
      si -= lr[j] * xi[j] + li[j] * xr[j];
    }
    xr[i] = sr;
    xi[i] = si;
  }
  for (int i = n - 1; i >= 0; --i) {
    const double* ur = LU.re.data() + (size_t)i * ld;
    const double* ui = LU.im.data() + (size_t)i * ld;
    double sr = xr[i], si = xi[i];
    for (int j = i + 1; j < n; ++j) {
      sr -= ur[j] * xr[j] - ui[j] * xi[j];
      si -= ur[j] * xi[j] + ui[j] * xr[j];
    }
    const double den = ur[i] * ur[i] + ui[i] * ui[i];
    xr[i] = (sr * ur[i] + si * ui[i]) / den;
    xi[i] = (si * ur[i] - sr * ui[i]) / den;
  }
}

}  // namespace

std::vector<cd> expm_column(const CMat& A0) {
  const int n = A0.n;
  static const double theta[5] = {1.495585217958292e-2, 2.539398330063230e-1, 9.504178996162932e-1,
                                  2.097847961257068e0, 5.371920351148152e0};
  static const int degrees[5] = {3, 5, 7, 9, 13};
  double nrm = 0.0;
  for (int j = 0; j < n; ++j) {
    double sum = 0.0;
    for (int i = 0; i < n; ++i) sum += std::abs(A0(i, j));
    if (!(sum <= nrm)) nrm = sum;  // keeps a NaN
  }
  std::vector<cd> col(n);
  if (!std::isfinite(nrm)) {  // no exponential: the callers reject a column that is not finite
    const double nan = std::numeric_limits<double>::quiet_NaN();
    std::fill(col.begin(), col.end(), cd(nan, nan));
    return col;
  }
  int d = 0;
  while (d < 4 && nrm > theta[d]) ++d;
  int s = 0;
  if (nrm > theta[4]) s = std::max(0, (int)std::ceil(std::log2(nrm / theta[4])));
  const double scale = std::ldexp(1.0, -s);
  Split A(n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      A.re[(size_t)i * A.ld + j] = A0(i, j).real() * scale;
      A.im[(size_t)i * A.ld + j] = A0(i, j).imag() * scale;
    }
  Split U(n), V(n);
  pade(A, degrees[d], U, V);
  Split N = V, D = V;
  add(N, 1.0, U);
  add(D, -1.0, U);
  std::vector<int> perm;
  factorize(D, perm);
  Vec xr(n, 0.0), xi(n, 0.0), yr(n), yi(n);
  // Beyond 2^6 applications the approximant is formed and squared down to 2^4 of them.
  if (s > 6) {
    Split X(n);
    for (int j = 0; j < n; ++j) {
      for (int i = 0; i < n; ++i) xr[i] = N.re[(size_t)i * N.ld + j], xi[i] = N.im[(size_t)i * N.ld + j];
      solve(D, perm, xr, xi);
      for (int i = 0; i < n; ++i) X.re[(size_t)i * X.ld + j] = xr[i], X.im[(size_t)i * X.ld + j] = xi[i];
    }
    for (; s > 4; --s) X = matmul(X, X);
    std::fill(xr.begin(), xr.end(), 0.0);
    std::fill(xi.begin(), xi.end(), 0.0);
    xr[0] = 1.0;
    for (int k = 0; k < 1 << s; ++k) {
      matvec(X, xr, xi, yr, yi);
      xr.swap(yr);
      xi.swap(yi);
    }
  } else {
    xr[0] = 1.0;
    for (int k = 0; k < 1 << s; ++k) {
      matvec(N, xr, xi, yr, yi);
      solve(D, perm, yr, yi);
      xr.swap(yr);
      xi.swap(yi);
    }
  }
  for (int i = 0; i < n; ++i) col[i] = cd(xr[i], xi[i]);
  return col;
}

}  // namespace picuda
