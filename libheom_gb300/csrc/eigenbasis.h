// A common eigenbasis of commuting Hermitian matrices to twice the FP64
// precision (host code): the basis and what is formed in it carry one FP64
// rounding where they are used, not the eigensolver's.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace heomgb {

// An unevaluated sum h + l, |l| <= ulp(h) / 2 (Dekker, Numer. Math. 18, 1971).
struct Twofold {
  double h = 0.0, l = 0.0;
  Twofold() = default;
  Twofold(double x) : h(x) {}  // NOLINT: a double is one
  Twofold(double a, double b) : h(a), l(b) {}
};
inline Twofold two_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
inline Twofold quick_sum(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return {s, b - (s - a)};
}
inline Twofold operator+(Twofold a, Twofold b) {
  Twofold s = two_sum(a.h, b.h), t = two_sum(a.l, b.l);
  s = quick_sum(s.h, s.l + t.h);
  return quick_sum(s.h, s.l + t.l);
}
inline Twofold operator-(Twofold a) { return {-a.h, -a.l}; }
inline Twofold operator-(Twofold a, Twofold b) { return a + -b; }
inline Twofold operator*(Twofold a, Twofold b) {
  const double p = a.h * b.h, e = std::fma(a.h, b.h, -p);
  return quick_sum(p, e + (a.h * b.l + a.l * b.h));
}
inline Twofold operator/(Twofold a, Twofold b) {
  const double q = a.h / b.h;
  const Twofold r = a - b * Twofold(q);
  return quick_sum(q, r.h / b.h);
}

struct TwofoldC {
  Twofold re, im;
  TwofoldC() = default;
  TwofoldC(std::complex<double> z) : re(z.real()), im(z.imag()) {}  // NOLINT
  TwofoldC(Twofold a, Twofold b) : re(a), im(b) {}
  std::complex<double> hi() const { return {re.h, im.h}; }
  std::complex<double> lo() const { return {re.l, im.l}; }
};
inline TwofoldC operator+(TwofoldC a, TwofoldC b) { return {a.re + b.re, a.im + b.im}; }
inline TwofoldC operator*(TwofoldC a, TwofoldC b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
inline TwofoldC conj(TwofoldC a) { return {a.re, -a.im}; }

using MatrixC = std::vector<TwofoldC>;
inline MatrixC twofold(const std::vector<std::complex<double>>& A) { return MatrixC(A.begin(), A.end()); }
// A B and W^dagger A W (n x n, row-major)
inline MatrixC product(const MatrixC& A, const MatrixC& B, int n) {
  MatrixC C(A.size());
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < n; ++k)
      for (int j = 0; j < n; ++j) C[i * n + j] = C[i * n + j] + A[i * n + k] * B[k * n + j];
  return C;
}
inline MatrixC dagger(const MatrixC& A, int n) {
  MatrixC C(A.size());
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) C[j * n + i] = conj(A[i * n + j]);
  return C;
}
inline MatrixC in_basis(const MatrixC& A, const MatrixC& W, int n) {
  return product(dagger(W, n), product(A, W, n), n);
}

// The eigenvectors W of a Hermitian M, known to about FP64 precision, refined
// in place (three steps of Ogita and Aishima, Japan J. Indust. Appl. Math. 35,
// 2018; each doubles the digits).  Columns whose eigenvalues agree to rounding
// are only made orthonormal.
inline void refine_eigenvectors(const MatrixC& M, int n, MatrixC& W) {
  for (int step = 0; step < 3; ++step) {
    MatrixC R = product(dagger(W, n), W, n);
    const MatrixC S = in_basis(M, W, n);
    double top = 0.0;
    for (int i = 0; i < n; ++i) top = std::max(top, std::abs(S[i * n + i].re.h));
    for (TwofoldC& r : R) r = {-r.re, -r.im};
    for (int i = 0; i < n; ++i) R[i * n + i].re = R[i * n + i].re + Twofold(1.0);  // I - W^dagger W
    std::vector<Twofold> lam(n);
    for (int i = 0; i < n; ++i) lam[i] = S[i * n + i].re / (Twofold(1.0) - R[i * n + i].re);
    MatrixC E(W.size());
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) {
        const TwofoldC r = R[i * n + j], s = S[i * n + j];
        const Twofold gap = lam[j] - lam[i];
        if (i != j && std::abs(gap.h) > 1e-12 * top)
          E[i * n + j] = {(s.re + lam[j] * r.re) / gap, (s.im + lam[j] * r.im) / gap};
        else
          E[i * n + j] = {r.re * Twofold(0.5), r.im * Twofold(0.5)};
      }
    const MatrixC D = product(W, E, n);
    for (size_t i = 0; i < W.size(); ++i) W[i] = W[i] + D[i];
  }
}

// Whether every V is Hermitian as it stands and `W` (about the eigenvectors of a
// combination `M` of them) can be refined to a basis in which all of them are
// diagonal to the rounding of their largest entry; then vd holds the
// diagonals.  Eigenvalues that agree to that rounding are made equal, so that no
// term hangs on their difference.
inline bool common_eigenbasis(const std::vector<std::vector<std::complex<double>>>& V,
                              const std::vector<std::complex<double>>& M, int n, MatrixC& W,
                              std::vector<std::vector<std::complex<double>>>& vd) {
  const double half_ulp = 0x1p-53;
  refine_eigenvectors(twofold(M), n, W);
  vd.assign(V.size(), std::vector<std::complex<double>>(n));
  for (size_t u = 0; u < V.size(); ++u) {
    double top = 0.0;
    for (const std::complex<double>& v : V[u]) top = std::max(top, std::abs(v));
    const MatrixC D = in_basis(twofold(V[u]), W, n);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        if (i != j && !(std::abs(D[i * n + j].hi()) <= half_ulp * top)) return false;
    for (int i = 0; i < n; ++i) {
      double v = D[i * n + i].re.h;
      if (!(std::abs(v) > 2 * half_ulp * top)) v = 0.0;
      for (int j = 0; j < i; ++j)
        if (std::abs(v - vd[u][j].real()) <= 2 * half_ulp * top) v = vd[u][j].real();
      vd[u][i] = v;
    }
  }
  return true;
}

// Finite, Hermitian entry by entry, not zero.
inline bool plain_hermitian(const std::vector<std::complex<double>>& V, int n) {
  bool any = false;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const std::complex<double> v = V[i * n + j];
      if (!std::isfinite(v.real()) || !std::isfinite(v.imag()) || v != std::conj(V[j * n + i])) return false;
      any = any || v != 0.0;
    }
  return any;
}

}  // namespace heomgb
