// Residuals of libheom_gb300/csrc/eigenbasis.h in long double arithmetic; prints OK.
#include <cstdio>
#include <random>

#include "eigenbasis.h"

using namespace heomgb;
using cd = std::complex<double>;

namespace {

// orthonormal columns to about 1e-8 of a random unitary: a poor start that the refinement has to mend
MatrixC poor(const MatrixC& W, std::mt19937_64& g) {
  std::normal_distribution<double> r;
  MatrixC P = W;
  for (TwofoldC& w : P) w = TwofoldC(cd(w.re.h + 1e-9 * r(g), w.im.h + 1e-9 * r(g)));
  return P;
}

int fail(const char* what, int n, double v) {
  std::printf("%s n=%d %.3g\n", what, n, v);
  return 1;
}

}  // namespace

int main() {
  std::mt19937_64 g(1);
  std::normal_distribution<double> r;
  for (int n : {1, 2, 3, 7, 13}) {
    // W0 by Gram-Schmidt in twofold arithmetic
    MatrixC W0(n * n);
    for (TwofoldC& w : W0) w = TwofoldC(cd(r(g), r(g)));
    for (int pass = 0; pass < 2; ++pass)
      for (int j = 0; j < n; ++j) {
        for (int k = 0; k < j; ++k) {
          TwofoldC dot;
          for (int i = 0; i < n; ++i) dot = dot + conj(W0[i * n + k]) * W0[i * n + j];
          for (int i = 0; i < n; ++i) {
            const TwofoldC t = dot * W0[i * n + k];
            W0[i * n + j] = W0[i * n + j] + TwofoldC(-t.re, -t.im);
          }
        }
        Twofold s;
        for (int i = 0; i < n; ++i) s = s + W0[i * n + j].re * W0[i * n + j].re + W0[i * n + j].im * W0[i * n + j].im;
        const double q = std::sqrt(s.h);
        const Twofold root = Twofold(q) + (s - Twofold(q) * Twofold(q)) / Twofold(2 * q);
        for (int i = 0; i < n; ++i) W0[i * n + j] = {W0[i * n + j].re / root, W0[i * n + j].im / root};
      }
    std::vector<double> ev(n);
    for (int i = 0; i < n; ++i) ev[i] = i + 0.5 * std::sin(3.0 * i) - 2.0;
    MatrixC D(n * n);
    for (int i = 0; i < n; ++i) D[i * n + i].re = Twofold(ev[i]);
    const MatrixC Mf = in_basis(D, dagger(W0, n), n);
    std::vector<cd> M(n * n);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j <= i; ++j) {
        M[i * n + j] = Mf[i * n + j].hi();
        if (i == j) M[i * n + j] = M[i * n + j].real();
        M[j * n + i] = std::conj(M[i * n + j]);
      }
    if (!plain_hermitian(M, n)) return fail("hermitian", n, 0);
    MatrixC W = poor(W0, g);
    std::vector<std::vector<cd>> vd;
    if (!common_eigenbasis({M}, M, n, W, vd)) return fail("basis", n, 0);
    // residuals
    const MatrixC I = product(dagger(W, n), W, n), A = in_basis(twofold(M), W, n);
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j) {
        const TwofoldC x = I[i * n + j];
        const Twofold d = x.re - Twofold(i == j ? 1.0 : 0.0);
        if (std::abs(d.h) + std::abs(x.im.h) > 1e-28) return fail("orthonormal", n, d.h);
        if (i != j && std::abs(A[i * n + j].hi()) > 1e-27) return fail("diagonal", n, std::abs(A[i * n + j].hi()));
      }
    for (int i = 0; i < n; ++i)
      if (std::abs(vd[0][i].real() - ev[i]) > 1e-14) return fail("eigenvalue", n, vd[0][i].real() - ev[i]);
    if (n == 1) continue;
    std::vector<cd> N = M;  // not commuting; not Hermitian; not finite
    N[1] += 1e-9;
    N[n] += 1e-9;
    MatrixC X = W;
    if (common_eigenbasis({M, N}, M, n, X, vd)) return fail("not commuting", n, 0);
    N[n] = std::conj(N[1]) + 1e-16;
    if (plain_hermitian(N, n)) return fail("not hermitian", n, 0);
    N[1] = N[n] = std::nan("");
    if (plain_hermitian(N, n)) return fail("nan", n, 0);
  }
  if (plain_hermitian(std::vector<cd>(4), 2)) return fail("zero", 2, 0);
  std::printf("OK\n");
  return 0;
}
