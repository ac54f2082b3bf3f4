// Interior cell pairs of the ES kernel phi(z) = exp(beta (sqrt(1 - z^2) - 1)) as polynomials in the
// point's offset (host side; plain C++).
#pragma once

#include <algorithm>
#include <cmath>

namespace mpsq {

constexpr int kPairs = 7;            // interior cell pairs of the widest kernel (w = 16)
constexpr int kEven = 11, kOdd = 10; // coefficients of E and O

struct EsPairs {
  double e[kPairs][kEven];           // pair p: cells p + 1 and w - 2 - p
  double o[kPairs][kOdd];
};

// Chebyshev interpolation of phi on the interior cells, as monomials in v split into even and
// odd ones.  Formed in long double: in double the rounding of the samples near the ends of the
// support and of the interpolation left 2 to 5e-15 of the kernel's peak in the values; this way they
// are good to 2e-16 (sqrt and exp in double, which the polynomials stand for: 0.6 to 3e-15).
inline EsPairs make_pairs(int w, double beta) {
  using R = long double;
  constexpr int P = kEven + kOdd - 1;
  const R pi = 3.14159265358979323846264338327950288L;
  EsPairs out{};
  for (int i = 1; 2 * i < w; ++i) {
    if (i > kPairs) break;
    R f[P + 1], a[P + 1];
    for (int j = 0; j <= P; ++j) {
      const R v = std::cos(pi * (j + R(0.5)) / (P + 1));
      const R z = (v + 1 + 2 * i - w) / w;
      f[j] = std::exp(R(beta) * (std::sqrt(std::max(1 - z * z, R(0))) - 1));
    }
    for (int k = 0; k <= P; ++k) {
      R s = 0;
      for (int j = 0; j <= P; ++j) s += f[j] * std::cos(pi * k * (j + R(0.5)) / (P + 1));
      a[k] = 2 * s / (P + 1);
    }
    a[0] /= 2;
    R t0[P + 1] = {}, t1[P + 1] = {}, m[P + 1] = {};
    t0[0] = 1;
    t1[1] = 1;
    m[0] = a[0];
    m[1] = a[1];
    for (int k = 2; k <= P; ++k) {
      R tk[P + 1] = {};
      for (int q = 0; q <= P; ++q) tk[q] = (q > 0 ? 2 * t1[q - 1] : R(0)) - t0[q];
      for (int q = 0; q <= P; ++q) {
        m[q] += a[k] * tk[q];
        t0[q] = t1[q];
        t1[q] = tk[q];
      }
    }
    const bool middle = 2 * i == w - 1;          // its own mirror: even
    for (int q = 0; q < kEven; ++q) out.e[i - 1][q] = (double)m[2 * q];
    for (int q = 0; q < kOdd; ++q) out.o[i - 1][q] = middle ? 0.0 : (double)m[2 * q + 1];
  }
  return out;
}

}  // namespace mpsq
