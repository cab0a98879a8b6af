// tridiagonal.hpp — lowest eigenpairs of the Lanczos matrix T (diagonal
// a[0..n), off-diagonal b[0..n-1)), on the host, every few steps.
//
// The work is serial chains of FP64 divisions, which a GB300 SM issues at
// 1.75 lanes per clock: the one-warp kernel that did it on the device took
// 130 us per solve at order 50 and one pair, and 2.6 ms at order 112 and four
// pairs (33 us and 640 us per Lanczos step). The host takes a few and about
// 200 us, and the next steps run on the device meanwhile.
//
// The sign of a Ritz vector comes out of the last inverse iteration, whose
// shift is within rounding of the eigenvalue, so it depends on every rounding
// before it. All products that are added to something are therefore fused
// explicitly, as the device compiler fuses them, and nothing is left to the
// host compiler: the same T gives the same vectors, bit for bit, on every
// host and as the device kernel gave them.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace sed {

class Tridiagonal {
 public:
  std::vector<double> theta, est;  // eigenvalues and residual estimates b[n - 1] |s[n - 1]|

  explicit Tridiagonal(uint32_t nev) : theta(nev, 0.0), est(nev, 0.0), nev_(nev), s_(nev) {}
  void restart() { size_ = 0; }
  uint32_t size() const { return size_; }
  std::vector<double> const& vector(uint32_t j) const { return s_[j]; }

  // True when all nev pairs of T_n have an estimate of at most tol_est.
  bool solve(double const* a, double const* b, uint32_t n, bool breakdown, double tol_est) {
    uint32_t const found = std::min(nev_, n);
    double lo = 1e300, hi = -1e300;  // Gershgorin
    for (uint32_t i = 0; i < n; ++i) {
      double const r = (i ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < n ? std::fabs(b[i]) : 0.0);
      lo = std::fmin(lo, a[i] - r);
      hi = std::fmax(hi, a[i] + r);
    }
    double const scale = std::fmax(1.0, std::fmax(std::fabs(lo), std::fabs(hi)));
    bool all = found == nev_;
    for (uint32_t j = 0; j < found; ++j) {
      std::vector<double>& s = s_[j];
      // one pair: Rayleigh-quotient iteration from the previous Ritz vector,
      // if a Sturm count certifies that it found the lowest
      if (!(nev_ == 1 && size_ && refine(a, b, n, 1e-12 * scale, s))) {
        double const x = multisect(a, b, n, j, std::fma(-1e-12, scale, lo), std::fma(1e-12, scale, hi));
        s.resize(n);
        for (uint32_t i = 0; i < n; ++i)
          s[i] = 1.0 + 1e-3 * (double)((i * 7919u + j * 104729u) % 1000u) / 1000.0;
        for (int it = 0; it < 3; ++it) {  // inverse iteration, orthogonal to the lower pairs
          for (uint32_t q = 0; q < j; ++q) {
            std::vector<double> const& sq = s_[q];
            double dp = 0.0;
            for (uint32_t i = 0; i < n; ++i) dp = std::fma(sq[i], s[i], dp);
            for (uint32_t i = 0; i < n; ++i) s[i] = std::fma(-dp, sq[i], s[i]);
          }
          normalise(s);
          shifted_solve(a, b, n, x, s);
          normalise(s);
        }
        theta[j] = rayleigh(a, b, n, s);
      }
      est[j] = breakdown ? 0.0 : std::fabs(b[n - 1] * s[n - 1]);
      if (!(est[j] <= tol_est)) all = false;
    }
    size_ = n;
    return all;
  }

 private:
  uint32_t nev_, size_ = 0;
  std::vector<std::vector<double>> s_;
  std::vector<double> dl_, d_, du_, du2_;
  std::vector<uint8_t> piv_;

  bool refine(double const* a, double const* b, uint32_t n, double delta, std::vector<double>& s) {
    s.resize(n, 0.0);
    normalise(s);
    double sigma = rayleigh(a, b, n, s);
    for (int it = 0; it < 3; ++it) {
      shifted_solve(a, b, n, sigma, s);
      normalise(s);
      double const ns = rayleigh(a, b, n, s);
      bool const settled = std::fabs(ns - sigma) <= 1e-15 * std::fmax(1.0, std::fabs(ns));
      sigma = ns;
      if (settled) break;
    }
    if (!(sigma == sigma)) return false;
    double const x = sigma - delta;
    uint32_t below[1];
    count<1>(a, b, n, &x, below);
    if (below[0] != 0) return false;
    theta[0] = sigma;
    return true;
  }

  // Eigenvalues of T below each of P points (Sturm counts of negative
  // pivots): P independent chains of divisions.
  template <int P>
  static void count(double const* a, double const* b, uint32_t n, double const* x, uint32_t* c) {
    double d[P];
    for (int q = 0; q < P; ++q) {
      d[q] = a[0] - x[q];
      c[q] = d[q] < 0.0;
    }
    for (uint32_t i = 1; i < n; ++i) {
      double const bb = b[i - 1] * b[i - 1];
      for (int q = 0; q < P; ++q) {
        double const t = bb / (d[q] == 0.0 ? 1e-300 : d[q]);
        d[q] = (a[i] - x[q]) - t;
        c[q] += d[q] < 0.0;
      }
    }
  }

  // The j-th eigenvalue in [lo, hi]: 33 sections per round. Counts do not
  // fall with x, so the first of the 32 inner points above the eigenvalue is
  // found from every fourth and then the three between.
  static double multisect(double const* a, double const* b, uint32_t n, uint32_t j, double lo, double hi) {
    for (int round = 0; round < 24; ++round) {
      if (hi - lo <= 2e-16 * std::fmax(std::fabs(lo), std::fabs(hi)) + 1e-300) break;
      auto point = [&](int t) { return lo + (hi - lo) * (double)t / 33.0; };  // t = 1..32
      double x[8];
      uint32_t c[8];
      for (int q = 0; q < 8; ++q) x[q] = point(4 * (q + 1));
      count<8>(a, b, n, x, c);
      int first = 33, q8 = 0;
      while (q8 < 8 && c[q8] <= j) ++q8;
      if (q8 < 8) {
        for (int q = 0; q < 3; ++q) x[q] = point(4 * q8 + q + 1);
        count<3>(a, b, n, x, c);
        int q3 = 0;
        while (q3 < 3 && c[q3] <= j) ++q3;
        first = 4 * q8 + q3 + 1;
      }
      double const nlo = first == 1 ? lo : point(first - 1);
      double const nhi = first == 33 ? hi : point(first);
      lo = nlo;
      hi = nhi;
    }
    return 0.5 * (lo + hi);
  }

  // Solves (T - sigma I) z = r in place (r -> z) by Gaussian elimination with
  // partial pivoting on the tridiagonal (the dgttrf/dgtts2 scheme); exactly
  // singular pivots are perturbed.
  void shifted_solve(double const* a, double const* b, uint32_t n, double sigma, std::vector<double>& r) {
    dl_.resize(n);
    d_.resize(n);
    du_.resize(n);
    du2_.resize(n);
    piv_.resize(n);
    double *dl = dl_.data(), *d = d_.data(), *du = du_.data(), *du2 = du2_.data();
    double const tiny = 1e-300;
    for (uint32_t i = 0; i < n; ++i) d[i] = a[i] - sigma;
    for (uint32_t i = 0; i + 1 < n; ++i) {
      dl[i] = b[i];
      du[i] = b[i];
    }
    for (uint32_t i = 0; i + 1 < n; ++i) {
      if (i + 2 < n) du2[i] = 0.0;
      if (std::fabs(d[i]) >= std::fabs(dl[i])) {
        if (d[i] == 0.0) d[i] = tiny;
        double const f = dl[i] / d[i];
        dl[i] = f;
        d[i + 1] = std::fma(-f, du[i], d[i + 1]);
        piv_[i] = 0;
      } else {
        double const f = d[i] / dl[i];
        d[i] = dl[i];
        dl[i] = f;
        double const t = du[i];
        du[i] = d[i + 1];
        d[i + 1] = std::fma(-f, d[i + 1], t);
        if (i + 2 < n) {
          du2[i] = du[i + 1];
          du[i + 1] = -f * du[i + 1];
        }
        piv_[i] = 1;
      }
    }
    if (d[n - 1] == 0.0) d[n - 1] = tiny;
    for (uint32_t i = 0; i + 1 < n; ++i) {
      if (piv_[i]) {
        double const t = r[i];
        r[i] = r[i + 1];
        r[i + 1] = std::fma(-dl[i], r[i], t);
      } else {
        r[i + 1] = std::fma(-dl[i], r[i], r[i + 1]);
      }
    }
    r[n - 1] /= d[n - 1];
    if (n > 1) r[n - 2] = std::fma(-du[n - 2], r[n - 1], r[n - 2]) / d[n - 2];
    for (int i = (int)n - 3; i >= 0; --i)
      r[i] = std::fma(-du2[i], r[i + 2], std::fma(-du[i], r[i + 1], r[i])) / d[i];
  }

  // s^T T s / s^T s. Of the two products that meet first in a row either can
  // be the fused one; the device's loop, unrolled by four, took a[i] s[i] in
  // three rows of four.
  static double rayleigh(double const* a, double const* b, uint32_t n, std::vector<double> const& s) {
    double num = 0.0, den = 0.0;
    for (uint32_t i = 0; i < n; ++i) {
      double ts = a[i] * s[i];
      if (i) ts = (i & 3) ? std::fma(a[i], s[i], b[i - 1] * s[i - 1]) : std::fma(b[i - 1], s[i - 1], ts);
      if (i + 1 < n) ts = std::fma(b[i], s[i + 1], ts);
      num = std::fma(s[i], ts, num);
      den = std::fma(s[i], s[i], den);
    }
    return num / den;
  }

  static void normalise(std::vector<double>& s) {
    double m = 0.0;
    for (double const v : s) m = std::fma(v, v, m);
    if (std::isinf(m)) {  // the shift was an eigenvalue to the last bit
      for (double& v : s) v *= 0x1p-600;
      m = 0.0;
      for (double const v : s) m = std::fma(v, v, m);
    }
    double const inv = 1.0 / std::sqrt(m);
    for (double& v : s) v *= inv;
  }
};

}  // namespace sed
