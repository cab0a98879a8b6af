"""The host solver for the Lanczos matrix (csrc/tridiagonal.hpp) against
numpy's dense eigensolver, at orders around the blocks it works in."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spin-ed_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include "tridiagonal.hpp"
int main() {  // nev, then orders n and their a[n], b[n]; prints theta, est and vectors per order
  unsigned nev, n;
  if (std::scanf("%u", &nev) != 1) return 1;
  sed::Tridiagonal T(nev);
  while (std::scanf("%u", &n) == 1) {
    std::vector<double> a(n), b(n);
    for (double& v : a) if (std::scanf("%lf", &v) != 1) return 1;
    for (double& v : b) if (std::scanf("%lf", &v) != 1) return 1;
    std::printf("%d\n", (int)T.solve(a.data(), b.data(), n, false, 1e-3));
    for (unsigned j = 0; j < nev && j < n; ++j) {
      std::printf("%.17g %.17g", T.theta[j], T.est[j]);
      for (double v : T.vector(j)) std::printf(" %.17g", v);
      std::printf("\n");
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def solver(tmp_path_factory):
    d = tmp_path_factory.mktemp("tri")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I" + CSRC, str(d / "main.cpp"), "-o", str(d / "tri")])
    return str(d / "tri")


@pytest.mark.parametrize("nev,orders", [(1, [1, 2, 3, 4, 8, 60, 61, 200]), (4, [2, 4, 5, 33, 64, 200]), (16, [16, 48])])
def test_lowest_pairs(solver, nev, orders):
    rng = np.random.default_rng(nev)
    a, b = rng.uniform(-40.0, 20.0, 200), rng.uniform(1.0, 15.0, 200)
    text = f"{nev}\n" + "".join(f"{n} " + " ".join(f"{v:.17g}" for v in np.concatenate([a[:n], b[:n]])) + "\n"
                                for n in orders)
    lines = iter(subprocess.run([solver], input=text, capture_output=True, text=True, check=True).stdout.splitlines())
    for n in orders:
        T = np.diag(a[:n]) + np.diag(b[:n - 1], 1) + np.diag(b[:n - 1], -1)
        want = np.linalg.eigvalsh(T)
        norm = np.abs(T).sum(axis=1).max()
        ok = bool(int(next(lines)))
        est = []
        for j in range(min(nev, n)):
            v = np.array([float(x) for x in next(lines).split()])
            theta, s = v[0], v[2:]
            est.append(v[1])
            # Sturm counts and Rayleigh quotients are backward stable: a few
            # roundings per row of the largest element
            assert abs(theta - want[j]) <= 4 * n * 2.0 ** -53 * norm
            assert abs(np.linalg.norm(s) - 1.0) <= n * 2.0 ** -52
            r = np.linalg.norm(T @ s - theta * s)
            if nev == 1:
                # the iteration ends when its Rayleigh quotient settles: for
                # the lowest pair r^2 <= (theta - lambda) (lambda_max - lambda)
                assert r <= (4 * n * 2.0 ** -53 * norm * 2 * norm) ** 0.5
            else:
                assert r <= 64 * n * 2.0 ** -53 * norm
            assert v[1] == abs(b[n - 1] * s[-1])
        assert ok == (n >= nev and max(est) <= 1e-3)
