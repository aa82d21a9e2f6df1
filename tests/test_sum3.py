"""Sums of three FP32 values (homogenization's r.r and r.(D^-1 r) in mixed precision):
of one system's products, over eight decades of residuals and over the moduli that FP32
holds, they are within 2^-60 of the sum before their one rounding to FP64 and within
2^-53, all that FP64 can hold of it, after.  FP64 sums of the same products are no
closer."""
from fractions import Fraction

import numpy as np
import pytest

from host_cpp import run_cpp

PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "tg_sum3.h"
using tg::Sum3;
// 256 threads take every 256th product each, as a CTA does; then the 32 lanes of a warp.
int main(int, char** a) {
  const int n = std::atoi(a[1]);
  std::vector<float> v(n), d(n);
  FILE* f = std::fopen(a[2], "rb");
  if (std::fread(v.data(), 4, n, f) + std::fread(d.data(), 4, n, f) != size_t(2 * n)) return 1;
  std::vector<Sum3<float>> s(256, Sum3<float>{0, 0, 0}), w = s;
  for (int i = 0; i < n; ++i) {
    tg::sum3_square(s[i % 256], v[i]);
    tg::sum3_weighted_square(w[i % 256], d[i], v[i]);
  }
  for (auto* t : {&s, &w})
    for (int o = 128; o > 0; o >>= 1)
      for (int i = 0; i < o; ++i) (*t)[i] = tg::sum3_join((*t)[i], (*t)[i + o]);
  for (const auto& t : {s[0], w[0]})
    std::printf("%.9g %.9g %.9g %.17g\\n", t.h, t.m, t.l, tg::sum3_total(t.h, t.m, t.l));
}
"""


@pytest.mark.parametrize("n", [1, 255, 3 * 8 ** 3, 3 * 32 ** 3])
@pytest.mark.parametrize("low", [1.0, 1e-8])
@pytest.mark.parametrize("modulus", [1e-35, 1.0, 2.1e11, 1e35])
def test_products_of_a_system(tmp_path, n, low, modulus):
    rng = np.random.default_rng(n)
    v = rng.standard_normal(n) * np.exp(rng.uniform(np.log(low), 0.0, n))
    v = (v / np.linalg.norm(v)).astype(np.float32)
    d = 1.0 / (0.235 * modulus * rng.integers(1, 9, n))
    d = (d * 2.0 ** int(np.log2(0.235 * modulus) / 2)).astype(np.float32)  # as they are scaled
    (tmp_path / "data").write_bytes(v.tobytes() + d.tobytes())
    out = run_cpp(tmp_path, PROGRAM, n, tmp_path / "data").stdout.split("\n")
    terms = ([Fraction(float(x)) ** 2 for x in v],
             [Fraction(float(y)) * Fraction(float(x)) ** 2 for x, y in zip(v, d)])
    for line, exact in zip(out, (sum(terms[0]), sum(terms[1]))):
        h, m, l, total = line.split()
        pieces = sum(Fraction(float(np.float32(s))) for s in (h, m, l))
        assert abs(pieces - exact) <= exact * Fraction(2) ** -60
        assert abs(Fraction(float(total)) - exact) <= exact * Fraction(2) ** -53


def test_fp64_sums_are_no_closer(tmp_path):
    """What the sums replace: FP64 products added up in the same order."""
    n, rng = 3 * 32 ** 3, np.random.default_rng(1)
    v = rng.standard_normal(n).astype(np.float32)
    d = rng.uniform(0.1, 1.0, n).astype(np.float32)
    (tmp_path / "data").write_bytes(v.tobytes() + d.tobytes())
    line = run_cpp(tmp_path, PROGRAM, n, tmp_path / "data").stdout.split("\n")[1]
    exact = sum(Fraction(float(y)) * Fraction(float(x)) ** 2 for x, y in zip(v, d))
    v64 = v.astype(np.float64).reshape(-1, 256)
    t = v64 * (d.reshape(-1, 256) * v64)
    s = np.zeros(256)
    for row in t:
        s = s + row
    while s.size > 1:
        s = s[:s.size // 2] + s[s.size // 2:]
    fp64 = abs(Fraction(float(s[0])) - exact)
    assert abs(Fraction(float(line.split()[3])) - exact) <= fp64
