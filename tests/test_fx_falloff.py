"""The broadening of fall-off rates in the fixed-point arithmetic of the FP64
state tiles (crs_fx.cuh), compiled for the host and compared with 80-bit or
quad floating point (CPU)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

# For each binary order of the centre, from 1 down to 2^-40 and at a few orders
# far below, centres of one, two and three terms at random log2 Pr.  Bound of
# the broadening factor's logarithm (base 2): log2 of a term is rounded to
# 2^-49 and its exponential to 2^-51 of its value (1.25 units, relative, ln 2
# of a unit of the logarithm: 1.3 units), the logarithm of the sum adds 2
# units; the weight, at most 1, multiplies these.  The weight itself is within
# 2^-54 for A and B within 2 units each (its slope in A / B is below 0.7 and
# B at least 1 apart from the pole of A / B): times |log2 F|, (|zF| + 2) 2^-49
# covers it with the unit of the product.  In all (6 + |zF|) 2^-49.
SOURCE = r"""
#include "crs_fx.cuh"
#include <cstdio>
#include <random>
#include <vector>
using namespace crs::fx;
typedef long double ld;
int main() {
  std::vector<int64_t> et(EXP_WORDS), lt(2 * (LOGN + 1));
  for (int j = 0; j <= EXPN; ++j) et[j] = llroundl(ldexpl(exp2l((ld)j / EXPN), 56)) + 8;
  for (int j = 0; j <= LOGN; ++j) {
    const ld F = 1 + (ld)j / LOGN;
    lt[2 * j] = llroundl(ldexpl(1, 62) / F);
    lt[2 * j + 1] = llroundl(ldexpl(log2l(F), YB));
  }
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> U(0, 1);
  ld worst = 0;
  int outside = 0, cancel = 0;
  for (int i = 0; i < 200000; ++i) {
    const int order = i % 45;
    const double top = order < 41 ? -order : order == 41 ? -100 : order == 42 ? -500 : -900;
    const int terms = 1 + (i / 45) % 3;
    const bool troe = (i / 135) % 2;
    Sum S;
    ld c = 0;
    for (int k = 0; k < terms; ++k) {
      const ld y = top + (k ? -30 * U(g) * U(g) : -U(g));
      uint64_t M;
      int E;
      exp2m(llroundl(ldexpl(y, YB)) & ~1LL, et.data(), M, E);
      S.add(M, E, false);
      c += exp2l(y);
    }
    if (S.outside()) {
      ++outside;
      continue;
    }
    const int64_t zP = (int64_t)((U(g) - 0.5) * 80 * 0x1p49) & ~1LL;
    bool ok;
    const ld got = ldexpl((ld)broadening(S.log2(lt.data()), zP, troe, ok), -YB);
    const ld z = ldexpl((ld)zP, -YB), f = log2l(c), l10 = log2l(10.0L);
    ld A = z / l10, B = 1;
    if (troe) {
      A = z / l10 - 0.67L * f / l10 - 0.4L;
      B = 0.806L - 1.1762L * f / l10 - 0.14L * z / l10;
    }
    const ld want = f * (B * B) / (A * A + B * B);
    const ld e = ok ? ldexpl(fabsl(got - want), YB) / (6 + fabsl(f)) : 1e9L;
    worst = e > worst ? e : worst;
  }
  // a difference that loses more than four bits, a negative one, one below
  // the general arithmetic's limit and none at all are left to it
  auto two = [&](double a, double b, bool neg) {
    Sum S;
    uint64_t M;
    int E;
    exp2m((int64_t)(a * 0x1p49) & ~1LL, et.data(), M, E);
    S.add(M, E, false);
    exp2m((int64_t)(b * 0x1p49) & ~1LL, et.data(), M, E);
    S.add(M, E, neg);
    return S.outside();
  };
  cancel += two(-3.0, -3.01, true) + two(-3.0, -2.0, true) + two(-1000.0, -1001.0, false) +
            Sum().outside() + two(-3500.0, -3500.0, false) + two(5.0, -1.0, false);
  cancel += 10 * (two(-3.0, -4.0, true) + two(-4.0, -3500.0, true) + two(-3500.0, -4.0, false) +
                  two(0.0, 0.0, false));
  printf("%Lg %d %d\n", worst, outside, cancel);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_broadening_of_small_centres(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I",
                    os.path.join(REPO, "create_rate_subs_gb300", "csrc"), str(src), "-o", exe],
                   check=True)
    worst, outside, cancel = subprocess.run([exe], check=True, capture_output=True,
                                            text=True).stdout.split()
    assert float(worst) <= 1 and int(outside) == 0 and int(cancel) == 6
