"""The fixed-point functions of the FP64 state-tile kernel (crs_fx.cuh),
compiled for the host and compared with 80-bit or quad floating point (CPU)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

# Bounds, in units of the exponent's last place 2^-49: a table exponential is
# the truncation of its polynomial (2^-54) plus the rounding of g (2^-51) and
# of 1 + p (2^-56); a logarithm the rounding of u (2^-51), of its 32-bit
# correction (2^-51) and of the sum (2^-49); a net rate two exponentials and
# one FP64 rounding.
SOURCE = r"""
#include "crs_fx.cuh"
#include <cstdio>
#include <random>
#include <vector>
using namespace crs::fx;
typedef long double ld;
int main() {
  std::vector<int64_t> et(EXP_WORDS), lt(2 * (LOGN + 1)), hp(2 * (LOGN + 1));
  for (int j = 0; j <= EXPN; ++j) et[j] = llroundl(ldexpl(exp2l((ld)j / EXPN), 56)) + 8;
  for (int j = 0; j <= LOGN; ++j) {
    const ld F = 1 + (ld)j / LOGN;
    lt[2 * j] = hp[2 * j] = llroundl(ldexpl(1, 62) / F);
    lt[2 * j + 1] = llroundl(ldexpl(log2l(F), YB));
    hp[2 * j + 1] = llroundl(ldexpl(log2l(F), 62));
  }
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> U(0, 1);
  ld e[5] = {0, 0, 0, 0, 0};
  auto up = [&](int k, ld v) { e[k] = fabsl(v) > e[k] ? fabsl(v) : e[k]; };
  for (int i = 0; i < 300000; ++i) {
    const int64_t y = (int64_t)((U(g) - 0.5) * 2000 * 0x1p49) & ~1LL;
    uint64_t M;
    int E;
    exp2m(y, et.data(), M, E);
    // 2^y without its integer part: an 80-bit argument keeps the fraction
    const int64_t n = y >> YB;
    const ld f = exp2l(ldexpl((ld)(y - (n << YB)), -YB));
    up(0, ldexpl((ld)M, E - 56 - (int)n) / f - 1);
    const double v = ldexp(1 + U(g), i % 2 ? (int)(U(g) * 2000 - 1000) : -(int)(U(g) * 3));
    up(1, ldexpl((ld)(log2d(v, lt.data()) - (int64_t)ilogb(v) * (1LL << YB)), -YB) -
              log2l(ldexp(v, -ilogb(v))));
    const double T = 100 * pow(60, U(g));
    up(2, ldexpl((ld)log2hp(T, hp.data()), -58) - log2l(T));
    int64_t a = (int64_t)pow(2, U(g) * 61), b = (int64_t)pow(2, U(g) * 61);
    if (i & 1) a = -a;
    bool ok;
    const int64_t r = ratio2(a, b, ok);
    const ld R = (ld)b / hypotl(a, b);
    up(3, ok ? ldexpl((ld)r, -61) - R * R : 1);
    int64_t z = (y + (int64_t)((U(g) - .5) * pow(2, U(g) * 58))) & ~1LL;
    z |= i % 5 == 0;
    bool sp;
    const double net = net_of<true>(y, z, et.data(), sp);
    if (!sp) {
      const ld q = exp2l(ldexpl((ld)((z & ~1LL) - y), -YB)), s = (z & 1) ? -q : q;
      up(4, (ldexpl(ldexpl(net, (int)-n) / f, 0) - (1 - s)) / (1 + q));
    }
  }
  // scratch limits: overflow, underflow and zero
  bool sp;
  int bad = 0;
  bad += net_special<true>(1030LL << YB, 1029LL << YB, et.data()) ==
         net_special<true>(1030LL << YB, 1029LL << YB, et.data());  // inf - inf
  bad += !std::isinf(net_special<true>(1030LL << YB, 1LL << YB, et.data()));
  bad += net_special<false>(-1060LL << YB, 0, et.data()) != ldexp(1.0, -1060);
  bad += net_of<true>(ZERO_EXP, ZERO_EXP + 2, et.data(), sp) != 0.0 || sp;
  bad += net_of<true>(5LL << YB, 5LL << YB, et.data(), sp) != 0.0 || sp;
  bad += net_of<false>((3LL << YB) | 1, 0, et.data(), sp) != -8.0 || sp;
  printf("%Lg %Lg %Lg %Lg %Lg %d\n", e[0], e[1], e[2], e[3], e[4], bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_fixed_point_functions(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I",
                    os.path.join(REPO, "create_rate_subs_gb300", "csrc"), str(src), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    exp2, log2, hp, ratio, net = (float(v) for v in out[:5])
    u = 2.0 ** -49
    assert exp2 <= u and log2 <= 2 * u and hp <= 4 * 2.0 ** -58 and ratio <= 2.0 ** -50
    assert net <= 2 * u
    assert int(out[5]) == 0
