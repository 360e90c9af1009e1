// 64-bit fixed-point arithmetic of the FP64 state-tile kernel (crs_fx.cu).
//
// GB300 retires one FP64 warp instruction per SM sub-partition in ~70
// clocks and a 32 x 32 -> 64 bit integer multiply-add in a few, so the smooth
// parts of a rate -- exponents, exponentials, logarithms -- are evaluated as
// 64-bit integers:
//   * an exponent is the base-2 logarithm of its value in units of 2^-49
//     (range +-16384): a fixed step of 1.2e-15 of the value, where a double
//     resolves an exponent of 16 binary orders as finely, smaller ones more
//     finely and larger ones less;
//   * bit 0 of every exponent is the sign of its value: adding exponents
//     multiplies the values, signs included;
//   * a 64-bit number is split into two signed 32-bit digits, v = hi 2^32 +
//     lo, and a product keeps hi hi and the two mixed products (three
//     multiply-adds); the dropped lo lo is at most a quarter of the unit.
// Values return to FP64 from 57-bit mantissas with one rounding each.  Plain
// integer code: the same functions compile for the host, where the tests
// compare them with 64-bit floating point.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define FX_FN __host__ __device__ __forceinline__
#else
#define FX_FN inline
#endif

namespace crs {
namespace fx {

constexpr int YB = 49;                         // fraction bits of an exponent
// The ranges (in binary orders) that keep the sum of a rate's exponents inside
// 64 bits and a zero factor zero; what lies outside is left to the general
// arithmetic.  A rate has a constant, at most four concentrations and a fall-
// off factor.
constexpr int CONST_MAX = 800, TERMS_MAX = 500;  // an exponent: c0, its functions of T
constexpr int RATE_MAX = CONST_MAX + TERMS_MAX;
constexpr int RHO_MAX = 60;                      // density: 2^-60 to 2^60
constexpr int W_MAX = 20;                        // 1 / W: 2^-20 to 2^20
constexpr int CONC_MAX = 1 + W_MAX + RHO_MAX;    // mass fractions below 2
constexpr int DE_MAX = 100;                      // the factor d T^e of an SRI form
constexpr int FALL_MIN = -2750, FALL_MAX = DE_MAX + 4;
constexpr int ZERO = -3050;                      // a zero factor
constexpr int NORMAL_MIN = -1081;                // results below it are zero (normal_of)
static_assert(4 * ZERO - RATE_MAX + FALL_MIN > -(1 << (63 - YB)) &&
                  4 * CONC_MAX + RATE_MAX + FALL_MAX < 1 << (63 - YB),
              "the exponent of a rate stays within 64 bits");
static_assert(ZERO + 3 * CONC_MAX + RATE_MAX + FALL_MAX < NORMAL_MIN &&
                  FALL_MIN + 4 * CONC_MAX + RATE_MAX < NORMAL_MIN,
              "a rate with a zero factor is zero");
static_assert(-1022 - W_MAX - RHO_MAX > ZERO, "no concentration is below a zero one");
constexpr int64_t ZERO_EXP = -((int64_t)-ZERO << YB);  // exponent of a zero factor
constexpr int64_t FALL_MIN_EXP = -((int64_t)-FALL_MIN << YB);
constexpr int LOGN = 512;                      // logarithm table: F = 1 + j / 512
// The small tables, in 8-byte words: 2^(j/256) in units of 2^-56 plus 8 units
// (257 entries and one of padding), then pairs (1/F in units of 2^-62, log2 F
// in units of 2^-49).
constexpr int EXPN = 256;
constexpr int EXP_WORDS = EXPN + 2;
constexpr int TAB_BYTES = EXP_WORDS * 8 + (LOGN + 1) * 16;

// ---- the machine's integer operations -------------------------------------
FX_FN int mulhi(int a, int b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int)(((int64_t)a * b) >> 32);
#endif
}
FX_FN int clz64(int64_t v) {
#if defined(__CUDA_ARCH__)
  return __clzll(v);
#else
  return v ? __builtin_clzll((unsigned long long)v) : 64;
#endif
}
FX_FN uint64_t bits_of(double v) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t u;
  memcpy(&u, &v, 8);
  return u;
#endif
}
FX_FN double of_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double v;
  memcpy(&v, &u, 8);
  return v;
#endif
}
// floor(2^61 / d) to 24 bits, 2^30 <= d < 2^31
FX_FN unsigned recip61(unsigned d) {
#if defined(__CUDA_ARCH__)
  return __float2uint_rz(__frcp_rn((float)d) * 2305843009213693952.0f);
#else
  return (unsigned)((1.0f / (float)d) * 2305843009213693952.0f);
#endif
}

// ---- products ---------------------------------------------------------------
struct Dg {
  int hi, lo;
};

FX_FN Dg split(int64_t v) {
  const int lo = (int)(unsigned)(uint64_t)v;
  return Dg{(int)(v >> 32) + (int)((unsigned)lo >> 31), lo};
}

// a b + c as one instruction, spelt out where the sums are short
FX_FN int64_t mad(int a, int b, int64_t c) {
#if defined(__CUDA_ARCH__)
  int64_t d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
#else
  return (int64_t)a * b + c;
#endif
}

// (a b) 2^(S - 64), rounded
template <int S>
FX_FN int64_t mul(Dg a, Dg b) {
  const int64_t mid = mad(a.lo, b.hi, mad(a.hi, b.lo, 1LL << (31 - S)));
  if (S == 0) return mad(a.hi, b.hi, mid >> 32);
  return (int64_t)((uint64_t)mad(a.hi, b.hi, 0) << S) + (mid >> (32 - S));
}

// floor(v 2^lsb) towards zero for |v| < 2^(62 - lsb); infinities and NaN
// give a meaningless number
FX_FN int64_t d2fx(double v, int lsb) {
  const uint64_t u = bits_of(v);
  const int e = (int)(u >> 52) & 0x7ff;
  const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  int sh = 1023 + 62 - lsb - e;
  sh = sh < 0 ? 0 : sh > 63 ? 63 : sh;
  const int64_t r = (int64_t)((m << 10) >> sh);
  return (int64_t)u < 0 ? -r : r;
}

// 2^y as M 2^(E - 56), M in [2^56, 2^57]: y split into an integer, the
// nearest of 257 table points j / 256 and |r| <= 2^-9, 2^r = 1 + r (d1 + r
// (d2 + r (d3 + r d4))) with d_n = (ln 2)^n / n! (truncation below 2^-54).
// The table holds 2^(j/256) + 8 units: the rounding of M's four last bits.
// The sign (bit 0 of y) is dropped.
FX_FN void exp2m(int64_t y, const int64_t *tab, uint64_t &M, int &E) {
  const int vh = (int)(y >> 32);
  const unsigned vl = (unsigned)(uint64_t)y & ~1u;
  E = vh >> (YB - 32);
  const int j = ((vh & ((1 << (YB - 32)) - 1)) + (1 << (YB - 41))) >> (YB - 40);
  const int64_t S = tab[j];
  // r in units of 2^-71: the fraction less j / 256, modulo 2^64
  const int rh = (int)(((unsigned)vh << 22 | vl >> 10) ^ (unsigned)j << 31);  // 2^-39
  const int rl = (int)(vl << 22);
  constexpr int D4 = 5043;        // 2^-19
  constexpr int D3 = 3724818;     // 2^-26
  constexpr int D2 = 2063529982;  // 2^-33
  constexpr int64_t D1 = 99893036290645748LL;  // 2^-57
  const int t = mulhi(rh, D4) + D3;
  const int g = mulhi(rh, t) + D2;
  const int64_t h = D1 + (mad(rh, g, 0) >> 15);
  const Dg r{rh + (int)((unsigned)rl >> 31), rl};
  const Dg p = split(mul<0>(r, split(h))), s = split(S);  // 2^-64
  const int64_t mid = mad(s.lo, p.hi, mad(s.hi, p.lo, 1LL << 31));
  M = (uint64_t)mad(s.hi, p.hi, S + (mid >> 32));
}

// log2 of m 2^-63, m in [2^63, 2^64), in units of 2^-49: m = F (1 + u) with F
// the nearest table point, |u| <= 2^-10, log2(1 + u) = u (c1 + u (c2 + ...))
// to u^5 (truncation below 2^-62).
FX_FN int64_t log2m(uint64_t m, const int64_t *ltab) {
  const unsigned mh = (unsigned)(m >> 32) & 0x7fffffffu;
  const int j = (int)((mh + (1u << 21)) >> 22);
  const int64_t d = (int64_t)((m & 0x7fffffffffffffffull) - ((uint64_t)j << 54)) >> 10;  // 2^-53
#if defined(__CUDA_ARCH__)
  const longlong2 c = *reinterpret_cast<const longlong2 *>(ltab + 2 * j);
  const int64_t inv = c.x, lf = c.y;
#else
  const int64_t inv = ltab[2 * j], lf = ltab[2 * j + 1];
#endif
  const int64_t u = mul<0>(split(d), split(inv));  // 2^-51
  const int u32 = (int)((u + 512) >> 10);          // 2^-41
  constexpr int C5 = 5;                            // 2^-4
  constexpr int C4 = -2955;                        // 2^-13
  constexpr int C3 = 2017034;                      // 2^-22
  constexpr int C2 = -1549082005;                  // 2^-31
  constexpr int64_t C1 = 6653256548922161246LL;    // 2^-62
  int g = mulhi(u32, C5) + C4;
  g = mulhi(u32, g) + C3;
  g = mulhi(u32, g) + C2;
  const int64_t h = C1 + (mad(u32, g, 0) >> 10);
  return lf + mul<0>(split(u), split(h));
}

// An exponent with bit 0 cleared (to the nearest even number), ready for a
// sign.
FX_FN int64_t even(int64_t y) { return (y + 1) & ~1LL; }

// log2 |v| of a normal double (bit 0 arbitrary)
FX_FN int64_t log2d(double v, const int64_t *ltab) {
  const uint64_t u = bits_of(v);
  const int e = ((int)(u >> 52) & 0x7ff) - 1023;
  return (int64_t)e * (1LL << YB) + log2m((u << 11) | 0x8000000000000000ull, ltab);
}

// log2 of a 2^-lsb, a > 0 (bit 0 arbitrary)
FX_FN int64_t log2i(int64_t a, int lsb, const int64_t *ltab) {
  const int lz = clz64(a);
  return (int64_t)(63 - lz - lsb) * (1LL << YB) + log2m((uint64_t)a << lz, ltab);
}

// log2 of a normal positive double in units of 2^-58 (|log2| < 16): the
// temperature's, which Kc polynomials multiply by tens.  hp: 1/F as in
// ltab, log2 F in units of 2^-62 (pairs).
FX_FN int64_t log2hp(double v, const int64_t *hp) {
  const uint64_t u = bits_of(v);
  const int e = ((int)(u >> 52) & 0x7ff) - 1023;
  const uint64_t m = (u << 11) | 0x8000000000000000ull;
  const unsigned mh = (unsigned)(m >> 32) & 0x7fffffffu;
  const int j = (int)((mh + (1u << 21)) >> 22);
  const int64_t d = (int64_t)((m & 0x7fffffffffffffffull) - ((uint64_t)j << 54));  // 2^-63
  const Dg w = split(mul<1>(split(d * 2), split(hp[2 * j])));  // d 2^-64, 1/F 2^-62: 2^-63
  // log2(1 + w) by its Taylor series to w^7 (truncation below 2^-66)
  constexpr int64_t C[7] = {6653256548922161246LL, -3326628274461080623LL, 2217752182974053749LL,
                            -1663314137230540311LL, 1330651309784432249LL, -1108876091487026874LL,
                            950465221274594464LL};  // 2^-62
  int64_t h = C[6];
  for (int n = 5; n >= 0; --n) h = C[n] + mul<1>(w, split(h));
  h = mul<1>(w, split(h)) + hp[2 * j + 1];  // 2^-62
  return (int64_t)e * (1LL << 58) + (h >> 4);
}

// The sum of up to three signed numbers M 2^(E - 56), M in [2^56, 2^57], in
// units of 2^(e - 60) with e the largest term's exponent: a fall-off centre
// may be any power of two, and an absolute unit would leave a small one
// without its last bits (in units of 2^-59, centres near 2^-20: up to 5e-12 of
// the factor).
struct Sum {
  int64_t v = 0;
  int e = -4000;
  FX_FN void add(uint64_t M, int E, bool neg) {
    const int64_t m = (int64_t)(M << 4);
    const int d = E - e, n = d > 63 ? 63 : d < -63 ? 63 : d < 0 ? -d : d;
    const int64_t t = neg ? -m : m;
    v = d > 0 ? (v >> n) + t : v + (t >> n);
    e = d > 0 ? E : e;
  }
  // Not a positive number that the general arithmetic would leave as it is:
  // below its limit of 1e-300, above two (E <= 1), or less than 1/16 of the
  // largest term, whose exponent's rounding the difference would magnify.
  FX_FN bool outside() const { return e > 1 || e < -990 || v < (1LL << 56); }
  // log2 of the sum (bit 0 arbitrary)
  FX_FN int64_t log2(const int64_t *ltab) const;
};

// b^2 / (a^2 + b^2) in units of 2^-61 for |a|, |b| < 2^62; ok = false when
// both are zero.  The quotient of the 64-bit squares from a 24-bit
// reciprocal R0 of the denominator and two terms of its residual eps,
// 1 / (1 - eps) = 1 + eps + eps^2 (next term below 2^-66).
FX_FN int64_t ratio2(int64_t a, int64_t b, bool &ok) {
  a = a < 0 ? -a : a;
  b = b < 0 ? -b : b;
  const int s = clz64((a > b ? a : b) | 1) - 2;
  const Dg da = split(a << s), db = split(b << s);
  int64_t B = mul<2>(db, db);
  B = B < 0 ? 0 : B;
  int64_t D = mul<2>(da, da) + B;
  ok = D > 0;
  const int s2 = clz64(D | 1) - 1;
  D = (int64_t)((uint64_t)D << s2);
  B = (int64_t)((uint64_t)B << s2);
  const unsigned R0 = recip61((unsigned)(D >> 32));
  const uint64_t one =
      (D >> 32) * (uint64_t)R0 + (((uint64_t)(unsigned)(uint64_t)D * R0) >> 32);
  const int eps = (int)((int64_t)((1ull << 61) - one) >> 8);  // 2^-53
  const uint64_t q0 =
      (B >> 32) * (uint64_t)R0 + (((uint64_t)(unsigned)(uint64_t)B * R0) >> 32);  // 2^-61
  const int64_t t1 = mad((int)(q0 >> 31), eps, 0);
  const int64_t t2 = mad((int)(t1 >> 32), eps, 0);
  return (int64_t)q0 + (t1 >> 22) + (t2 >> 43);
}

// log2 of the broadening factor, log2 of the centre over 1 + (A / B)^2 (Troe)
// or of the SRI base over 1 + log10(Pr)^2; zF: log2 of the centre or base, zP:
// log2 Pr.  ok = false: 0 / 0.
constexpr int64_t LOG2_10 = 1870079266285788LL;   // log2 10
constexpr int64_t C04 = 748031706514315LL;        // 0.4 log2 10
constexpr int64_t C0806 = 1507283888626345LL;     // 0.806 log2 10
constexpr int64_t K067 = 3089829632346349896LL;   // 0.67, 2^-62
constexpr int64_t K11762 = 5424265094874293653LL; // 1.1762
constexpr int64_t K014 = 645636042579834307LL;    // 0.14
FX_FN int64_t broadening(int64_t zF, int64_t zP, bool troe, bool &ok) {
  int64_t A = zP, B = LOG2_10;
  const Dg kF = split(zF);
  if (troe) {
    A = zP - mul<2>(kF, split(K067)) - C04;
    B = C0806 - mul<2>(kF, split(K11762)) - mul<2>(split(zP), split(K014));
  }
  return mul<3>(kF, split(ratio2(A, B, ok)));
}

FX_FN int64_t Sum::log2(const int64_t *ltab) const { return log2i(v > 1 ? v : 1, 60 - e, ltab); }

// The value of one exponent (bit 0: its sign), with overflow to infinity and
// gradual underflow.
FX_FN double value_of(int64_t y, const int64_t *tab) {
  uint64_t M;
  int E;
  exp2m(y, tab, M, E);
  const double m = (double)(int64_t)M;  // M <= 2^57: rounds once
  return ldexp((y & 1) ? -m : m, E - 56);
}

// The value of one exponent as a normal double by integer operations; zero
// far below the normal range.  far: overflow or gradual underflow, which
// value_of has to form: NaN.
FX_FN double normal_of(int64_t y, const int64_t *tab, bool &far) {
  uint64_t M;
  int E;
  exp2m(y, tab, M, E);
  const unsigned e = (unsigned)(E + 1022);
  const bool in = e <= 2044u;
  far = !in && E > NORMAL_MIN;
  const unsigned lo = (unsigned)(M >> 4);
  const unsigned hi = ((unsigned)(M >> 36) + (e << 20)) ^ ((unsigned)y << 31);
  return of_bits((uint64_t)(in ? hi : far ? 0x7ff80000u : 0u) << 32 | (in ? lo : 0u));
}

// +-2^yf -+ 2^yr (bit 0 of each exponent: its sign).  REV false: the first
// term alone.  special: a term lies outside the normal range, the result is NaN
// and net_special has to form it; the code has no branch.
template <bool REV>
FX_FN double net_of(int64_t yf, int64_t yr, const int64_t *tab, bool &special) {
  const double f = normal_of(yf, tab, special);
  if (!REV) return f;
  bool far;
  const double r = normal_of(yr, tab, far);
  special |= far;
  return f - r;
}

// net_of for any range: terms that overflow give infinities (and their
// difference NaN), tiny results underflow gradually.
template <bool REV>
FX_FN double net_special(int64_t yf, int64_t yr, const int64_t *tab) {
  const double f = value_of(yf, tab);
  return REV ? f - value_of(yr, tab) : f;
}

}  // namespace fx
}  // namespace crs
