// Tables of the FP64 state-tile kernel (crs_fx.cu): every rate and
// equilibrium constant as fixed-point coefficients of normalised functions
// of T, built once at load time in extended precision.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/crs_tables.h"
#include "crs_fx.cuh"
#include "crs_fx_tab.cuh"

namespace crs {
namespace fx {
namespace {

typedef long double ld;
const ld LOG2E = 1.442695040888963407359924681001892137L;

// Coefficients of 1, L, I, t, t^2, t^3, t^4 on one temperature interval.
struct Form {
  ld c[7] = {0, 0, 0, 0, 0, 0, 0};
};

// Centre and half width of T, log2 T and 1/T on an interval, and the
// integers with which the kernel normalises them: F = (x - m) 2^s K 2^-62,
// the coefficients use the half width that these integers realise.
struct Norm {
  ld mT, hT, mL, hL, mI, hI;
  int64_t word[BASIS];
};

void normalise(ld a, ld b, int lsb, ld *mid, ld *half, int64_t *w) {
  const int64_t m = llroundl(std::ldexp((a + b) / 2, lsb));
  const int64_t x = (int64_t)std::ceil(std::ldexp((b - a) / 2, lsb)) + 2;
  int s = 0;
  while ((x << (s + 1)) < (1LL << 62)) ++s;
  const int64_t K = (int64_t)std::floor(std::ldexp((ld)1, 123) / (ld)(x << s));
  *mid = std::ldexp((ld)m, -lsb);
  *half = std::ldexp((ld)1, 123 - s - lsb) / (ld)K;
  w[0] = m;
  w[1] = K;
  w[2] = s;
}

Norm norm_of(double a, double b) {
  Norm n;
  normalise(a, b, 49, &n.mT, &n.hT, n.word);
  normalise(std::log2((ld)a), std::log2((ld)b), 58, &n.mL, &n.hL, n.word + 3);
  normalise(1 / (ld)b, 1 / (ld)a, 68, &n.mI, &n.hI, n.word + 6);
  return n;
}

// log2 of a rate row: base + b log2 T + i / T
struct Row {
  ld base = 0, b = 0, i = 0;
  bool neg = false, ok = false;
};

Row row_of(const Tab &t, int r) {
  const double *p = t.rate_par + 4 * r;  // A, logA, b, Ta
  Row w;
  const int kind = t.rate_kind[r];
  if (kind > RATE_POW || p[0] == 0.0 || !std::isfinite(p[0])) return w;
  w.ok = true;
  w.neg = p[0] < 0;
  w.base = kind == RATE_EXP ? (ld)p[1] * LOG2E : std::log2(std::fabs((ld)p[0]));
  if (kind == RATE_EXP || kind == RATE_NEGEXP) {
    w.b = p[2];
    w.i = -(ld)p[3] * LOG2E;
  } else if (kind == RATE_POW) {
    w.b = t.rate_npow[r];
  }
  return w;
}

// base + b log2 T + i / T + p[0] T + ... + p[3] T^4 on the interval of n
Form form_of(const Norm &n, ld base, ld b, ld i, const ld *p) {
  Form f;
  f.c[0] = base + b * n.mL + i * n.mI;
  f.c[1] = b * n.hL;
  f.c[2] = i * n.hI;
  if (p) {
    static const int binom[5][5] = {{1}, {1, 1}, {1, 2, 1}, {1, 3, 3, 1}, {1, 4, 6, 4, 1}};
    for (int k = 0; k <= 4; ++k)
      for (int d = k > 1 ? k : 1; d <= 4; ++d) {
        const ld v = p[d - 1] * binom[d][k] * std::pow(n.mT, (ld)(d - k)) * std::pow(n.hT, (ld)k);
        f.c[k == 0 ? 0 : 2 + k] += v;
      }
  }
  return f;
}

// The bounds that keep every sum of the kernel inside 64 bits: with
// coefficients of at most 500 in all, six products of the low digits (2^31
// by 2^29) and of the high ones (500 2^20 by 2^31) stay below 2^63; with
// constants of at most 4000, an exponent plus four concentrations stays
// within 2^14.
bool within(const Form &f) {
  ld s = 0;
  for (int k = 1; k < 7; ++k) s += std::fabs(f.c[k]);
  return std::isfinite((double)f.c[0]) && std::fabs(f.c[0]) <= 4000 && s <= 500;
}

int64_t constant(ld v) { return llroundl(std::ldexp(v, YB)); }

// a coefficient as the kernel loads it: {hi, lo} digits
int64_t coefficient(ld v) {
  const Dg d = split(llroundl(std::ldexp(v, 52)));
  return (int64_t)(((uint64_t)(unsigned)d.lo << 32) | (unsigned)d.hi);
}
// a 64-bit number as an int2 {high, low}
int64_t number(int64_t v) {
  return (int64_t)(((uint64_t)v << 32) | ((uint64_t)v >> 32));
}

struct Buf {
  std::vector<unsigned char> b;
  template <class T>
  int put(const std::vector<T> &v) {
    const size_t off = (b.size() + 127) / 128 * 128;
    b.resize(off + v.size() * sizeof(T) + 16);
    if (!v.empty()) memcpy(b.data() + off, v.data(), v.size() * sizeof(T));
    return (int)off;
  }
};

// One exponential term: log2|a| + x T (or x / T); dead: zero on the whole
// interval.  Returns false when it does not fit the scheme.
bool term(const Norm &n, ld a, ld x, bool inv, int64_t *w, int *flags, int bit) {
  if (a == 0) return true;
  if (!std::isfinite((double)a) || !std::isfinite((double)x)) return false;
  const ld m = inv ? n.mI : n.mT, h = inv ? n.hI : n.hT;
  ld c0 = std::log2(std::fabs(a)) + x * m, c1 = x * h;
  *flags |= bit;
  if (c0 + std::fabs(c1) < -1200) {
    c0 = -3500;
    c1 = 0;
  }
  if (std::fabs(c0) > 4000 || std::fabs(c1) > 450) return false;
  w[0] = number((constant(c0) & ~1LL) | (a < 0));
  w[1] = coefficient(c1);
  return true;
}

}  // namespace

void build(const Tab &t, FxTab &f, std::vector<unsigned char> &out) {
  f = FxTab();
  out.clear();
  const int N = t.N, R = t.R, NPM = t.NPM;
  f.N = N;
  f.R = R;
  f.NPM = NPM;
  if (R < 1 || N > 65534) return;
  // interval bounds: the most common T_common in the middle
  double mid = 1000.0;
  {
    std::vector<double> tc(t.sp_tmid, t.sp_tmid + N);
    std::sort(tc.begin(), tc.end());
    int best = 0;
    for (int i = 0, j; i < N; i = j) {
      for (j = i; j < N && tc[j] == tc[i]; ++j) {
      }
      if (j - i > best && tc[i] > 250.0 && tc[i] < 4000.0) {
        best = j - i;
        mid = tc[i];
      }
    }
  }
  f.tb[0] = 120.0;
  f.tb[1] = 200.0;
  f.tb[2] = mid;
  f.tb[3] = 6000.0;
  std::vector<int64_t> basis;
  Norm nm[NI];
  for (int q = 0; q < NI; ++q) {
    nm[q] = norm_of(f.tb[q], f.tb[q + 1]);
    basis.insert(basis.end(), nm[q].word, nm[q].word + BASIS);
  }
  // pressure modification
  std::vector<int32_t> pmh(4 * (size_t)std::max(NPM, 1), 0);
  std::vector<int64_t> pmc((size_t)PMC * NI * std::max(NPM, 1), 0);
  std::vector<char> pm_ok(std::max(NPM, 1), 1);
  std::vector<int32_t> pm_rxn(std::max(NPM, 1), 0);
  for (int r = 0; r < R; ++r)
    if (t.pm_idx[r] >= 0) pm_rxn[t.pm_idx[r]] = r;
  ld worst = 0;
  for (int p = 0; p < NPM; ++p) {
    ld s = 0;
    for (int e = t.pm_eff_ptr[p]; e < t.pm_eff_ptr[p + 1]; ++e)
      s += std::fabs((ld)t.pm_eff_val[e] * t.inv_mw[t.pm_eff_sp[e]]);
    worst = std::max(worst, s);
  }
  // third-body sums: |sum| <= 2 and 1 / mw < 2 in units of 2^eff_shift
  f.eff_shift = 1;
  while (std::ldexp(worst, -f.eff_shift) > 1 && f.eff_shift < 60) ++f.eff_shift;
  if (std::ldexp(worst, -f.eff_shift) > 1) return;
  std::vector<int64_t> eff_k;
  for (int p = 0; p < NPM; ++p) {
    int flags = 0;
    const bool thd = t.pm_kind[p] == PM_THD;
    const int sp = thd ? -1 : t.pm_sp[p];
    if (sp < 0) flags |= PMF_SUM;
    bool ok = true;
    if (!thd) {
      const Row a = row_of(t, t.pm_k0[p]), b = row_of(t, t.pm_kinf[p]);
      ok = a.ok && b.ok && !a.neg && !b.neg;
      if (t.pm_kind[p] == PM_FALL_LOW) flags |= PMF_LOW;
      const double *c = t.pm_troe + 5 * p, *d = t.pm_sri + 5 * p;
      const int form = t.pm_form[p];
      if (form == FORM_TROE) flags |= PMF_TROE;
      if (form == FORM_SRI) flags |= PMF_SRI;
      for (int q = 0; q < NI && ok; ++q) {
        int64_t *w = pmc.data() + (size_t)PMC * (NI * p + q);
        const Form z = form_of(nm[q], a.base - b.base, a.b - b.b, a.i - b.i, nullptr);
        ok = within(z);
        if (!ok) break;
        w[0] = number(constant(z.c[0]));
        w[1] = coefficient(z.c[1]);
        w[2] = coefficient(z.c[2]);
        if (form == FORM_TROE) {
          ok = c[1] != 0.0 && c[3] != 0.0 &&
               term(nm[q], c[0], -LOG2E / c[1], false, w + 3, &flags, PMF_T1) &&
               term(nm[q], c[2], -LOG2E / c[3], false, w + 5, &flags, PMF_T2) &&
               (!t.pm_troe_t2[p] ||
                term(nm[q], 1.0, -LOG2E * c[4], true, w + 7, &flags, PMF_T3));
        } else if (form == FORM_SRI) {
          ok = d[2] != 0.0 && term(nm[q], 1.0, -LOG2E / d[2], false, w + 5, &flags, PMF_T2) &&
               term(nm[q], d[0], -LOG2E * d[1], true, w + 7, &flags, PMF_T3);
          if (ok && t.pm_sri_de[p]) {
            flags |= PMF_DE;
            ok = d[3] > 0.0;
            if (ok) {
              const Form y = form_of(nm[q], std::log2((ld)d[3]), d[4], 0, nullptr);
              ok = within(y);
              w[9] = number(constant(y.c[0]));
              w[10] = coefficient(y.c[1]);
            }
          }
        }
      }
    }
    for (int e = t.pm_eff_ptr[p]; e < t.pm_eff_ptr[p + 1]; ++e)
      eff_k.push_back([&] {
        const Dg d = split(llroundl(std::ldexp(
            (ld)t.pm_eff_val[e] * t.inv_mw[t.pm_eff_sp[e]], 61 - f.eff_shift)));
        return (int64_t)(((uint64_t)(unsigned)d.lo << 32) | (unsigned)d.hi);
      }());
    pmh[4 * p] = flags;
    pmh[4 * p + 1] = sp;
    pmh[4 * p + 2] = pm_rxn[p];
    pm_ok[p] = ok;
  }
  // reactions
  std::vector<int32_t> hdr(8 * (size_t)R, 0), thr_ptr(R + 1, 0);
  std::vector<double> thr;
  std::vector<int64_t> coef;
  std::vector<int> weight(R);
  f.uniform = 1;
  int generic = 0;
  for (int r = 0; r < R; ++r) {
    const int j = t.rev_idx[r], p = t.pm_idx[r];
    const Row a = row_of(t, r);
    bool ok = a.ok && (p < 0 || pm_ok[p]);
    int flags = 0;
    int fac[2][4], cnt[2] = {0, 0};
    for (int side = 0; side < 2; ++side) {
      const int32_t *ptr = side ? t.px_ptr : t.rx_ptr, *sp = side ? t.px_sp : t.rx_sp;
      const int32_t *nint = side ? t.px_nint : t.rx_nint;
      for (int q = 0; q < 4; ++q) fac[side][q] = N;
      if (side && j < 0) break;
      for (int e = ptr[r]; e < ptr[r + 1]; ++e) {
        if (nint[e] < 0) ok = false;
        for (int q = 0; q < nint[e]; ++q, ++cnt[side])
          if (cnt[side] < 4) fac[side][cnt[side]] = sp[e];
      }
      ok &= cnt[side] <= 4;
    }
    // thresholds: the interval bounds and the reaction's own T_common values
    std::vector<double> th = {f.tb[1], f.tb[2]};
    if (j >= 0)
      for (int g = t.kc_ptr[j]; g < t.kc_ptr[j + 1]; ++g) {
        const double x = t.kc_tmid[g];
        if (x > f.tb[0] && x < f.tb[3] && std::find(th.begin(), th.end(), x) == th.end()) {
          th.push_back(x);
          f.uniform = 0;
        }
      }
    std::sort(th.begin(), th.end());
    const int base = (int)(coef.size() / COEF);
    for (size_t q = 0; q <= th.size(); ++q) {
      const double hi = q < th.size() ? th[q] : f.tb[3];
      int iv = 0;
      while (hi > f.tb[iv + 1]) ++iv;
      int64_t w[COEF] = {0};
      const Form y = form_of(nm[iv], a.base, a.b, a.i, nullptr);
      ok &= within(y);
      Form z = y;
      if (j >= 0) {
        ld b0 = a.base - std::log((ld)t.kc_pref[j]) * LOG2E, b1 = a.b, bi = a.i, pl[4] = {0, 0, 0, 0};
        for (int g = t.kc_ptr[j]; g < t.kc_ptr[j + 1]; ++g) {
          const double *c = (hi <= t.kc_tmid[g] ? t.kc_lo : t.kc_hi) + 7 * g;
          b0 -= (ld)c[0] * LOG2E;
          b1 -= c[1];
          for (int k = 0; k < 4; ++k) pl[k] -= (ld)c[2 + k] * LOG2E;
          bi += (ld)c[6] * LOG2E;
        }
        z = form_of(nm[iv], b0, b1, bi, pl);
        ok &= within(z);
      }
      if (ok) {
        w[0] = number(constant(y.c[0]));
        w[1] = coefficient(y.c[1]);
        w[2] = coefficient(y.c[2]);
        w[3] = number(constant(z.c[0]));
        for (int k = 1; k < 7; ++k) w[3 + k] = coefficient(z.c[k]);
      }
      coef.insert(coef.end(), w, w + COEF);
    }
    thr.insert(thr.end(), th.begin(), th.end());
    thr_ptr[r + 1] = (int32_t)thr.size();
    if (j >= 0) flags |= RF_REV;
    if (p >= 0) flags |= t.pm_kind[p] == PM_THD ? RF_THD : RF_FALL;
    if (cnt[0] > 2) flags |= RF_MORE_R;
    if (cnt[1] > 2) flags |= RF_MORE_P;
    if (a.neg) flags |= RF_NEG;
    // instruction counts, in units of ten
    weight[r] = (j >= 0 ? 26 : 15) + (p < 0 ? 0 : flags & RF_THD ? 4 : 45);
    if (!ok) {
      flags |= RF_GEN;
      weight[r] = 900;
      ++generic;
    }
    int32_t *h = hdr.data() + 8 * (size_t)r;
    h[0] = r;
    h[1] = flags;
    h[2] = base;
    h[3] = p;
    for (int side = 0; side < 2; ++side) {
      h[4 + 2 * side] = fac[side][0] | (fac[side][1] << 16);
      h[5 + 2 * side] = fac[side][2] | (fac[side][3] << 16);
    }
  }
  // a reaction in FP64 costs this kernel about four times what it costs the
  // kernels that evaluate every reaction so; beyond a fifth of such
  // reactions those are faster
  f.usable = generic * 5 <= R;
  Buf b;
  std::vector<int64_t> small(EXP_ENTRIES + 2 * (LOGN + 1)), hp(2 * (LOGN + 1)), lw(N);
  for (int k = 0; k < EXP_ENTRIES; ++k)
    small[k] = llroundl(std::ldexp(std::exp2((ld)k / EXP_ENTRIES), 56));
  for (int k = 0; k <= LOGN; ++k) {
    const ld F = 1 + (ld)k / LOGN;
    small[EXP_ENTRIES + 2 * k] = hp[2 * k] = llroundl(std::ldexp((ld)1, 62) / F);
    small[EXP_ENTRIES + 2 * k + 1] = llroundl(std::ldexp(std::log2(F), YB));
    hp[2 * k + 1] = llroundl(std::ldexp(std::log2(F), 62));
  }
  for (int k = 0; k < N; ++k) lw[k] = llroundl(std::ldexp(std::log2((ld)t.inv_mw[k]), YB));
  f.small = b.put(small);
  f.hp = b.put(hp);
  f.basis = b.put(basis);
  f.lw = b.put(lw);
  f.hdr = b.put(hdr);
  f.coef = b.put(coef);
  f.thr_ptr = b.put(thr_ptr);
  f.thr = b.put(thr);
  f.pmh = b.put(pmh);
  f.pmc = b.put(pmc);
  f.eff_ptr = b.put(std::vector<int32_t>(t.pm_eff_ptr, t.pm_eff_ptr + NPM + 1));
  f.eff_sp = b.put(std::vector<int32_t>(t.pm_eff_sp, t.pm_eff_sp + t.pm_eff_ptr[NPM]));
  f.eff_k = b.put(eff_k);
  // work lists: longest first onto the least loaded warp
  for (int l = 0; l < NLIST; ++l) {
    const int nw = warps_of(l);
    auto deal = [&](const std::vector<int> &w) {
      std::vector<int> order(w.size());
      for (size_t i = 0; i < w.size(); ++i) order[i] = (int)i;
      std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return w[a] > w[c]; });
      std::vector<std::vector<int>> bins(nw);
      std::vector<long long> load(nw, 0);
      for (int i : order) {
        const int best = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        bins[best].push_back(i);
        load[best] += w[i];
      }
      return bins;
    };
    std::vector<std::vector<int>> bins = deal(weight);
    std::vector<int32_t> ptr(1, 0), rev, list;
    for (auto &v : bins) {
      auto plain = [&](int r) { return hdr[8 * (size_t)r + 1] == (RF_REV | (hdr[8 * (size_t)r + 1] & (RF_MORE_R | RF_MORE_P | RF_NEG))); };
      std::sort(v.begin(), v.end(), [&](int a, int c) {
        const bool pa = plain(a), pc = plain(c);
        return pa != pc ? pa : a < c;
      });
      rev.push_back((int32_t)std::count_if(v.begin(), v.end(), plain));
      list.insert(list.end(), v.begin(), v.end());
      ptr.push_back((int32_t)list.size());
    }
    f.list_ptr[l] = b.put(ptr);
    f.list_rev[l] = b.put(rev);
    f.list[l] = b.put(list);
    std::vector<int> sw(N);
    for (int k = 0; k < N; ++k) sw[k] = 2 + t.spc_ptr[k + 1] - t.spc_ptr[k];
    bins = deal(sw);
    ptr.assign(1, 0);
    list.clear();
    for (auto &v : bins) {
      list.insert(list.end(), v.begin(), v.end());
      ptr.push_back((int32_t)list.size());
    }
    f.sum_ptr[l] = b.put(ptr);
    f.sum[l] = b.put(list);
  }
  f.bytes = (int)b.b.size();
  out.swap(b.b);
}

}  // namespace fx
}  // namespace crs
