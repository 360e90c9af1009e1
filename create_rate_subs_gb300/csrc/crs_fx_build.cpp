// Tables of the FP64 state-tile kernel (crs_fx.cu): every rate and
// equilibrium constant as fixed-point coefficients of normalised functions
// of T, built once at load time in extended precision.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "../../include/crs_tables.h"
#include "crs_fx.cuh"
#include "crs_fx_tab.cuh"
#include "crs_shapes.cuh"

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
  ld pw[5][5];  // T^d = sum_k pw[d][k] t^k
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
  static const int binom[5][5] = {{1}, {1, 1}, {1, 2, 1}, {1, 3, 3, 1}, {1, 4, 6, 4, 1}};
  for (int d = 0; d <= 4; ++d)
    for (int k = 0; k <= d; ++k)
      n.pw[d][k] = binom[d][k] * std::pow(n.mT, (ld)(d - k)) * std::pow(n.hT, (ld)k);
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
    for (int k = 0; k <= 4; ++k)
      for (int d = k > 1 ? k : 1; d <= 4; ++d) f.c[k == 0 ? 0 : 2 + k] += p[d - 1] * n.pw[d][k];
  }
  return f;
}

// The bounds that keep every sum of the kernel inside 64 bits: with
// coefficients of at most 500 in all, six products of the low digits (2^31
// by 2^29) and of the high ones (500 2^20 by 2^31) stay below 2^63; for the
// constants see CONST_MAX.
bool within(const Form &f, ld most = CONST_MAX, ld terms = TERMS_MAX) {
  ld s = 0;
  for (int k = 1; k < 7; ++k) s += std::fabs(f.c[k]);
  return std::isfinite((double)f.c[0]) && std::fabs(f.c[0]) <= most && s <= terms;
}

int64_t constant(ld v) { return llroundl(std::ldexp(v, YB)); }

// a coefficient as the kernel loads it: {hi, lo} digits
int64_t coefficient(ld v) {
  const Dg d = split(llroundl(std::ldexp(v, 52)));
  return (int64_t)(((uint64_t)(unsigned)d.lo << 32) | (unsigned)d.hi);
}
// a 64-bit number as an int2 {high, low}; the constant of a sum carries the
// 1 that rounds its exponent to an even number
int64_t number(int64_t v) {
  return (int64_t)(((uint64_t)v << 32) | ((uint64_t)v >> 32));
}

struct Buf {
  std::vector<unsigned char> b;
  // a section: its offset; what is added until the next one belongs to it
  int begin() {
    b.resize((b.size() + 127) / 128 * 128);
    return (int)b.size();
  }
  void add(const void *p, size_t n) {
    const unsigned char *c = static_cast<const unsigned char *>(p);
    b.insert(b.end(), c, c + n);
  }
  void end() { b.resize(b.size() + 16); }
  template <class T>
  int put(const std::vector<T> &v) {
    const int off = begin();
    add(v.data(), v.size() * sizeof(T));
    end();
    return off;
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
    c0 = ZERO;
    c1 = 0;
  }
  if (std::fabs(c0) > 4000 || std::fabs(c1) > 450) return false;
  w[0] = number((constant(c0) & ~1LL) | (a < 0));
  w[1] = coefficient(c1);
  return true;
}

// Items by weight, the heaviest first.
std::vector<int> by_weight(const std::vector<int> &w) {
  std::vector<int> order(w.size());
  for (size_t i = 0; i < w.size(); ++i) order[i] = (int)i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return w[a] > w[c]; });
  return order;
}

// Lists of items for as many warps as `load` has entries (what they carry
// already): in the order given, each onto the least loaded.
std::vector<std::vector<int>> deal(const std::vector<int> &w, const std::vector<int> &order,
                                   const std::vector<long long> &load) {
  std::vector<std::vector<int>> bins(load.size());
  // the least loaded on top, the first of equal ones
  typedef std::pair<long long, int> Load;
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> heap;
  for (size_t b = 0; b < load.size(); ++b) heap.push(Load(load[b], (int)b));
  for (int i : order) {
    Load l = heap.top();
    heap.pop();
    bins[l.second].push_back(i);
    l.first += w[i];
    heap.push(l);
  }
  return bins;
}

// a double as the float-float pair that the mixed kernels use
void pair_of(double v, float *w) {
  w[0] = (float)v;
  w[1] = (float)(v - (double)w[0]);
}

// The mixed-precision kernel's records and lists.
void build_mixed(const Tab &t, FxTab &f, Buf &b) {
  const int N = t.N, R = t.R;
  f.mixed = N + 2 < 65536;
  for (int j = 0; j < t.NREV; ++j) f.mixed &= t.kc_ptr[j + 1] - t.kc_ptr[j] <= 1;
  if (!f.mixed) return;
  // rows of the tile: the concentrations, one, zero
  struct Rec {
    int32_t slot;
    uint16_t fac[6];
    float rate[8], kc[32];
  };
  struct Eff {
    float w;
    int32_t row;
  };
  struct Other {
    Rec r;
    int32_t neff, ext, flags, sp;
    float fall[16], broad[8];
    Eff eff[MEFF];
  };
  static_assert(sizeof(Rec) == MREC && sizeof(Other) == MPAIR, "");
  std::vector<char> shape(R, 0);
  for (int p = t.seg[0]; p < t.seg[NSHAPE]; ++p) shape[t.perm[p]] = 1;
  std::vector<Other> rec(R);
  // kind: of shape groups, 2 x irreversible + third factors; third body,
  // fall-off, neither, general
  std::vector<int> weight(R), kind(R);
  for (int r = 0; r < R; ++r) {
    const int j = t.rev_idx[r], p = t.pm_idx[r];
    Other &o = rec[r];
    o = Other();
    o.r.slot = r * 256;
    bool ok = t.rate_kind[r] < RATE_PLOG;
    int most = 0;
    for (int side = 0; side < 2; ++side) {
      const int32_t *ptr = side ? t.px_ptr : t.rx_ptr, *sp = side ? t.px_sp : t.rx_sp;
      const int32_t *nint = side ? t.px_nint : t.rx_nint;
      int n = 0;
      for (int q = 0; q < 3; ++q) o.r.fac[3 * side + q] = (uint16_t)N;
      if (side && j < 0) break;
      for (int e = ptr[r]; e < ptr[r + 1]; ++e) {
        ok &= nint[e] >= 0;
        for (int q = 0; q < nint[e]; ++q, ++n)
          if (n < 3) o.r.fac[3 * side + n] = (uint16_t)sp[e];
      }
      ok &= n <= 3;
      most = std::max(most, n);
    }
    memcpy(o.r.rate, t.rate_ff + 8 * r, sizeof o.r.rate);
    if (j >= 0) {
      // the reverse exponent: forward minus the equilibrium constant's, each
      // block c0, c1 (ln T), c2 .. c5 (powers of T), 1/T and, of the first,
      // T_common
      memcpy(o.r.kc, t.kc_mix + 32 * j, sizeof o.r.kc);
      for (int blk = 0; blk < 32; blk += 16)
        for (int q = 0; q < 14; q += 2) {
          float *c = o.r.kc + blk + q;
          const int w = q == 0 ? 0 : q == 2 ? 2 : q == 12 ? 4 : -1;  // the rate row's term
          double v = -((double)c[0] + c[1]);
          if (w >= 0) v += (double)o.r.rate[w] + o.r.rate[w + 1];
          pair_of(v, c);
        }
    }
    int flags = j >= 0 ? MF_REV : 0;
    o.sp = -1;
    if (p >= 0) {
      const bool thd = t.pm_kind[p] == PM_THD;
      flags |= thd ? MF_THD : MF_FALL;
      if (!thd) {
        o.sp = t.pm_sp[p];
        memcpy(o.fall, t.rate_ff + 8 * t.pm_k0[p], 32);
        memcpy(o.fall + 8, t.rate_ff + 8 * t.pm_kinf[p], 32);
        o.fall[6] *= o.fall[14];  // the signs
        const int form = t.pm_form[p];
        if (t.pm_kind[p] == PM_FALL_LOW) o.flags |= PMF_LOW;
        if (form == FORM_TROE) o.flags |= PMF_TROE | (t.pm_troe_t2[p] ? PMF_T2 : 0);
        if (form == FORM_SRI) o.flags |= PMF_SRI | (t.pm_sri_de[p] ? PMF_DE : 0);
        if (form != FORM_LINDEMANN)
          memcpy(o.broad, (form == FORM_TROE ? t.troe_ff : t.sri_ff) + 8 * p, sizeof o.broad);
      }
      if (o.sp < 0) {
        // an even number of terms
        std::vector<Eff> more;
        for (int e = t.pm_eff_ptr[p]; e < t.pm_eff_ptr[p + 1]; ++e)
          more.push_back(Eff{t.eff_f[e], t.pm_eff_sp[e]});
        if (more.size() & 1) more.push_back(Eff{0.0f, N});
        o.neff = (int)more.size();
        const size_t in = std::min<size_t>(more.size(), MEFF);
        std::copy(more.begin(), more.begin() + in, o.eff);
        more.erase(more.begin(), more.begin() + in);
        if (!more.empty()) o.ext = b.put(more);
      }
    }
    // instruction counts, in units of ten
    if (shape[r]) {
      kind[r] = (j >= 0 ? 0 : 2) + (most > 2);
      weight[r] = j >= 0 ? 24 : 11;
      flags = 0;
    } else if (ok) {
      kind[r] = p < 0 ? 6 : flags & MF_THD ? 4 : 5;
      weight[r] = 28 + (p < 0 ? 0 : flags & MF_THD ? 2 + o.neff / 2 : 45);
    } else {
      flags = MF_GEN;
      kind[r] = 7;
      weight[r] = 250;
    }
    o.r.slot |= flags;
  }
  Rec none = Rec();  // completes a pair: both rates zero, into the slot of zeros
  none.slot = R * 256;
  for (int q = 0; q < 6; ++q) none.fac[q] = (uint16_t)(N + 1);
  const std::vector<int> order = by_weight(weight);
  for (int l = 0; l < NLIST; ++l) {
    const int nw = list_warps[l];
    std::vector<long long> load(nw, 0);
    load[0] = load[1] = 2 * N;  // the next tile's sums and functions of T
    load[2] = 20;
    std::vector<int32_t> ptr(1, 0), pairs;
    f.mrec[l] = b.begin();
    auto count = [&] { return (int32_t)((b.b.size() - f.mrec[l]) / MPAIR); };
    for (const auto &v : deal(weight, order, load)) {
      for (int c = 0; c < 4; ++c) {
        std::vector<Rec> two;
        for (int r : v)
          if (kind[r] == c) two.push_back(rec[r].r);
        if (two.size() & 1) two.push_back(none);
        for (size_t q = 0; q < two.size(); q += 2)
          two[q].slot |= (c & 1 ? MF_MORE : 0) | (c < 2 ? MF_REV : 0);
        b.add(two.data(), two.size() * MREC);
      }
      pairs.push_back(count() - ptr.back());
      for (int c = 4; c < 8; ++c)
        for (int r : v)
          if (kind[r] == c) b.add(&rec[r], MPAIR);
      ptr.push_back(count());
    }
    b.end();
    f.mlist_ptr[l] = b.put(ptr);
    f.mpairs[l] = b.put(pairs);
  }
}

// An upper bound of the tables' size (one: bytes of a plain reaction's
// record).
int64_t bytes_bound(const Tab &t, int64_t one) {
  const int64_t N = t.N, R = t.R, NPM = t.NPM, nnz = t.nu_ptr[R];
  const int64_t neff = t.pm_eff_ptr[NPM];
  const int64_t records = R * (one + PMH + PMC * NI + MPAIR);
  const int64_t terms = 16 * N + 4 * 3 * nnz;
  // the small tables and the sections' alignment (a section per pressure-
  // modified reaction with many colliders), then the lists, whose pairs are
  // completed once per warp that has reactions (and kind of pair)
  int64_t all = (1 << 15) + 8 * N + (20 + 144) * NPM + 24 * neff + 12 * nnz;
  for (int l = 0; l < NLIST; ++l) {
    const int64_t nw = list_warps[l];
    all += records + terms + 16 * N + std::min(nw, R) * one + std::min(4 * nw, R) * MREC +
           6 * 4 * (nw + 1);
  }
  return all;
}

// The tables that are the same for every mechanism, made once: 1,300
// exponentials and logarithms in extended precision.
struct Small {
  std::vector<int64_t> small, hp;
  Small() : small(EXP_WORDS + 2 * (LOGN + 1)), hp(2 * (LOGN + 1)) {
    for (int k = 0; k <= EXPN; ++k)
      small[k] = llroundl(std::ldexp(std::exp2((ld)k / EXPN), 56)) + 8;
    for (int k = 0; k <= LOGN; ++k) {
      const ld F = 1 + (ld)k / LOGN;
      small[EXP_WORDS + 2 * k] = hp[2 * k] = llroundl(std::ldexp((ld)1, 62) / F);
      small[EXP_WORDS + 2 * k + 1] = llroundl(std::ldexp(std::log2(F), YB));
      hp[2 * k + 1] = llroundl(std::ldexp(std::log2(F), 62));
    }
  }
};

}  // namespace

void build(const Tab &t, FxTab &f, std::vector<unsigned char> &out, int64_t limit) {
  f = FxTab();
  out.clear();
  const int N = t.N, R = t.R, NPM = t.NPM;
  f.N = N;
  f.R = R;
  f.NPM = NPM;
  if (R < 1 || R >= (1 << 22)) return;  // slot offsets in 30 bits
  limit = std::min<int64_t>(limit, INT32_MAX);  // the tables' offsets are ints
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
  f.tb[0] = 200.0;
  f.tb[1] = mid;
  f.tb[2] = 6000.0;
  std::vector<int64_t> basis;
  Norm nm[NI];
  for (int q = 0; q < NI; ++q) {
    nm[q] = norm_of(f.tb[q], f.tb[q + 1]);
    basis.insert(basis.end(), nm[q].word, nm[q].word + BASIS);
  }
  // pressure modification
  std::vector<int32_t> pmh(4 * (size_t)std::max(NPM, 1), 0), pm(2 * (size_t)std::max(NPM, 1), 0);
  std::vector<int64_t> pmc((size_t)PMC / 8 * NI * std::max(NPM, 1), 0);
  std::vector<char> pm_ok(std::max(NPM, 1), 1);
  std::vector<int32_t> pm_rxn(std::max(NPM, 1), 0);
  for (int r = 0; r < R; ++r)
    if (t.pm_idx[r] >= 0) pm_rxn[t.pm_idx[r]] = r;
  std::vector<double> eff;  // pairs: coefficient, row offset
  for (int p = 0; p < NPM; ++p) {
    int flags = 0;
    const bool thd = t.pm_kind[p] == PM_THD;
    const int sp = thd ? -1 : t.pm_sp[p];
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
        int64_t *w = pmc.data() + (size_t)PMC / 8 * (NI * p + q);
        const Form z = form_of(nm[q], a.base - b.base, a.b - b.b, a.i - b.i, nullptr);
        ok = within(z);
        if (!ok) break;
        w[0] = number(constant(z.c[0]) + 1);
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
              ok = within(y, DE_MAX / 2, DE_MAX / 2);
              w[9] = number(constant(y.c[0]) + 1);
              w[10] = coefficient(y.c[1]);
            }
          }
        }
      }
    }
    for (int e = t.pm_eff_ptr[p]; e < t.pm_eff_ptr[p + 1]; ++e) {
      eff.push_back(t.pm_eff_val[e] * t.inv_mw[t.pm_eff_sp[e]]);
      const int64_t off = (int64_t)t.pm_eff_sp[e] * 256;
      double w;
      memcpy(&w, &off, 8);
      eff.push_back(w);
    }
    pmh[4 * p] = flags;
    pmh[4 * p + 1] = sp < 0 ? -1 : sp * 256;
    pm[2 * p] = sp < 0 ? pm_rxn[p] * 256 : -1;
    pm_ok[p] = ok;
  }
  // reactions: thresholds where their coefficients change (the interval
  // bounds and their own T_common values), then the records
  std::vector<std::vector<double>> thr(R);
  size_t nthr = 1;
  bool uniform = true;
  for (int r = 0; r < R; ++r) {
    std::vector<double> &th = thr[r];
    th = {f.tb[1]};
    const int j = t.rev_idx[r];
    if (j >= 0)
      for (int g = t.kc_ptr[j]; g < t.kc_ptr[j + 1]; ++g) {
        const double x = t.kc_tmid[g];
        if (x > f.tb[0] && x < f.tb[NI] && std::find(th.begin(), th.end(), x) == th.end()) {
          th.push_back(x);
          uniform = false;
        }
      }
    std::sort(th.begin(), th.end());
    nthr = std::max(nthr, th.size());
  }
  f.nthr = uniform ? 0 : (int)nthr;
  const int nco = (int)nthr + 1;
  const int one = HEAD + COEF * nco + (uniform ? 0 : ((int)nthr + 1) / 2 * 16);
  f.stride[0] = 2 * one;
  f.stride[1] = one + PMH + PMC * NI;
  if (bytes_bound(t, one) > limit) return;
  std::vector<std::vector<unsigned char>> rec(R);
  std::vector<int> weight(R), kind(R);
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
      for (int q = 0; q < 4; ++q) fac[side][q] = N;  // the row of zeros
      if (side && j < 0) break;
      for (int e = ptr[r]; e < ptr[r + 1]; ++e) {
        if (nint[e] < 0) ok = false;
        for (int q = 0; q < nint[e]; ++q, ++cnt[side])
          if (cnt[side] < 4) fac[side][cnt[side]] = sp[e];
      }
      ok &= cnt[side] <= 4;
    }
    std::vector<unsigned char> co((size_t)COEF * nco, 0);
    const std::vector<double> &th = thr[r];
    for (size_t q = 0; q <= th.size(); ++q) {
      const double hi = q < th.size() ? th[q] : f.tb[NI];
      int iv = 0;
      while (hi > f.tb[iv + 1]) ++iv;
      int64_t w[COEF / 8] = {0};
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
        w[0] = number(constant(y.c[0]) + 1);
        w[1] = coefficient(y.c[1]);
        w[2] = coefficient(y.c[2]);
        w[3] = number(constant(z.c[0]) + 1);
        for (int k = 1; k < 7; ++k) w[3 + k] = coefficient(z.c[k]);
      }
      memcpy(co.data() + COEF * q, w, COEF);
    }
    if (j >= 0) flags |= RF_REV;
    if (p >= 0) flags |= t.pm_kind[p] == PM_THD ? RF_THD : RF_FALL;
    if (cnt[0] > 2 || cnt[1] > 2) flags |= RF_MORE;
    if (a.neg) flags |= RF_NEG;
    // instruction counts, in units of ten
    weight[r] = (j >= 0 ? 24 : 20) + (p < 0 ? 0 : flags & RF_THD ? 21 : 84);
    kind[r] = p >= 0 ? 2 : j >= 0 ? 0 : 1;
    if (!ok) {
      flags |= RF_GEN;
      weight[r] = 900;
      kind[r] = 3;
      ++generic;
    }
    const int32_t h[12] = {r * 256, flags, p, r,
                           fac[0][0] * 256, fac[0][1] * 256, fac[1][0] * 256, fac[1][1] * 256,
                           fac[0][2] * 256, fac[0][3] * 256, fac[1][2] * 256, fac[1][3] * 256};
    std::vector<unsigned char> &at = rec[r];
    auto add = [&](const void *v, size_t n) {
      at.insert(at.end(), (const unsigned char *)v, (const unsigned char *)v + n);
    };
    add(h, HEAD);
    if (kind[r] != 0) {
      static const unsigned char none[PMH + PMC * NI] = {0};
      add(p >= 0 ? (const void *)(pmh.data() + 4 * p) : none, PMH);
      add(p >= 0 ? (const void *)(pmc.data() + (size_t)PMC / 8 * NI * p) : none, PMC * NI);
    }
    add(co.data(), co.size());
    if (!uniform) {
      std::vector<double> v((nthr + 1) / 2 * 2, INFINITY);
      std::copy(th.begin(), th.end(), v.begin());
      add(v.data(), v.size() * sizeof(double));
    }
  }
  // General reactions gain nothing here.  131,072 states of 53/325 with PLOG in 5,
  // 10, 15 and 19% of the reactions: 2.39, 3.68, 5.22 and 6.40 ms, by the kernels
  // that evaluate every reaction in FP64 5.73, 7.17, 8.73 and 9.91; more was not
  // measured and goes to those
  f.usable = generic * 5 <= R;
  for (int k = 0; k < N; ++k) f.usable &= std::fabs(std::log2(t.inv_mw[k])) <= W_MAX;
  Buf b;
  b.b.reserve((size_t)bytes_bound(t, one));
  static const Small constants;
  std::vector<int64_t> lw(N);
  for (int k = 0; k < N; ++k) lw[k] = llroundl(std::ldexp(std::log2((ld)t.inv_mw[k]), YB));
  f.small = b.put(constants.small);
  f.hp = b.put(constants.hp);
  f.basis = b.put(basis);
  f.lw = b.put(lw);
  f.pm = b.put(pm);
  f.eff_ptr = b.put(std::vector<int32_t>(t.pm_eff_ptr, t.pm_eff_ptr + NPM + 1));
  f.eff = b.put(eff);
  // species' terms: coefficients +-1 (small integers repeated) or weighted
  std::vector<std::vector<int32_t>> terms(N);
  std::vector<int32_t> wterm, where(4 * (size_t)N, 0);
  std::vector<double> wnu;
  for (int k = 0; k < N; ++k) {
    bool small_int = true;
    for (int e = t.spc_ptr[k]; e < t.spc_ptr[k + 1]; ++e)
      small_int &= std::fabs(t.spc_nu[e]) <= 3 && t.spc_nu[e] == std::rint(t.spc_nu[e]);
    int32_t *w = where.data() + 4 * (size_t)k;
    w[0] = k;
    w[2] = (int32_t)wterm.size();
    for (int e = t.spc_ptr[k]; e < t.spc_ptr[k + 1]; ++e) {
      if (small_int) {
        for (int q = 0; q < std::abs((int)t.spc_nu[e]); ++q)
          terms[k].push_back((int32_t)((unsigned)t.spc_r[e] * 256u |
                                       (t.spc_nu[e] < 0 ? 0x80000000u : 0u)));
      } else {
        wterm.push_back(t.spc_r[e] * 256);
        wnu.push_back(t.spc_nu[e]);
      }
    }
    while (terms[k].size() % 4) terms[k].push_back(R * 256);
    w[1] = (int32_t)(terms[k].size() / 4);
    w[3] = (int32_t)wterm.size() - w[2];
  }
  f.wterm = b.put(wterm);
  f.wnu = b.put(wnu);
  std::vector<int> sw(N);
  for (int k = 0; k < N; ++k) sw[k] = 2 + t.spc_ptr[k + 1] - t.spc_ptr[k];
  // the reaction that completes a pair: both rates zero, into the slot of
  // zeros
  std::vector<unsigned char> nothing(one, 0);
  {
    const int32_t h[12] = {R * 256, RF_REV, -1, -1, N * 256, N * 256, N * 256, N * 256,
                           N * 256, N * 256, N * 256, N * 256};
    memcpy(nothing.data(), h, HEAD);
    const int64_t z = number(ZERO_EXP);
    for (int q = 0; q < nco; ++q) {
      memcpy(nothing.data() + HEAD + COEF * q, &z, 8);
      memcpy(nothing.data() + HEAD + COEF * q + 24, &z, 8);
    }
  }
  // work lists
  const std::vector<int> order = by_weight(weight), species_order = by_weight(sw);
  for (int l = 0; l < NLIST; ++l) {
    const int nw = list_warps[l];
    // warps 0 and 1 also form the next tile's sums (chains of N dependent
    // FP64 additions), warp 2 its functions of T
    std::vector<long long> load(nw, 0);
    load[0] = load[1] = 2 * N;
    load[2] = 60;
    std::vector<std::vector<int>> bins = deal(weight, order, load);
    for (int c = 0; c < 2; ++c) {
      std::vector<int32_t> ptr(1, 0);
      f.rec[l][c] = b.begin();
      for (auto &v : bins) {
        std::sort(v.begin(), v.end(), [&](int x, int y) {
          return kind[x] != kind[y] ? kind[x] < kind[y] : x < y;
        });
        int n = 0;
        for (int r : v)
          if ((kind[r] != 0) == (c == 1)) {
            b.add(rec[r].data(), rec[r].size());
            ++n;
          }
        if (c == 0) {
          if (n & 1) b.add(nothing.data(), nothing.size());
          n = (n + 1) / 2;
        }
        ptr.push_back(ptr.back() + n);
      }
      b.end();
      f.list_ptr[l][c] = b.put(ptr);
    }
    bins = deal(sw, species_order, std::vector<long long>(nw, 0));
    std::vector<int32_t> ptr(1, 0), tptr(1, 0), seg, term;
    for (auto &v : bins) {
      std::stable_sort(v.begin(), v.end(), [&](int x, int y) {
        return (where[4 * x + 3] > 0) < (where[4 * y + 3] > 0);
      });
      for (int k : v) {
        seg.insert(seg.end(), where.begin() + 4 * k, where.begin() + 4 * k + 4);
        term.insert(term.end(), terms[k].begin(), terms[k].end());
      }
      ptr.push_back((int32_t)(seg.size() / 4));
      tptr.push_back((int32_t)(term.size() / 4));
    }
    for (int q = 0; q < 8; ++q) term.push_back(R * 256);  // read ahead
    seg.insert(seg.end(), {0, 0, 0, 0});  // read ahead
    f.seg_ptr[l] = b.put(ptr);
    f.seg[l] = b.put(seg);
    f.term_ptr[l] = b.put(tptr);
    f.term[l] = b.put(term);
  }
  build_mixed(t, f, b);
  f.bytes = (int)b.b.size();
  out.swap(b.b);
}

}  // namespace fx
}  // namespace crs
